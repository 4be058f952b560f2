"""2D+t meshes whose sides end at, before and after a strip of the cull (31 x 4
corners) and whose steps are one chunk or several, in every layout, of noise and
of smooth values: identical to the exact C restatement."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, gpu_run, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["noise", "smooth"])
@pytest.mark.parametrize("layout", ["multi", "separate", "separate_offset", "per_vertex"])
@pytest.mark.parametrize("dims", [[1, 1, 2], [31, 4, 2], [32, 5, 3], [30, 3, 9], [63, 9, 1], [94, 17, 5]])
def test_strips(ctx, dims, layout, kind):
    rng = np.random.default_rng(11)
    off, gdims = ([3, 2, 1], [d + o + 2 for d, o in zip(dims, [3, 2, 1])]) if layout == "separate_offset" \
        else (None, None)
    shape = tuple(reversed(gdims or dims))
    v = rng.standard_normal(shape + (2,))
    if kind == "smooth":  # a circle of zeros that grows in time
        t, y, x = np.indices(shape)
        v[..., 0] = x - shape[2] / 2 + 0.01 * v[..., 0]
        v[..., 1] = y - shape[1] / 2 + 0.1 * t + 0.01 * v[..., 1]
    v = v.astype(np.float32 if layout.startswith("sep") else np.float64)
    if layout == "multi":
        case = cases.Case("strip", "regular", 2, cases.MULTI, v, 2.0 ** 20, dims)
    elif layout == "per_vertex":
        case = cases.Case("strip", "regular", 2, cases.PER_VERTEX,
                          [np.ascontiguousarray(v[..., j].ravel()) for j in range(2)], 2.0 ** 20, dims)
    else:
        arrays = [np.ascontiguousarray(v[..., j]) for j in range(2)]
        if off:
            cut = tuple(slice(o, o + d) for o, d in zip(reversed(off), reversed(dims)))
            arrays = [np.ascontiguousarray(np.pad(a[cut], ((0, 0), (0, 1), (0, 2)))) for a in arrays]
        case = cases.Case("strip", "regular", 2, cases.SEPARATE, arrays, 2.0 ** 20, dims, off, gdims)
    o = oracle_run(case)
    assert_identical(gpu_run(ctx, case), o)
    for chunk in (1, 2):
        ctx.set_option(api.OPT_TIME_CHUNK, chunk)
        try:
            assert_identical(gpu_run(ctx, case), o)
        finally:
            ctx.set_option(api.OPT_TIME_CHUNK, 0)
