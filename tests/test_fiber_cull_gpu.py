"""Fiber candidates by sign classes: tile edges (32 x 8 corners, 4 time steps),
layouts, offsets, quantised ties and values off the 32-bit lattice range,
against the exact C restatement."""
import numpy as np
import pytest

from ftk2_b200 import api
from oracle import bridge
from test_fiber_gpu import assert_same

pytestmark = pytest.mark.gpu


def _values(kind, shape, dtype, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(shape)
    if kind == "ties":      # a few lattice steps around zero, many exact zeros
        v = np.round(2 * v) / 2.0 ** 20
    elif kind == "huge":    # some values past 2^31 lattice steps, some past 2^63
        v = np.where(rng.random(shape) < 0.2, v * 1e4, v)
        v = np.where(rng.random(shape) < 0.05, v * 1e15, v)
    return v.astype(dtype)


@pytest.mark.parametrize("dims", [[2, 2, 2], [32, 8, 4], [33, 9, 5], [34, 10, 6], [65, 17, 9]])
@pytest.mark.parametrize("kind", ["noise", "ties", "huge"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_fiber_tiles(ctx, dims, kind, dtype):
    shape, thr = tuple(dims[::-1]), (0.125, -0.0625) if kind == "noise" else (0.0, 0.0)
    f = [_values(kind, shape, dtype, s) for s in (1, 2)]
    keep: list = []
    off, glob = [3, 2, 1], [d + o + 2 for d, o in zip(dims, (3, 2, 1))]
    for offset, gdims in ((None, None), (off, glob)):
        want = bridge.run_restatement(bridge.make_regular_mesh(dims, offset, gdims),
                                      bridge.make_field(f, bridge.LAYOUT_SEPARATE, 2, sos_q=2.0 ** 20, keep=keep,
                                                        fiber_thr=thr))
        want = {k: getattr(want, k) for k in ("simplices", "bary", "lam", "track_id", "edges")}
        mesh = api.regular_mesh_desc(dims, offset, gdims)
        assert_same(ctx.fiber(mesh, api.field_desc(f, api.LAYOUT_SEPARATE, 2, keep=keep), thr, 2.0 ** 20), want)
    both = np.stack(f, -1)
    whole = ctx.fiber(api.regular_mesh_desc(dims), api.field_desc(both, api.LAYOUT_MULTICOMPONENT, 2, keep=keep), thr,
                      2.0 ** 20)
    flat = [a.reshape(-1) for a in f]
    same = ctx.fiber(api.regular_mesh_desc(dims), api.field_desc(flat, api.LAYOUT_SEPARATE, 2, keep=keep), thr,
                     2.0 ** 20)
    sep = ctx.fiber(api.regular_mesh_desc(dims), api.field_desc(f, api.LAYOUT_SEPARATE, 2, keep=keep), thr, 2.0 ** 20)
    for r in (whole, same):
        assert_same(r, {k: getattr(sep, k) for k in ("simplices", "bary", "lam", "track_id", "edges")})
