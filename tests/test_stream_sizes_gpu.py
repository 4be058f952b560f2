"""Streams of white noise, whose windows and stores lie below, between and
above the sizes the rank sort takes (12,288 tuples, 24,576 keys): every prefix
equals the one-shot result, and that the exact C restatement."""
import numpy as np
import pytest

from ftk2_b200 import synthetic as S
from oracle import bridge
import cases
from test_pack_gpu import _noise
from test_parity_gpu import oracle_run
import test_stream_gpu as ts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[5, 4, 3], [3, 3, 3, 2], [16, 15, 14, 3], [90, 80, 4]])
def test_regular(ctx, dims):
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, _noise(dims, 7), 2.0 ** 20, dims)
    r = ts.stream_case(ctx, case, classify=True, check_every=True)
    ts.assert_identical(r, oracle_run(case))


@pytest.mark.parametrize("plane,nt", [((4, 3, 3), 3), ((12, 11, 7), 4), ((20, 19, 9), 3)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_extruded(ctx, plane, nt, dtype):
    coords, tets = S.extruded_tet_mesh(*plane, seed=2)
    rng = np.random.default_rng(8)
    v = [rng.standard_normal(nt * coords.shape[0]).astype(dtype) for _ in range(3)]
    case = cases.Case("noise", "extruded", 3, cases.PER_VERTEX, v, 2.0 ** 20, coords=coords, cells=tets,
                      n_layers=nt - 1)
    r = ts.ext_stream_case(ctx, case, check_every=True)
    ts.assert_identical(r, oracle_run(case))


@pytest.mark.parametrize("nt", [2, 5])
def test_extruded_triangles(ctx, nt):
    rng = np.random.default_rng(9)
    nx, ny = 23, 19
    i, j = np.meshgrid(np.arange(nx - 1), np.arange(ny - 1), indexing="xy")
    a = (i + nx * j).ravel()
    tri = np.concatenate([np.stack([a, a + 1, a + nx + 1], 1), np.stack([a, a + nx + 1, a + nx], 1)])
    v = [rng.standard_normal(nt * nx * ny) for _ in range(2)]
    case = cases.Case("noise", "extruded", 2, cases.PER_VERTEX, v, 2.0 ** 20, coords=np.zeros((nx * ny, 3)),
                      cells=tri.astype(np.uint64), n_layers=nt - 1)
    r = ts.ext_stream_case(ctx, case, check_every=True)
    ts.assert_identical(r, oracle_run(case))


@pytest.mark.parametrize("kind", ["regular", "extruded"])
@pytest.mark.parametrize("loud", [(3, 7), (2, 3, 9)])
def test_windows_of_sudden_size(ctx, kind, loud):
    """Steps without features between noisy ones: windows far larger than four
    times the last, which are run again, and empty ones."""
    nt = 11
    rng = np.random.default_rng(10)
    if kind == "regular":
        dims = [19, 17, nt]
        v = rng.standard_normal((nt, 17, 19, 2))
    else:
        coords, tets = S.extruded_tet_mesh(9, 8, 5, seed=2)
        v = rng.standard_normal((nt, coords.shape[0], 3))
    quiet = [t for t in range(nt) if t not in loud]
    v[quiet] = np.abs(v[quiet]) + 0.1
    if kind == "regular":
        case = cases.Case("sudden", "regular", 2, cases.MULTI, v, 2.0 ** 20, dims)
        r = ts.stream_case(ctx, case, classify=True, check_every=True)
    else:
        arrays = [np.ascontiguousarray(v[..., j].ravel()) for j in range(3)]
        case = cases.Case("sudden", "extruded", 3, cases.PER_VERTEX, arrays, 2.0 ** 20, coords=coords, cells=tets,
                          n_layers=nt - 1)
        r = ts.ext_stream_case(ctx, case, check_every=True)
    o = oracle_run(case)
    assert len(o.track_id) > 1200
    ts.assert_identical(r, o)
