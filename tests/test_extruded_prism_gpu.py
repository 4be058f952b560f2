"""Extruded meshes whose base cells end at, before and after a block's share
(512 cells) of the extraction kernel, over one layer and several, of values
without a cull (white noise) and with one: identical to the exact C
restatement."""
import numpy as np
import pytest

from ftk2_b200 import synthetic as S
import cases
from test_extruded_gpu import _tri_plane, assert_identical, gpu_run, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smooth", [False, True], ids=["noise", "smooth"])
@pytest.mark.parametrize("n_layers", [0, 1, 3])
@pytest.mark.parametrize("ncell", [1, 511, 512, 513, 1025])
@pytest.mark.parametrize("m", [2, 3])
def test_prism_blocks(ctx, m, ncell, n_layers, smooth):
    coords, cells = S.extruded_tet_mesh(10, 9, 4, seed=3) if m == 3 else _tri_plane(30, 21, 3)
    assert len(cells) >= ncell
    n = coords.shape[0] * (n_layers + 1)
    dtype = np.float32 if n_layers == 1 else np.float64
    v = np.random.default_rng(5).standard_normal((m, n))
    if smooth:  # one sign change along the vertex ids
        v = 0.01 * v + np.linspace(-1.0, 2.0, n)
    case = cases.Case("prism", "extruded", m, cases.PER_VERTEX, list(v.astype(dtype)), 2.0 ** 20, coords=coords,
                      cells=np.ascontiguousarray(cells[-ncell:]), n_layers=n_layers)
    o = oracle_run(case)
    g = gpu_run(ctx, case)
    assert_identical(g, o)
    assert g.n_simplices == o.n_tested


@pytest.mark.parametrize("pages", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("m", [2, 3])
def test_many_cells_on_one_face(ctx, m, pages):
    """Cells that share one face, more of them than one round of a star
    group's lanes takes (three tets, four triangles)."""
    books, n_layers = 40, 6
    per = m + pages
    face, tip = np.arange(m), m + np.arange(pages)[:, None]
    book = np.concatenate([np.broadcast_to(face, (pages, m)), tip], 1)
    cells = (np.arange(books)[:, None, None] * per + book).reshape(-1, m + 1).astype(np.uint64)
    n = books * per
    v = np.random.default_rng(pages).standard_normal((m, n * (n_layers + 1)))
    case = cases.Case("pages", "extruded", m, cases.PER_VERTEX, list(v), 2.0 ** 20, coords=np.zeros((n, 3)),
                      cells=np.ascontiguousarray(cells), n_layers=n_layers)
    o = oracle_run(case)
    assert len(o.edges) > 0
    assert_identical(gpu_run(ctx, case), o)


@pytest.mark.parametrize("n_layers", [1, 2, 3])
def test_sort_by_rank_and_by_passes(ctx, n_layers):
    """Feature counts on both sides of the rank sort's 12,288."""
    coords, tets = S.extruded_tet_mesh(12, 11, 7, seed=2)
    v = np.random.default_rng(8).standard_normal((3, (n_layers + 1) * coords.shape[0]))
    case = cases.Case("noise", "extruded", 3, cases.PER_VERTEX, list(v), 2.0 ** 20, coords=coords, cells=tets,
                      n_layers=n_layers)
    o = oracle_run(case)
    assert (len(o.track_id) > 12288) == (n_layers == 3)
    assert_identical(gpu_run(ctx, case), o)
