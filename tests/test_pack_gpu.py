"""Result delivery: every size of result, packed inside the pipeline (extract)
and after it (run, then fetch), against the exact C restatement."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


def _noise(dims, seed):
    """White noise: several features per vertex."""
    m = len(dims) - 1
    return np.random.default_rng(seed).standard_normal(tuple(dims[::-1]) + (m,))


# no feature; a few; more than the context's own pinned block holds (both
# dimensions); more than is ever packed (copied array by array)
@pytest.mark.parametrize("dims", [[6, 5, 3], [9, 7, 3], [71, 60, 5], [13, 11, 10, 4], [181, 160, 5]])
@pytest.mark.parametrize("graphs", [1, 0])
def test_every_result_size(dims, graphs):
    f = np.abs(_noise(dims, 3)) if dims == [6, 5, 3] else _noise(dims, 3)
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, f, 2.0 ** 20, dims)
    want = oracle_run(case)
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    with api.Context(0) as ctx:
        ctx.set_option(api.OPT_USE_GRAPHS, graphs)
        for _ in range(2):  # the second time the buffers have their size
            assert_identical(ctx.extract(mesh, fld, api.params(case.sos_q)), want)
        n, _ = ctx.run(mesh, fld, api.params(case.sos_q))
        assert n == len(want.track_id)
        assert_identical(ctx.fetch(), want)
        assert_identical(ctx.fetch(), want)


@pytest.mark.parametrize("dims", [[9, 7, 3], [13, 11, 10, 4]])
def test_classes_and_no_edges(dims):
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, _noise(dims, 4), 2.0 ** 20, dims)
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    with api.Context(0) as ctx:
        typed = ctx.extract(mesh, fld, api.params(case.sos_q, classify=True))
        ctx.run(mesh, fld, api.params(case.sos_q, classify=True))
        assert np.array_equal(typed.cp_class, ctx.fetch().cp_class) and (typed.cp_class > 0).any()
        bare = ctx.extract(mesh, fld, api.params(case.sos_q, want_edges=False))
    assert np.array_equal(bare.simplices, typed.simplices) and np.array_equal(bare.lam, typed.lam)
    assert np.array_equal(bare.track_id, np.arange(len(bare.track_id))) and len(bare.edges) == 0
    assert not bare.cp_class.any() and bare.n_tracks == 0


def test_inside_list_longer_than_its_first_capacity():
    """Values that all quantise to 0: every simplex passes the inside test by
    its ties and only the solve rejects (more than 131,072 listed simplices)."""
    dims = [17, 15, 13, 3]
    case = cases.Case("flat", "regular", 3, cases.MULTI, 1e-8 * _noise(dims, 5), 2.0 ** 20, dims)
    want = oracle_run(case)
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    with api.Context(0) as ctx:
        for _ in range(2):
            assert_identical(ctx.extract(mesh, fld, api.params(case.sos_q)), want)
        assert ctx.get_option(api.INFO_LAST_TESTED) > 131072
