"""Results above 32 MB, copied array by array through the ring of pinned chunks,
in both dimensions, with classes and without edges, against the exact C
restatement and the same run's packed form."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_pack_gpu import _noise
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[240, 190, 5], [27, 26, 25, 4]])
def test_large_results(dims):
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, _noise(dims, 6), 2.0 ** 20, dims)
    want = oracle_run(case)
    k = len(dims)
    assert len(want.track_id) * (20 * k + 12) > 32 << 20
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    with api.Context(0) as ctx:
        for _ in range(2):
            got = ctx.extract(mesh, fld, api.params(case.sos_q))
            assert_identical(got, want)
            assert not got.cp_class.any()
        ctx.run(mesh, fld, api.params(case.sos_q, classify=True))
        typed = ctx.fetch()
        assert_identical(typed, want)
        assert (typed.cp_class > 0).any()
        bare = ctx.extract(mesh, fld, api.params(case.sos_q, want_edges=False))
        assert np.array_equal(bare.simplices, want.simplices) and np.array_equal(bare.lam, want.lam)
        assert np.array_equal(bare.track_id, np.arange(len(want.track_id))) and len(bare.edges) == 0
