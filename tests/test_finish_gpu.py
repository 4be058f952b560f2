"""The short chain's last step: feature counts around a block (1,024), the
blocks that find roots (8,192) and the chain's capacity (16,384), with edges and
without, packed and left on the device, against the exact C restatement."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_pack_gpu import _noise
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,lo,hi", [([2, 2, 2], 0, 1024), ([16, 11, 3], 512, 1536), ([40, 33, 3], 4096, 8192),
                                        ([43, 38, 4], 8192, 16384), ([60, 46, 4], 16384, 32768),
                                        ([9, 8, 7, 2], 1024, 8192)])
def test_counts(dims, lo, hi):
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, _noise(dims, 5), 2.0 ** 20, dims)
    want = oracle_run(case)
    assert lo <= len(want.track_id) < hi
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    with api.Context(0) as ctx:
        for _ in range(2):
            assert_identical(ctx.extract(mesh, fld, api.params(case.sos_q)), want)
        ctx.run(mesh, fld, api.params(case.sos_q))
        assert_identical(ctx.fetch(), want)
        r = ctx.extract(mesh, fld, api.params(case.sos_q, want_edges=False))
        assert np.array_equal(r.simplices, want.simplices) and np.array_equal(r.lam, want.lam)
        assert len(r.edges) == 0 and np.array_equal(r.track_id, np.arange(len(want.track_id)))
        ctx.set_option(api.OPT_FEATURE_CAPACITY, max(1, len(want.track_id) - 1))
        assert_identical(ctx.extract(mesh, fld, api.params(case.sos_q)), want)
