"""The long chain's radix sort splits its keys by the feature capacity: the
results are the same for every number of blocks, at each end of the rule that
chooses it."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


def test_sort_blocks():
    f = np.random.default_rng(8).standard_normal((3, 12, 12, 12, 3))
    case = cases.Case("noise", "regular", 3, cases.MULTI, f, 2.0 ** 20, [12, 12, 12, 3])
    want = oracle_run(case)
    assert 17000 < len(want.track_id) < 28000
    keep: list = []
    mesh, fld = cases.gpu_inputs(case, keep)
    for capacity in (28672, 131071, 131072, 262143, 262144, 266240):
        with api.Context(0) as ctx:
            ctx.set_option(api.OPT_FEATURE_CAPACITY, capacity)
            assert_identical(ctx.extract(mesh, fld, api.params(case.sos_q)), want)
