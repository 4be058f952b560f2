"""2D+t meshes through every form of the cull that takes them -- strips (mode
0), tile statistics with TMA staging (mode 1), and a batch staged by TMA or by
plain copies -- against the exact C restatement; and the strips' failure path."""
import numpy as np
import pytest

from ftk2_b200 import api
from ftk2_b200 import synthetic as S
import cases
from test_parity_gpu import assert_identical, gpu_run, oracle_run

pytestmark = pytest.mark.gpu


def _case(dtype, dims=(200, 152, 12)):
    g = S.gaussian_sum_gradient(dims[:2], dims[2], seed=3, n_blobs=40, sigma=(3, 9), dtype=dtype)
    return cases.Case("blobs", "regular", 2, cases.MULTI, g, 2.0 ** 20, list(dims))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [0, 1])
def test_modes(dtype, mode):
    case = _case(dtype)
    with api.Context(0) as c:
        c.set_option(api.OPT_CULL_MODE, mode)
        assert_identical(gpu_run(c, case), oracle_run(case))
        assert c.get_option(api.INFO_LAST_CULL_MODE) == mode
        assert c.get_option(api.INFO_LAST_TMA) == mode


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("plain", [0, 1])
def test_batch_staging(dtype, plain):
    some = [_case(dtype), _case(dtype, (64, 48, 5)), _case(dtype, (33, 20, 3))]
    keep: list = []
    with api.Context(0) as c:
        c.set_option(api.OPT_DISABLE_TMA, plain)
        got = c.extract_batch([api.regular_mesh_desc(x.local_dims) for x in some],
                              [api.field_desc(x.arrays, x.layout, 2, keep=keep) for x in some],
                              [api.params(x.sos_q) for x in some])
    for r, x in zip(got, some):
        assert_identical(r, oracle_run(x))


@pytest.mark.parametrize("graphs", [0, 1])
def test_bounded_wait_runs_out_in_strips(graphs):
    case = _case(np.float64, (64, 48, 5))
    with api.Context(0) as c:
        c.set_option(api.OPT_USE_GRAPHS, graphs)
        c.set_option(api.OPT_TEST_STALL_POLLS, 64)
        with pytest.raises(api.Ftk2bError) as e:
            gpu_run(c, case)
        assert e.value.status == api.TIMEOUT
        c.set_option(api.OPT_TEST_STALL_POLLS, 0)
        assert_identical(gpu_run(c, case), oracle_run(case))
        assert c.get_option(api.INFO_LAST_TMA) == 0
