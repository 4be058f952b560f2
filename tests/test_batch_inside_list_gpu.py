"""A batch whose list of simplices inside by their ties alone is far longer than
its first capacity (65,536) while few or none of them solve: the call runs again
with room for the list, and gives what each field gives by itself."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_pack_gpu import _noise
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [1, 0])
@pytest.mark.parametrize("flat", [[[17, 15, 13, 3]], [[70, 60, 9], [14, 13, 12, 3]]])
def test_long_inside_list(flat, graphs):
    some = [cases.Case("flat", "regular", len(d) - 1, cases.MULTI, 1e-8 * _noise(d, 5), 2.0 ** 20, d) for d in flat]
    some.append(cases.Case("noise", "regular", 2, cases.MULTI, _noise([20, 19, 4], 6), 2.0 ** 20, [20, 19, 4]))
    want = [oracle_run(x) for x in some]
    keep: list = []
    with api.Context(0) as c:
        c.set_option(api.OPT_USE_GRAPHS, graphs)
        args = ([api.regular_mesh_desc(x.local_dims) for x in some],
                [api.field_desc(x.arrays, x.layout, x.ncomp, keep=keep) for x in some],
                [api.params(x.sos_q) for x in some])
        for _ in range(2):
            for r, w in zip(c.extract_batch(*args), want):
                assert_identical(r, w)
        assert c.get_option(api.INFO_LAST_TESTED) > 65536
