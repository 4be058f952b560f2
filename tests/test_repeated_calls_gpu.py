"""Calls that repeat and calls that do not: the first launch of a call, its
capture and its replays, arrays that take turns in numbers the context
remembers and does not, and arrays whose values change in place."""
import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


def _case(dims, seed):
    f = np.random.default_rng(seed).standard_normal(tuple(dims[::-1]) + (len(dims) - 1,))
    return cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, f, 2.0 ** 20, list(dims))


@pytest.mark.parametrize("count", [3, 16, 17, 20])
@pytest.mark.parametrize("fetch", [True, False])
def test_arrays_in_turn(count, fetch):
    import torch
    some = [_case([12, 11, 4], s) for s in range(count)]
    want = [oracle_run(x) for x in some]
    keep: list = []
    flds = [api.field_desc(torch.from_numpy(x.arrays).cuda(), x.layout, 2, keep=keep) for x in some]
    mesh = api.regular_mesh_desc([12, 11, 4])
    with api.Context(0) as c:
        for _ in range(3):
            for f, w in zip(flds, want):
                if fetch:
                    assert_identical(c.extract(mesh, f, api.params(2.0 ** 20)), w)
                else:
                    c.run(mesh, f, api.params(2.0 ** 20))
                    assert_identical(c.fetch(), w)


@pytest.mark.parametrize("dims", [[12, 11, 4], [7, 6, 5, 3], [60, 46, 5]])
def test_values_that_change_in_place(dims):
    import torch
    a = torch.empty(tuple(dims[::-1]) + (len(dims) - 1,), dtype=torch.float64, device="cuda")
    keep: list = []
    fld, mesh = api.field_desc(a, api.LAYOUT_MULTICOMPONENT, len(dims) - 1, keep=keep), api.regular_mesh_desc(dims)
    with api.Context(0) as c:
        for seed in range(4):
            x = _case(dims, seed)
            a.copy_(torch.from_numpy(x.arrays))
            torch.cuda.synchronize()
            assert_identical(c.extract(mesh, fld, api.params(2.0 ** 20)), oracle_run(x))
