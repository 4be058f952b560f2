"""Batches of different sizes on threads of their own: the shared memory limit
of their star-edge kernel belongs to the kernel, not to the call."""
import threading

import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 60), (3, 200)])
def test_two_batches_at_once(sizes):
    f = 1.0 + np.zeros((3, 8, 8, 2))
    f[:, 2:6, 2:6] = np.random.default_rng(2).standard_normal((3, 4, 4, 2))
    case = cases.Case("patch", "regular", 2, cases.MULTI, f, 2.0 ** 20, [8, 8, 3])
    want = oracle_run(case)
    errors = []

    def work(n):
        try:
            import torch
            keep: list = []
            fld = api.field_desc(torch.from_numpy(f).cuda(), api.LAYOUT_MULTICOMPONENT, 2, keep=keep)
            torch.cuda.synchronize()
            args = ([api.regular_mesh_desc(case.local_dims)] * n, [fld] * n, [api.params(case.sos_q)] * n)
            with api.Context(0) as ctx:
                ctx.set_option(api.OPT_USE_GRAPHS, 0)
                for _ in range(400):
                    r = ctx.extract_batch(*args)
                    assert_identical(r[-1], want)
        except Exception as e:  # seen by the main thread
            errors.append(e)

    th = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
