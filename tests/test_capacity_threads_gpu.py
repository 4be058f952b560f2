"""Contexts of different feature capacities on threads of their own: the short
chain's shared memory limit belongs to the kernel, not to the call."""
import threading

import numpy as np
import pytest

from ftk2_b200 import api
import cases
from test_parity_gpu import assert_identical, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [0, 1])
def test_two_capacities_at_once(graphs):
    f = 1.0 + np.zeros((3, 12, 12, 2))
    f[:, 4:8, 4:8] = np.random.default_rng(2).standard_normal((3, 4, 4, 2))
    case = cases.Case("patch", "regular", 2, cases.MULTI, f, 2.0 ** 20, [12, 12, 3])
    want = oracle_run(case)
    assert 0 < len(want.track_id) < 1000
    errors = []

    def work(capacity):
        try:
            keep: list = []
            mesh, fld = cases.gpu_inputs(case, keep)
            with api.Context(0) as ctx:
                ctx.set_option(api.OPT_FEATURE_CAPACITY, capacity)
                for i in range(1500):
                    ctx.set_option(api.OPT_USE_GRAPHS, graphs)
                    r = ctx.extract(mesh, fld, api.params(case.sos_q))
                    if i % 100 == 0:
                        assert_identical(r, want)
        except Exception as e:  # seen by the main thread
            errors.append(e)

    th = [threading.Thread(target=work, args=(c,)) for c in (1000, 16384)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
