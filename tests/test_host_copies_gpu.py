"""Host memory traffic by several threads: level-set results below the pinned
block's size, above it, and longer than the ring of pinned chunks; stream
checkpoints that hold the one-chain content hash."""
import numpy as np
import pytest

from ftk2_b200 import api
from oracle import contour_oracle
import test_stream_gpu as ts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[6, 5, 4, 3], [15, 14, 12, 5], [24, 22, 20, 4]])
def test_level_set_result_sizes(dims):
    f = np.random.default_rng(11).standard_normal(tuple(dims[::-1]))
    want = contour_oracle.contour(f, 0.0, dims, q=2.0 ** 20)
    with api.Context(0) as ctx:
        for _ in range(2):
            r = ctx.contour(api.regular_mesh_desc(dims), f, 0.0, 2.0 ** 20)
            for k in ("simplices", "lam", "bary", "track_id", "cells"):
                assert np.array_equal(getattr(r, k), want[k]), k
            assert not r.scalar.any()


def test_restore_takes_the_one_chain_hash(ctx):
    case = ts._ext_cases()[2]
    keep: list = []
    nv, nt = case.coords.shape[0], case.n_layers + 1
    mesh = api.extruded_mesh_desc(nv, case.cells, case.n_layers, keep)
    step = lambda t: [np.ascontiguousarray(a[t * nv:(t + 1) * nv]) for a in case.arrays]
    with api.Stream(ctx, mesh, api.field_desc(step(0), case.layout, case.ncomp, keep=keep),
                    api.params(case.sos_q)) as st:
        st.push(api.field_desc(step(0), case.layout, case.ncomp, keep=keep))
        blob = st.checkpoint()
    words = np.asarray(case.cells, dtype=np.uint64).ravel().tolist()
    mask = (1 << 64) - 1
    h = 0x9E3779B97F4A7C15 ^ len(words)
    for w in words:
        h ^= (w + 0x9E3779B97F4A7C15 + (h << 6) + (h >> 2)) & mask
        h = (h * 0xBF58476D1CE4E5B9) & mask
    at = blob.index(len(words).to_bytes(8, "little"), 64) + 8  # the hash follows the count
    old = blob[:at] + h.to_bytes(8, "little") + blob[at + 8:]
    assert old != blob
    with api.Stream.restore(ctx, old) as st:
        for t in range(1, nt):
            st.push(api.field_desc(step(t), case.layout, case.ncomp, keep=keep))
        ts.assert_identical(st.result(), ts.ext_one_shot(ctx, case, nt))
    with pytest.raises(api.Ftk2bError):
        api.Stream.restore(ctx, blob[:at] + (h ^ 1).to_bytes(8, "little") + blob[at + 8:])
