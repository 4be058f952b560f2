"""Stream checkpoints say which form their content hash has: unstructured blobs
are version 2, regular ones (which hold no hash) version 1; both versions with
either hash are read, others refused."""
import struct

import numpy as np
import pytest

from ftk2_b200 import api
import test_stream_gpu as ts

pytestmark = pytest.mark.gpu


def _with_version(blob, v):
    return blob[:8] + struct.pack("<I", v) + blob[12:]


def _version(blob):
    return struct.unpack_from("<I", blob, 8)[0]


def test_unstructured_versions(ctx):
    case = ts._ext_cases()[2]
    keep: list = []
    nv, nt = case.coords.shape[0], case.n_layers + 1
    mesh = api.extruded_mesh_desc(nv, case.cells, case.n_layers, keep)
    step = lambda t: api.field_desc([np.ascontiguousarray(a[t * nv:(t + 1) * nv]) for a in case.arrays], case.layout,
                                    case.ncomp, keep=keep)
    with api.Stream(ctx, mesh, step(0), api.params(case.sos_q)) as st:
        st.push(step(0))
        blob = st.checkpoint()
    assert _version(blob) == 2
    want = ts.ext_one_shot(ctx, case, nt)
    for v in (1, 2):
        with api.Stream.restore(ctx, _with_version(blob, v)) as st:
            for t in range(1, nt):
                st.push(step(t))
            ts.assert_identical(st.result(), want)
    for v in (0, 3):
        with pytest.raises(api.Ftk2bError):
            api.Stream.restore(ctx, _with_version(blob, v))


def test_regular_blobs_stay_version_1(ctx):
    case = ts._cases()[0]
    keep: list = []
    fld = api.field_desc(ts.steps_of(case, 0), case.layout, case.ncomp, keep=keep)
    with api.Stream(ctx, api.regular_mesh_desc(case.local_dims), fld, api.params(case.sos_q)) as st:
        st.push(fld)
        blob = st.checkpoint()
        one = st.result()
    assert _version(blob) == 1
    with api.Stream.restore(ctx, blob) as st:
        ts.assert_identical(st.result(), one)
