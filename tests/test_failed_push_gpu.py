"""A push whose cull reports an error (a bounded copy wait that ran out) leaves
the stream as it was: the step can be pushed again, or another in its place,
and the result is that of a stream that never saw the failed push.  The error
is made on the host: a library loaded first stands in for the cull's launcher
(cpp/failing_cull.cpp)."""
import os
import shutil
import subprocess
import sys

import pytest

from ftk2_b200 import build

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, os, sys
shim = ctypes.CDLL(sys.argv[1], ctypes.RTLD_GLOBAL)
import numpy as np
from ftk2_b200 import api, build
dims, nt = [int(v) for v in sys.argv[2].split("x")], 4
f = np.random.default_rng(3).standard_normal((nt + 1,) + tuple(dims[::-1]) + (len(dims),))
other = f[nt]
with api.Context(0) as ctx:
    assert shim.failing_cull_library(build.LIB.encode())
    mesh = api.regular_mesh_desc(dims + [1])
    keep = []
    step = lambda a: api.field_desc(np.ascontiguousarray(a), api.LAYOUT_MULTICOMPONENT, len(dims), keep=keep)
    results = []
    for fail_at in (None, 1, 2, 3):
        with api.Stream(ctx, mesh, step(f[0]), api.params(2.0 ** 20)) as st:
            for t in range(nt):
                if t == fail_at:
                    before = st.info()[:2]
                    shim.failing_cull_next(1)
                    try:
                        st.push(step(other))
                        raise SystemExit("the failed push was taken")
                    except api.Ftk2bError as e:
                        assert e.status == api.TIMEOUT, e
                    assert st.info()[:2] == before
                st.push(step(f[t]))
            results.append(st.result())
want = results[0]
assert want.n_tracks > 20, want.n_tracks
for got in results[1:]:
    assert got.n_tracks == want.n_tracks, (got.n_tracks, want.n_tracks)
    for k in ("simplices", "lam", "track_id", "edges"):
        assert np.array_equal(getattr(got, k), getattr(want, k)), k
print("ok")
"""


@pytest.mark.parametrize("dims", ["23x19", "9x8x7"])
def test_failed_push_leaves_no_trace(tmp_path, dims):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(nvcc))
    lib = str(tmp_path / "failing_cull.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "failing_cull.cpp"),
                    "-o", lib, "-L", os.path.join(cuda, "lib64"), "-lcudart", "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, lib, dims], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
