"""Host memory functions of the C library when no memory is left (no GPU): see
cpp/host_memory_check.cpp, which replaces operator new for the whole process."""
import os
import shutil
import subprocess

import pytest

from ftk2_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_memory(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    build.build()
    cuda = os.path.dirname(os.path.dirname(nvcc))
    exe = str(tmp_path / "host_memory_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "host_memory_check.cpp"), "-o", exe, "-L", build.OUT_DIR,
                    "-lftk2b", "-Wl,-rpath," + build.OUT_DIR, "-L", os.path.join(cuda, "lib64"), "-lcudart"],
                   check=True)
    env = dict(os.environ, LD_LIBRARY_PATH=os.path.join(cuda, "lib64") + ":" + os.environ.get("LD_LIBRARY_PATH", ""))
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
