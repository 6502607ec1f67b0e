"""The kernels' shared-memory opt-in (honei_b200/csrc/smem_opt_in.hh): per device, raised
and never lowered, safe between threads.  The helper runs here against a stand-in for the
CUDA calls; that a kernel goes through it is read from its source, since a second device
is what the plain call fails on."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "honei_b200", "csrc")


def test_helper(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "smem_opt_in_test")
    res = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-I", "/usr/local/cuda/include",
                          os.path.join(ROOT, "tests", "cpp", "smem_opt_in_test.cc"), "-o", exe, "-lpthread"],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout


def test_launches_go_through_the_helper():
    """The one other write of the limit would be a kernel that a second device refuses, or
    that one thread takes from another."""
    direct = [f for f in sorted(os.listdir(CSRC))
              if "cudaFuncAttributeMaxDynamicSharedMemorySize" in open(os.path.join(CSRC, f)).read()]
    assert direct == ["smem_opt_in.hh"]
