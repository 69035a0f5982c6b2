"""Refused kernel launches of a matvec are reported (tests/launch_status_check.cu)."""
import glob
import os
import subprocess

import pytest

from scadyn_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refused_launches_are_reported(tmp_path):
    build.build()
    exe = tmp_path / "launch_status_check"
    objs = sorted(glob.glob(os.path.join(build.HERE, "_build", "*.o")))
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                           os.path.join(HERE, "launch_status_check.cu"), *objs, "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    if r.returncode == 77:
        pytest.skip("needs a machine without a device")
    assert r.returncode == 0, r.stdout + r.stderr
