"""Refused kernel launches of a matvec and a T assembly without memory are
reported (tests/launch_status_check.cu, tests/t_assemble_status_check.cu)."""
import glob
import os
import subprocess

import pytest

from scadyn_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("check", ["launch_status_check", "t_assemble_status_check"])
def test_failures_are_reported(tmp_path, check):
    build.build()
    exe = tmp_path / check
    objs = sorted(glob.glob(os.path.join(build.HERE, "_build", "*.o")))
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                           os.path.join(HERE, check + ".cu"), *objs, "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    if r.returncode == 77:
        pytest.skip("needs a machine without a device")
    assert r.returncode == 0, r.stdout + r.stderr
