"""The fused y-z pass's shared-memory image ends where its last exchange line
does (tests/yz_image_check.cu)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "scadyn_b200", "csrc")


def test_image_ends_with_the_last_exchange_line(tmp_path):
    exe = tmp_path / "yz_image_check"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-I", CSRC,
                           os.path.join(HERE, "yz_image_check.cu"), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
