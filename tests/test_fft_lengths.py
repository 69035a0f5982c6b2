"""Every length of the fused y-z FFT pass: on the host, the pass against a
direct convolution (tests/fft_lengths_check.cu); on the GPU, the matvec of a
host operator on grids that select each length, fused, with three passes and
with powers of two, against numpy's FFTs."""
import os
import subprocess

import numpy as np
import pytest

from tests.test_fft_yz import CSRC

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_length_on_the_host(tmp_path):
    exe = str(tmp_path / "fft_lengths_check")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-I", CSRC,
                           os.path.join(HERE, "fft_lengths_check.cu"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _operator(n, T=40, seed=1):
    """A host operator with interpolation-sized projector weights at random boxes of an n grid and a unit near zone."""
    rng = np.random.default_rng(seed)
    nc = (np.array(n) - 2) // 2
    cube = rng.integers(0, nc, (T, 3))
    cube[0], cube[1] = 0, nc - 1
    first = 2 * cube[:, 0] + n[0] * (2 * cube[:, 1] + n[1] * 2 * cube[:, 2])
    j = np.arange(27)
    indS = (first[:, None] + j % 3 + n[0] * (j // 3 % 3 + n[1] * (j // 9)) + 1).astype(np.int32)
    P = [rng.standard_normal((T, 27)) + 1j * rng.standard_normal((T, 27)) for _ in range(4)]
    return P, indS, np.tile(np.eye(3, dtype=np.complex64), (T, 1, 1)), np.stack([np.arange(T)] * 2, 1).astype(np.int32) + 1


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(8, 10, 16), (18, 20, 12), (20, 18, 22), (24, 22, 32), (26, 30, 40), (40, 44, 48),
                               (42, 54, 26), (56, 50, 20), (64, 58, 18), (96, 70, 30), (12, 96, 66), (100, 8, 24)])
def test_grids_of_every_length(n):
    from scadyn_b200 import api
    from tests import np_restate
    P, indS, sp, ind = _operator(n)
    T = len(indS)
    G = np_restate.build_G(*n, 1.0, np.zeros(3), 0.3)
    rng = np.random.default_rng(n[0])
    x = rng.standard_normal(3 * T) + 1j * rng.standard_normal(3 * T)
    want = np_restate.compute_Ax2(x, *P, indS, G.transpose(2, 1, 0), sp, ind, 0.3, *n, merged=True)
    for kw in (dict(), dict(fft_passes=api.FFT_PASSES_THREE), dict(fft_lengths=api.FFT_POW2)):
        s = api.Solver(*n, 1.0, (0.0, 0.0, 0.0), T, **kw)
        s.set_wavenumber(0.3)
        s.set_projectors(*P, indS)
        s.build_G()
        s.set_nearzone(sp, ind)
        y = s.compute_Ax2(x)
        s.close()
        # three FFT pairs of at most 512 points and 27-term sums: some tens of roundings of 1.1e-16
        assert np.linalg.norm(y - want) / np.linalg.norm(want) < 1e-13, kw
