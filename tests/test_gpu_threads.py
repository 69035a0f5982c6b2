"""Contexts of different sizes used by several host threads at once: their
kernels' instantiations are shared (the same FFT lengths, the same near-zone
kernels), the shared memory of their launches is not.  Every thread's matvecs
and solves have the bits of the context used alone."""
import threading

import numpy as np
import pytest

from scadyn_b200 import api
from tests.diag_operator import diagonal_solver, random_columns

pytestmark = pytest.mark.gpu


def test_contexts_of_other_sizes_in_other_threads():
    rng = np.random.default_rng(2)
    jobs = []
    # 40, 36 and 34 nodes an axis (length 80), groups of 2, 7 and 24 tets
    for tets, per_box in ((13000, 2), (30000, 7), (98000, 24)):
        lam = rng.uniform(1.0, 1.5, tets) + 1j * rng.uniform(-0.2, 0.2, tets)
        s = diagonal_solver(lam, per_box)
        mat = random_columns(9, s.n, seed=tets)
        kw = dict(tol=1e-6, m=20, cycles=2, want_x=True)
        want = [s.compute_Ax2(mat[0]), s.solve_columns(mat, block=9, **kw)[2],
                s.solve_columns(mat[:1], **kw)[2]]
        jobs.append((s, mat, kw, want))
    errors = []

    def work(s, mat, kw, want):
        try:
            for _ in range(4):
                for _ in range(40):
                    assert np.array_equal(s.compute_Ax2(mat[0]), want[0])
                assert np.array_equal(s.solve_columns(mat, block=9, **kw)[2], want[1])
                assert np.array_equal(s.solve_columns(mat[:1], **kw)[2], want[2])
        except BaseException as e:   # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, *_ in jobs:
        s.close()
    assert not errors, errors
