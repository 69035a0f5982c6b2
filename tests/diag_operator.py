"""A host operator whose product is known: no grid part (zero projectors) and a
near zone of diagonal blocks lambda_t I, so that A x = lambda x and the Krylov
space of any right-hand side has as many dimensions as there are distinct
lambdas.  The tets lie in ascending boxes, so that slot order is the host's."""
import numpy as np

from scadyn_b200 import api


def diagonal_solver(lam, per_box=7, **choices):
    """Solver of A = diag(lam_t I_3), lam one complex value per tet."""
    T = len(lam)
    nc = 2
    while per_box * nc ** 3 < T:
        nc += 1
    N = 2 * nc + 2
    box = np.arange(T) // per_box
    cube = np.stack([box % nc, box // nc % nc, box // nc ** 2], 1)
    j = np.arange(27)
    first = 2 * cube[:, 0] + N * (2 * cube[:, 1] + N * 2 * cube[:, 2])
    indS = (first[:, None] + j % 3 + N * (j // 3 % 3 + N * (j // 9)) + 1).astype(np.int32)
    sp = np.zeros((T, 3, 3), np.complex128)
    sp[:, range(3), range(3)] = np.asarray(lam, np.complex128)[:, None]
    s = api.Solver(N, N, N, 1.0, (0.0, 0.0, 0.0), T, **choices)
    s.set_wavenumber(0.3)
    zero = np.zeros((T, 27), np.complex128)
    s.set_projectors(zero, zero, zero, zero, indS)
    s.build_G()
    s.set_nearzone(sp, np.stack([np.arange(T)] * 2, 1).astype(np.int32) + 1)
    return s


def random_columns(ncol, n, seed=3):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((ncol, n)) + 1j * rng.standard_normal((ncol, n))
