"""FP64 Arnoldi steps that exhaust the Krylov space, where the step is
re-orthogonalised (||w|| falls by more than 1e-13): the solution is right and
every column has the same bits with w resident in shared memory, in any batch,
and with w streamed (64 columns of 118 chunks exceed the resident items, and
warps take items from a queue), run after run.  The space ends at an even or an odd step (the partial sums of
successive Gram-Schmidt terms alternate between two places), over several CTAs."""
import numpy as np
import pytest

from scadyn_b200 import api
from tests.diag_operator import diagonal_solver, random_columns

pytestmark = pytest.mark.gpu

T = 10000


@pytest.mark.parametrize("dims", [2, 3, 4])
def test_exhausted_krylov_space(dims):
    values = np.array([1.0 + 0.1j, 2.0 - 0.3j, 1.4 + 0.5j, 0.7 - 0.2j])[:dims]
    lam = values[np.arange(T) % dims]
    s = diagonal_solver(lam)
    mat = random_columns(64, s.n)
    kw = dict(tol=1e-8, m=10, cycles=2, precision=api.PREC_FP64, want_x=True)
    want = mat / np.repeat(lam, 3)
    _, it, X, _ = s.solve_columns(mat, block=64, **kw)
    assert (it == dims).all()
    # a residual of some 1e-14 |b|, |b| about 250
    assert np.abs(X - want).max() < 1e-11
    for _ in range(4):
        _, it1, X1, _ = s.solve_columns(mat, block=64, **kw)
        assert np.array_equal(it1, it) and np.array_equal(X1, X)
        for block in (1, 7, 16):
            _, it1, X1, _ = s.solve_columns(mat[:16], block=block, **kw)
            assert np.array_equal(it1, it[:16]) and np.array_equal(X1, X[:16]), block
    s.close()
