"""The Arnoldi tick on both sides of 524,288 unknowns, where its chunks grow
beyond 256 elements (2,048 of them, then fewer of 512): FP64 modified
Gram-Schmidt, and the mixed form with classical and modified Gram-Schmidt, solve
a diagonal operator, and every column has the same bits alone and in a batch."""
import numpy as np
import pytest

from scadyn_b200 import api
from tests.diag_operator import diagonal_solver, random_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tets", [174762, 174763])
def test_long_vectors(tets):
    rng = np.random.default_rng(1)
    lam = rng.uniform(0.8, 1.2, tets) + 1j * rng.uniform(-0.1, 0.1, tets)
    s = diagonal_solver(lam, per_box=24)
    mat = random_columns(3, s.n)
    want = mat / np.repeat(lam, 3)
    for precision, gs, tol in ((api.PREC_FP64, api.GS_DEFAULT, 1e-8), (api.PREC_MIXED, api.GS_CLASSICAL, 1e-11),
                               (api.PREC_MIXED, api.GS_MODIFIED, 1e-11)):
        kw = dict(tol=tol, m=20, cycles=4, precision=precision, gram_schmidt=gs, inner_tol=1e-4, want_x=True)
        _, it, X, rc = s.solve_columns(mat, block=3, **kw)
        assert rc == api.SCD_OK and (it > 1).all()
        # |x - b/lambda| <= |residual| / min |lambda|
        assert (np.linalg.norm(X - want, axis=1) <= tol / 0.8 * np.linalg.norm(mat, axis=1)).all()
        _, it1, X1, _ = s.solve_columns(mat, block=1, **kw)
        assert np.array_equal(it1, it) and np.array_equal(X1, X)
    s.close()
