"""scd_T_assemble_noalloc gives the bits of the T columns that scd_solve_columns
assembles from the same solutions, over the counts of splits (1, 3, 17, 64) and
of outputs whose splits fit the fixed scratch together, a few at a time or (more
than 131,072 outputs) not even two."""
import numpy as np
import pytest

from scadyn_b200 import api
from tests.diag_operator import diagonal_solver, random_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tets,ncol", [(100, 30), (3000, 130), (11000, 7), (11000, 64), (11000, 100),
                                       (600, 362), (600, 363)])
def test_same_bits(tets, ncol):
    import torch
    lam = np.where(np.arange(tets) % 2, 1.0 + 0.1j, 2.0 - 0.3j)
    s = diagonal_solver(lam)
    mat = random_columns(ncol, s.n)
    Tc, _, X, _ = s.solve_columns(mat, block=32, tol=1e-8, m=10, want_x=True)
    n = s.n
    s.close()
    dev = torch.device("cuda:0")
    mat_d, X_d = torch.from_numpy(mat).to(dev), torch.from_numpy(X).to(dev)
    for ncb in (ncol, 5):
        T = torch.full((ncb, ncol), complex(np.nan, np.nan), dtype=torch.complex128, device=dev)
        api.T_assemble_noalloc(mat_d.data_ptr(), n, ncol, X_d.data_ptr(), ncb, T.data_ptr(),
                               torch.cuda.current_stream(dev).cuda_stream)
        torch.cuda.synchronize(dev)
        assert np.array_equal(T.cpu().numpy(), Tc[:ncb]), ncb
