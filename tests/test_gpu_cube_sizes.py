"""The matvec's anterpolation and interpolation over projection boxes of every
fill (a coarse grid with more tets per box than one stage of a kernel holds,
a fine one with nearly empty boxes) and over every right-hand-side count where
a kernel or a span changes: the FP64 matvec equals the oracle's, and every
column of a batched solve has the bits of the column solved alone."""
import numpy as np
import pytest

from oracle import oracle as O
from scadyn_b200 import api, meshgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1.2, 3.4, 4.4])
def problem(request):
    mesh = meshgen.ellipsoid(4.3, seed=11, eps=2.4 + 0.03j)
    k = 1.1 / mesh.a
    op = O.setup(mesh, k, grid_size=request.param, nthreads=0)
    g = op.geom
    s = api.Solver(g.Nx, g.Ny, g.Nz, g.delta, g.min_coord, g.T)
    s.set_wavenumber(k)
    s.set_projectors(op.S, op.Sx, op.Sy, op.Sz, op.indS)
    s.build_G()
    s.set_nearzone(op.sp_mat, op.sp_ind)
    rng = np.random.default_rng(5)
    mat = rng.standard_normal((35, s.n)) + 1j * rng.standard_normal((35, s.n))
    yield s, op, mat
    s.close()


def test_matvec_equals_oracle(problem):
    s, op, mat = problem
    y, yr = s.compute_Ax2(mat[0]), op.compute_Ax2(mat[0])
    assert np.linalg.norm(y - yr) / np.linalg.norm(yr) < 1e-11


@pytest.mark.parametrize("precision,block", [(api.PREC_FP64, b) for b in (2, 5, 7, 8, 17)] +
                         [(api.PREC_MIXED, b) for b in (3, 8, 20, 33)])
def test_batch_has_the_bits_of_one_column(problem, precision, block):
    s, _, mat = problem
    kw = dict(tol=1e-8, m=20, cycles=6, precision=precision, inner_tol=1e-3, want_x=True)
    one = s.solve_columns(mat[:block], block=1, **kw)
    many = s.solve_columns(mat[:block], block=block, **kw)
    assert np.array_equal(one[2], many[2]) and np.array_equal(one[1], many[1])
