"""The Arnoldi tick where its variants meet: FP64 solves of one column (w
resident in shared memory) and of enough columns that w streams from global
memory, and vectors of one chunk, of a ragged last chunk and of many, give
every column the same bits."""
import numpy as np
import pytest

from scadyn_b200 import api, geometry, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,ncol,precision", [
    (1.3, 6, api.PREC_FP64), (1.3, 6, api.PREC_MIXED),      # one chunk
    (2.6, 20, api.PREC_FP64), (2.6, 20, api.PREC_MIXED),    # a ragged last chunk
    (10.0, 48, api.PREC_FP64), (10.0, 40, api.PREC_MIXED),  # 295 chunks: 48 columns exceed the resident items
])
def test_columns_alone_and_together(radius, ncol, precision):
    mesh = meshgen.sphere(radius, seed=4, eps=2.1 + 0.05j)
    gs = max(2.0, geometry.cell_size_for_grid(mesh.coord, mesh.etopol, 26)) if radius > 5 else 2.0
    s = api.Solver.from_desc(api.grid_from_mesh(mesh.coord, mesh.etopol, grid_size=gs))
    s.set_wavenumber(1.5 / mesh.a)
    s.set_mesh(mesh.coord, mesh.etopol, mesh.param)
    s.build_G()
    s.pfft_projection_const()
    s.compute_near_zone_interactions_const()
    kw = dict(tol=1e-8, m=6, cycles=2, precision=precision, inner_tol=1e-3, max_outer=2)
    T, it = s.compute_T_matrix(4, ncol=ncol, block=ncol, **kw)
    cols = [0, ncol // 2, ncol - 1]
    T1, it1 = s.compute_T_columns(4, cols, block=1, **kw)
    s.close()
    assert np.isfinite(T).all()
    assert np.array_equal(T[:, cols], T1) and np.array_equal(it[cols], it1)
