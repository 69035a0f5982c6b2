"""The device-built near zone over the group sizes where its kernel's split of a
tile changes: boxes with one or two tets, groups between eight and sixteen, full
groups of 24 and boxes split into several groups, in complex128 against the
oracle's FP64 blocks; small and large kR (both methods of the Green function's
sine)."""
import numpy as np
import pytest

from oracle import oracle as O
from scadyn_b200 import api, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,ka", [(1.0, 1.0), (1.7, 2.0), (2.2, 1.0), (2.9, 30.0), (3.7, 1.0)])
def test_blocks_equal_oracle(cell, ka):
    mesh = meshgen.ellipsoid(2.7, seed=9, eps=2.25 + 0.01j)
    k = ka / mesh.a
    op = O.setup(mesh, k, grid_size=cell, nthreads=0, fp64_near=True)
    s = api.Solver.from_desc(api.grid_from_mesh(mesh.coord, mesh.etopol, grid_size=cell))
    s.set_wavenumber(k)
    s.set_mesh(mesh.coord, mesh.etopol, mesh.param)
    s.build_G()
    s.pfft_projection_const()
    s.compute_near_zone_interactions_const(api.STORE_C128)
    sp, ind = s.get_nearzone()
    s.close()
    order = np.lexsort((op.sp_ind[:, 1], op.sp_ind[:, 0]))
    assert np.array_equal(op.sp_ind[order], ind)
    want = op.sp_mat[order]
    # the parity bar of the device-built near zone (tests/test_gpu_setup.py)
    assert np.linalg.norm(sp - want) / np.linalg.norm(want) < 1e-9
