"""The first matvec of an operator finds what it needs laid out at set-up: it
allocates no device memory, for operators built on the device and handed over
by the host, and for a wavenumber that follows another; its bits are the next
one's."""
import numpy as np
import pytest

from scadyn_b200 import api, meshgen
from tests.diag_operator import diagonal_solver

pytestmark = pytest.mark.gpu


def _device():
    mesh = meshgen.sphere(9.0, seed=2, eps=2.1 + 0.05j)
    s = api.Solver.from_desc(api.grid_from_mesh(mesh.coord, mesh.etopol, grid_size=2.0))
    s.set_mesh(mesh.coord, mesh.etopol, mesh.param)
    for k in (0.8, 1.0):
        s.set_wavenumber(k / mesh.a)
        s.build_G()
        s.pfft_projection_const()
        s.compute_near_zone_interactions_const()
    return s


def _host():
    return diagonal_solver(np.linspace(1.0, 1.5, 30000) + 0.1j)


@pytest.mark.parametrize("make", [_device, _host])
def test_first_matvec_allocates_nothing(make):
    import torch
    s = make()          # the kernels are loaded and have their local memory
    x = np.exp(1j * np.arange(s.n))
    s.compute_Ax2(x)
    s.close()
    s = make()
    free = torch.cuda.mem_get_info()[0]
    y = s.compute_Ax2(x)
    assert torch.cuda.mem_get_info()[0] == free
    assert np.array_equal(y, s.compute_Ax2(x))
    s.close()
