"""Which lattices under the pressure rewrite take several steps per launch: the
64-bit storages up to the sizes where their tiles still win, float32 beyond; the same
bits either way."""
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, _lib, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,nx,ny,tiled", [
    ("fx64", 200, 60, True), ("fx64", 118, 101, True), ("fx64", 300, 130, False), ("fx64", 515, 230, False),
    ("f64", 200, 60, True), ("f64", 267, 112, True), ("f64", 251, 132, False), ("f64", 458, 128, False),
    ("f32", 515, 230, True), ("f16", 515, 230, True)])
def test_pressure_lattices(storage, nx, ny, tiled):
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=nx)
    b = BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3)
    one = Lattice(nx, ny, 1.3, b, storage=storage, bc_inline=True, seed=3).set_state(f, rho, u).step(16)
    lat = Lattice(nx, ny, 1.3, b, storage=storage, seed=3).set_state(f, rho, u).step(1)
    _lib.launches(reset=True)
    lat.step(15)
    assert (_lib.launches() < 15) == tiled
    assert all(torch.equal(x, y) for x, y in zip(one.read(), lat.read()))
