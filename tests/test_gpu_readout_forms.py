"""The read-out of the 64-bit storages on both sides of the sizes from which it goes
through shared memory, at widths and heights that leave partial tiles (32 x 8
nodes), with and without the populations: the bits of the oracle in exact float64,
1e-12 in fixed point (its float64 gate)."""
import numpy as np
import pytest

from lattice_boltzmann_parallel_solver_gb300 import Lattice
from lattice_boltzmann_parallel_solver_gb300 import lattice_boltzmann_method as L
from oracle import lbm_oracle as O

pytestmark = pytest.mark.gpu


def start(nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    rho = rng.uniform(0.98, 1.02, (nx, ny))
    u = rng.uniform(-0.02, 0.02, (nx, ny, 2))
    return O.equilibrium(rho, u), rho, u


@pytest.mark.parametrize("nx,ny", [(31, 2114), (32, 2048), (33, 1987), (2113, 31), (255, 257), (1031, 128), (129, 1017), (4099, 33)])
def test_forms_match_the_oracle(nx, ny):
    f, rho, u = start(nx, ny)
    ref = O.run(f, rho, u, 1.3, 2)
    exact = Lattice(nx, ny, 1.3, storage="f64", exact=True).set_state(f, rho, u).step(2)
    for got, want in zip(exact.read(), ref):
        assert np.array_equal(got.cpu().numpy(), want)
    for got, want in zip(exact.moments(), ref[1:]):
        assert np.array_equal(got.cpu().numpy(), want)
    fx = Lattice(nx, ny, 1.3).set_state(f, rho, u).step(2)
    for got, want in zip(fx.read(), ref):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
    for got, want in zip(L.lattice_boltzmann_step(f, rho, u, 1.3), O.run(f, rho, u, 1.3, 1)):
        assert np.array_equal(got, want)


def test_moments_of_a_large_lattice():
    nx, ny = 2051, 1027  # above 2^21 nodes
    f, rho, u = start(nx, ny)
    exact = Lattice(nx, ny, 1.3, storage="f64", exact=True).set_state(f, rho, u).step(1)
    for got, want in zip(exact.moments(), exact.read()[1:]):
        assert np.array_equal(got.cpu().numpy(), want.cpu().numpy())
    for got, want in zip(exact.moments(), O.run(f, rho, u, 1.3, 1)[1:]):
        assert np.array_equal(got.cpu().numpy(), want)
