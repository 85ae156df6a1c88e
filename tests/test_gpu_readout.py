"""The read-out at the edges of its tiles (32 x 8 nodes): sizes below, at and above
a tile's sides, every storage that goes through shared memory, against the NumPy
oracle, with and without the populations, and the host step's ranges of columns."""
import numpy as np
import pytest

from lattice_boltzmann_parallel_solver_gb300 import Lattice
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300 import lattice_boltzmann_method as L
from oracle import lbm_oracle as O

pytestmark = pytest.mark.gpu


def start(nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    rho = rng.uniform(0.98, 1.02, (nx, ny))
    u = rng.uniform(-0.02, 0.02, (nx, ny, 2))
    return O.equilibrium(rho, u), rho, u


@pytest.mark.parametrize("nx,ny", [(3, 3), (31, 7), (32, 8), (33, 9), (64, 1), (5, 65), (97, 23)])
def test_read_matches_the_oracle(nx, ny):
    f, rho, u = start(nx, ny)
    ref = O.run(f, rho, u, 1.3, 3)
    exact = Lattice(nx, ny, 1.3, storage="f64", exact=True).set_state(f, rho, u).step(3)
    for got, want in zip(exact.read(), ref):
        assert np.array_equal(got.cpu().numpy(), want)
    assert exact.read(want_f=False)[0] is None
    for got, want in zip(exact.moments(), ref[1:]):
        assert np.array_equal(got.cpu().numpy(), want)
    fx = Lattice(nx, ny, 1.3).set_state(f, rho, u).step(3)
    for got, want in zip(fx.read(), ref):
        # the float64 gate of the fixed-point storage
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("slabs", [1, 2, 3, 7])
def test_host_step_column_ranges(slabs):
    nx, ny = 100, 21
    f, rho, u = start(nx, ny)
    bnd = BU.couette_flow_boundary_conditions(nx, ny, 0.05, 1.0)
    got = L._step_host(bnd.geometry(nx, ny), f, rho, u, 1.1, 1, 0, slabs=slabs)
    for a, b in zip(got, O.run(f, rho, u, 1.1, 1, O.couette_boundary(nx, ny, 0.05, 1.0))):
        assert np.array_equal(a, b)
