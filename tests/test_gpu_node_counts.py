"""A node count per thread that has no vectorised kernel falls back to the
one-node-per-thread kernel with the same boundary constants: the same bits as
``generic`` with the sources inside the step, and the vectorised agreement where a
separate launch recomputes the boundary nodes."""
import numpy as np
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU

pytestmark = pytest.mark.gpu

NX, NY = 96, 41


def boundary(kind):
    return {"cavity": lambda: BU.cavity_boundary_conditions(NX, NY, 0.1, 1.0),
            "channel": lambda: BU.von_karman_boundary_conditions(NX, NY, 1.0, 0.1, 8, walls=True, plate_offset=1),
            "couette": lambda: BU.couette_flow_boundary_conditions(NX, NY, 0.05, 1.0),
            "poiseuille": lambda: BU.poiseuille_flow_boundary_conditions(NX, NY, 1.002 / 3, 1 / 3)}[kind]()


@pytest.mark.parametrize("storage,npt", [("fx64", 3), ("fx64", 6), ("fx64", 8), ("f64", 1), ("f64", 8), ("f32", 8)])
@pytest.mark.parametrize("kind", ("cavity", "channel", "couette", "poiseuille"))
def test_count_without_a_kernel(storage, npt, kind):
    f, rho, u = scenarios.von_karman_start(NX, NY, u_in=0.05, noise=1e-2, seed=npt)
    b = boundary(kind)
    ref = Lattice(NX, NY, 1.3, b, storage=storage, generic=True).set_state(f, rho, u).step(9).read()
    got = Lattice(NX, NY, 1.3, b, storage=storage, npt=npt).set_state(f, rho, u).step(9).read()
    assert all(torch.equal(x, y) for x, y in zip(ref, got))
    assert 8 * b.geometry(NX, NY).n_special <= NX * NY
    got = Lattice(NX, NY, 1.3, b, storage=storage, npt=npt, bc_inline=False).set_state(f, rho, u).step(9).read()
    # the tolerances of vectorised against generic over 25 steps
    assert float((ref[0] - got[0]).abs().max() / ref[0].abs().max()) <= (1e-6 if storage == "f32" else 1e-13)
    assert np.isfinite(got[1].cpu().numpy()).all()
