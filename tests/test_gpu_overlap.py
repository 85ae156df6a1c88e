"""Steps whose launches overlap (programmatic dependent launch inside one call)
against the same steps one call at a time, where every launch is a plain one:
the same bits, for each storage, boundary form and the batch."""
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300.batch import Batch, Member

pytestmark = pytest.mark.gpu

STORAGES = ("fx64", "f64", "f32", "f16", "bf16r")


def channel(nx, ny, seed=0):
    return scenarios.von_karman(nx, ny, plate=max(6, ny // 5 // 2 * 2), seed=seed)


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("nx,ny,split", [(24, 20, None), (131, 77, False), (420, 180, None), (1500, 300, False)])
def test_lattice_steps_in_one_call(storage, nx, ny, split):
    f, rho, u, omega, bnd = channel(nx, ny)
    kw = dict(storage=storage, bc_inline=split, seed=3, probe=(nx // 2, ny // 2) if split is None else None, probe_cap=32)
    a = Lattice(nx, ny, omega, bnd, **kw).set_state(f, rho, u).step(21)
    b = Lattice(nx, ny, omega, bnd, **kw).set_state(f, rho, u)
    for _ in range(21):
        b.step(1)
    assert all(torch.equal(x, y) for x, y in zip(a.read(), b.read()))
    if a.probe is not None:
        assert torch.equal(a.probe_trace(), b.probe_trace())


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("inline", [True, False])
def test_batch_steps_in_one_call(storage, inline):
    def members():
        out = []
        for j, (nx, ny) in enumerate(((64, 40), (211, 97), (330, 128))):
            f, rho, u, omega, bnd = channel(nx, ny, seed=j)
            out.append(Member(nx, ny, omega, bnd, steps=12, probe=(nx // 2, ny // 2), f0=f, rho0=rho, u0=u, seed=j))
        p = BU.poiseuille_flow_boundary_conditions(60, 30, 1.001 / 3, 1 / 3)
        f, rho, u = scenarios.von_karman_start(60, 30, u_in=0.02)
        out.append(Member(60, 30, 1.1, p, steps=12, f0=f, rho0=rho, u0=u))
        return out
    for blocks in (None, 0):
        a = Batch(members(), storage=storage, inline_bc=inline, blocks=blocks).start().run()
        b = Batch(members(), storage=storage, inline_bc=inline, blocks=blocks).start()
        for _ in range(11):
            b.run(1)
        for j in range(4):
            assert all(torch.equal(x, y) for x, y in zip(a.read(j), b.read(j)))
            if a.members[j].probe is not None:
                assert torch.equal(a.probe_trace(j), b.probe_trace(j))
