"""Several steps per launch (small lattices, the default) against one step per
launch (``bc_inline=True``): the same bits in populations, moments, probe trace
and outlet memory, for every storage and boundary form, at sizes from one
partial tile to the largest that is tiled, narrow lattices whose halo wraps
round, odd sizes, and step counts that leave every remainder."""
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, _lib, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU

pytestmark = pytest.mark.gpu

STORAGES = ("fx64", "f64", "f32", "f16", "bf16", "f16r", "bf16r")


def boundary(kind, nx, ny):
    if kind == "couette":
        return BU.couette_flow_boundary_conditions(nx, ny, 0.05, 1.0)
    if kind == "poiseuille":
        return BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3)
    if kind == "cavity":
        return BU.cavity_boundary_conditions(nx, ny, 0.1, 1.0)
    if kind == "channel":
        return BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, max(6, ny // 5 // 2 * 2), walls=True, plate_offset=1)
    return None


def pair(kind, nx, ny, storage, steps, probe, graph=False):
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=nx * ny)
    kw = dict(storage=storage, seed=11, probe=probe, probe_cap=steps + 1)
    if storage.endswith("r"):
        kw["dev_ref"] = (0.05, 0.01)
    b = boundary(kind, nx, ny)
    one = Lattice(nx, ny, 1.4, b, bc_inline=True, **kw).set_state(f, rho, u).step(steps)
    _lib.launches(reset=True)
    many = Lattice(nx, ny, 1.4, b, **kw).set_state(f, rho, u)
    many.step_graph(steps, chunk=14) if graph else many.step(steps)
    launched = _lib.launches()
    assert one.cur == many.cur
    assert all(torch.equal(x, y) for x, y in zip(one.read(), many.read()))
    assert torch.equal(one.probe_trace(), many.probe_trace())
    assert torch.equal(one.aux[one.cur], many.aux[many.cur])
    return launched


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("kind,nx,ny", [
    ("periodic", 8, 5), ("periodic", 33, 47), ("couette", 20, 30), ("cavity", 31, 29), ("channel", 24, 22),
    ("channel", 131, 77), ("channel", 421, 181), ("poiseuille", 16, 21), ("poiseuille", 17, 40),
    ("poiseuille", 201, 60), ("cavity", 300, 255), ("channel", 60, 400)])
def test_steps_per_launch(storage, kind, nx, ny):
    probes = [(nx // 2, ny // 2), (0, ny - 1), (nx - 1, 1), (nx - 2, ny // 3), (1, ny // 2)]
    for n, steps in enumerate((4, 5, 6, 16, 22)):
        launched = pair(kind, nx, ny, storage, steps, probes[n])
        if nx * ny < 30000 and nx >= 40:
            assert launched < steps


@pytest.mark.parametrize("storage", ("f32", "f16", "bf16r"))
def test_largest_tiled(storage):
    assert pair("channel", 640, 410, storage, 12, (480, 205)) < 12


@pytest.mark.parametrize("storage", ("fx64", "f16"))
def test_replayed_from_a_graph(storage):
    pair("channel", 211, 98, storage, 1 + 3 * 14 + 5, (100, 50), graph=True)
