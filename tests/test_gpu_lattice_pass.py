"""The boundary-node pass of a single lattice against the sources inside the step,
at sizes where the listed nodes are few enough for the pass to run (at most an
eighth of the lattice): in the body's launch, and as a second launch where a large
float32 lattice's boundary nodes are spread over it."""
import numpy as np
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, _lib, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300.geometry import BOUNCE

pytestmark = pytest.mark.gpu


def spread(every):
    def sources(nx, ny):
        m = np.zeros((nx, ny), dtype=bool)
        m[1::every, 2::5] = True
        m[0, : ny // 2] = True  # half of a side: no frame
        return [(m, i, BOUNCE, 0.001 * i) for i in (2, 5, 6)]
    return BU.Boundary([BU._Sources(sources)])


def boundary(kind, nx, ny):
    return {"cavity": lambda: BU.cavity_boundary_conditions(nx, ny, 0.1, 1.0),
            "channel": lambda: BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, 8, walls=True, plate_offset=1),
            "couette": lambda: BU.couette_flow_boundary_conditions(nx, ny, 0.05, 1.0),
            "poiseuille": lambda: BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3),
            "spread": lambda: spread(7)}[kind]()


@pytest.mark.parametrize("storage", ("f32", "f64", "fx64", "f16", "f16r"))
@pytest.mark.parametrize("kind", ("cavity", "channel", "couette", "poiseuille", "spread"))
@pytest.mark.parametrize("nx,ny", [(67, 54), (150, 91), (517, 70)])
def test_pass_runs(storage, kind, nx, ny):
    b = boundary(kind, nx, ny)
    assert 8 * b.geometry(nx, ny).n_special <= nx * ny
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=nx)
    kw = dict(storage=storage, seed=5, dev_ref=(0.05, 0.0) if storage == "f16r" else None)
    one = Lattice(nx, ny, 1.3, b, bc_inline=True, **kw).set_state(f, rho, u).step(8)
    other = Lattice(nx, ny, 1.3, b, bc_inline=False, **kw).set_state(f, rho, u).step(1)
    _lib.launches(reset=True)
    other.step(7)
    assert _lib.launches() == (7 if storage == "f32" else 14)
    assert all(torch.equal(x, y) for x, y in zip(one.read(), other.read()))
    assert torch.equal(one.aux[one.cur], other.aux[other.cur])


@pytest.mark.parametrize("asked", (None, False))
def test_large_lattice_with_spread_nodes(asked):
    nx, ny = 8209, 4100  # just above 2^25
    b = spread(101)
    assert nx * ny >= 1 << 25 and 8 * b.geometry(nx, ny).n_special <= nx * ny
    w = torch.tensor([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4, dtype=torch.float64, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    f = w * (1 + 0.01 * torch.rand((nx, ny, 9), dtype=torch.float64, device="cuda", generator=gen))
    lats = [Lattice(nx, ny, 1.3, b, storage="f32", bc_inline=inline).set_state(f).step(1) for inline in (True, asked)]
    _lib.launches(reset=True)
    lats[1].step(3)
    assert _lib.launches() == 6
    lats[0].step(3)
    assert all(torch.equal(x, y) for x, y in zip(lats[0].read(), lats[1].read()))


@pytest.mark.parametrize("storage,launches", [("f16r", 2), ("bf16r", 2), ("f16", 1)])
def test_reference_shifted_storages_from_2_22_nodes(storage, launches):
    nx, ny = 2051, 2047
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=3)
    b = boundary("channel", nx, ny)
    kw = dict(storage=storage, seed=5, dev_ref=(0.05, 0.0) if storage.endswith("r") else None)
    lats = [Lattice(nx, ny, 1.3, b, bc_inline=inline, **kw).set_state(f, rho, u).step(1) for inline in (True, None)]
    _lib.launches(reset=True)
    lats[1].step(2)
    assert _lib.launches() == 2 * launches
    lats[0].step(2)
    assert all(torch.equal(x, y) for x, y in zip(lats[0].read(), lats[1].read()))


@pytest.mark.parametrize("storage", ("f16r", "bf16"))
def test_spread_nodes_stay_inside_at_this_size(storage):
    nx, ny = 2051, 2047
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=3)
    kw = dict(storage=storage, seed=5, dev_ref=(0.05, 0.0) if storage.endswith("r") else None)
    lat = Lattice(nx, ny, 1.3, spread(40), **kw).set_state(f, rho, u).step(1)
    _lib.launches(reset=True)
    lat.step(2)
    assert _lib.launches() == 2
    one = Lattice(nx, ny, 1.3, spread(40), bc_inline=True, **kw).set_state(f, rho, u).step(3)
    assert all(torch.equal(x, y) for x, y in zip(lat.read(), one.read()))
