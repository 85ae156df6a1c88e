"""The boundary-node pass in blocks of the step's own launch against the sources
inside the step: the same bits for framed geometries, geometries whose sides mix
descriptors (no frame: the mask decides), inner obstacles at a row's ends, odd
widths, and the pressure rewrite with walls; single lattices in float32 (the
storage that takes it by default) and batches in every storage."""
import numpy as np
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300.batch import Batch, Member
from lattice_boltzmann_parallel_solver_gb300.geometry import BOUNCE

pytestmark = pytest.mark.gpu

KINDS = ("cavity", "channel", "couette", "poiseuille", "half side", "obstacles")


def boundary(kind, nx, ny):
    if kind == "cavity":
        return BU.cavity_boundary_conditions(nx, ny, 0.1, 1.0)
    if kind == "channel":
        return BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, max(6, ny // 5 // 2 * 2), walls=True, plate_offset=1)
    if kind == "couette":
        return BU.couette_flow_boundary_conditions(nx, ny, 0.05, 1.0)
    if kind == "poiseuille":
        return BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3)

    def sources(nxx, nyy):
        m = np.zeros((nxx, nyy), dtype=bool)
        if kind == "half side":  # part of the left column and of the bottom row
            m[0, : nyy // 2] = True
            m[: nxx // 3, 0] = True
        else:  # single nodes next to every side and at the ends of a chunk
            for x in (1, 2, 3, nxx // 2, nxx - 3, nxx - 2):
                m[x, 1::3] = True
        return [(m, i, BOUNCE, 0.001 * i) for i in (2, 5, 6)]
    return BU.Boundary([BU._Sources(sources)])


def start(nx, ny, seed):
    return scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=seed)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nx,ny", [(37, 24), (130, 61), (515, 40), (1030, 33)])
def test_lattice(kind, nx, ny):
    f, rho, u = start(nx, ny, nx)
    b = boundary(kind, nx, ny)
    one = Lattice(nx, ny, 1.3, b, storage="f32", bc_inline=True).set_state(f, rho, u).step(9)
    other = Lattice(nx, ny, 1.3, b, storage="f32", bc_inline=False).set_state(f, rho, u).step(9)
    assert all(torch.equal(x, y) for x, y in zip(one.read(), other.read()))
    assert torch.equal(one.aux[one.cur], other.aux[other.cur])


@pytest.mark.parametrize("storage", ("fx64", "f64", "f32", "f16", "bf16", "bf16r"))
@pytest.mark.parametrize("blocks", (None, 0))
def test_batch(storage, blocks):
    runs = []
    for inline in (True, False):
        members = []
        for j, kind in enumerate(KINDS):
            nx, ny = 60 + 37 * j, 24 + 11 * j
            f, rho, u = start(nx, ny, j)
            members.append(Member(nx, ny, 1.2, boundary(kind, nx, ny), steps=9 + j, probe=(nx - 1 - j % 2, j * 3), f0=f,
                                  rho0=rho, u0=u, seed=j))
        runs.append(Batch(members, storage=storage, inline_bc=inline, blocks=blocks).start().run())
    for j in range(len(KINDS)):
        assert all(torch.equal(x, y) for x, y in zip(runs[0].read(j), runs[1].read(j))), KINDS[j]
        assert torch.equal(runs[0].probe_trace(j), runs[1].probe_trace(j)), KINDS[j]
