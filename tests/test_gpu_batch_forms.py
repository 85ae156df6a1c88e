"""The form a batched step takes follows the storage, the batch's nodes in total
and where its boundary nodes lie, and every form gives the bits of the step with
the sources inside its tiles: the boundary-node pass as a launch of its own (two
launches a step) or in the body's launch (one), with probes on nodes the pass
records."""
import functools

import numpy as np
import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import _lib, scenarios
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300.batch import Batch, Member
from lattice_boltzmann_parallel_solver_gb300.geometry import BOUNCE

pytestmark = pytest.mark.gpu

STEPS = 6


def boundary(kind, nx, ny):
    if kind == "channel":
        return BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, max(6, ny // 5 // 2 * 2), walls=True, plate_offset=1)
    if kind == "poiseuille":
        return BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3)
    if kind == "periodic":
        return None

    def half(nxx, nyy):  # half of a side: no frame
        m = np.zeros((nxx, nyy), dtype=bool)
        m[0, : nyy // 2] = True
        return [(m, i, BOUNCE, 0.001 * i) for i in (2, 5, 6)]
    return BU.Boundary([BU._Sources(half)])


@functools.lru_cache(maxsize=8)
def start(nx, ny, seed):
    return scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=seed)


def members(kinds, sizes, storage):
    out = []
    for j, (nx, ny) in enumerate(sizes):
        f, rho, u = start(nx, ny, j % 4)
        kind = kinds[j % len(kinds)]
        # a wall, a pressure column and an inlet corner: nodes of the pass
        probe = {"channel": (nx // 3, 0), "poiseuille": (nx - 2, ny // 2), "half": (0, 1)}.get(kind, (1, 1))
        out.append(Member(nx, ny, 1.2, boundary(kind, nx, ny), steps=STEPS + 1, probe=probe, f0=f, rho0=rho, u0=u, seed=j,
                          dev_ref=(0.05, 0.0) if storage.endswith("r") else None))
    return out


def check(storage, kinds, sizes, launches, least, blocks=None):
    """``launches`` a step from ``least`` nodes in total (the sizes hold at least that many)."""
    runs = []
    for inline in (True, None):
        b = Batch(members(kinds, sizes, storage), storage=storage, inline_bc=inline, blocks=blocks).start()
        assert b.nodes >= least
        _lib.launches(reset=True)
        b.run()
        if inline is None:
            assert _lib.launches() == launches * STEPS + 1  # and the step counter
        runs.append(b)
    for j in range(len(sizes)):
        assert all(torch.equal(x, y) for x, y in zip(runs[0].read(j), runs[1].read(j))), j
        assert torch.equal(runs[0].probe_trace(j), runs[1].probe_trace(j)), j
        assert runs[0].probe_trace(j).shape[0] == STEPS


MILLION = [(701, 301), (640, 410), (515, 511), (905, 365)]  # 2^20 and 18,315 more


@pytest.mark.parametrize("storage", ("f16", "bf16", "f16r", "bf16r"))
@pytest.mark.parametrize("blocks", (None, 0))
def test_pass_as_a_second_launch(storage, blocks):
    check(storage, ("channel", "poiseuille"), MILLION, 2, 1 << 20, blocks)


@pytest.mark.parametrize("storage,kinds,sizes,launches,least", [
    # members without a frame, on both sides of 2^21 nodes
    ("f32", ("channel", "half"), MILLION, 1, 1 << 20),
    ("f32", ("half", "channel"), 2 * MILLION, 2, 1 << 21),
    ("fx64", ("channel", "half"), MILLION, 1, 1 << 20),
    ("fx64", ("half", "poiseuille"), 2 * MILLION, 2, 1 << 21),
    ("f64", ("half", "poiseuille"), MILLION, 1, 1 << 20),
    # framed members, on both sides of 2^22 / 2^23
    ("fx64", ("channel", "poiseuille"), 2 * MILLION, 1, 1 << 21),
    ("fx64", ("channel", "poiseuille"), 4 * MILLION, 2, 1 << 22),
    ("f32", ("channel", "poiseuille"), 4 * MILLION, 1, 1 << 22),
    ("f32", ("channel", "poiseuille"), 8 * MILLION, 2, 1 << 23),
    # a few small members in the same launch; members without pass nodes in one
    ("f16", ("channel", "poiseuille", "periodic"), MILLION[:3], 1, 1 << 18),
    ("fx64", ("channel", "poiseuille", "periodic"), MILLION[:3], 1, 1 << 18),
    ("fx64", ("periodic",), 4 * MILLION, 1, 1 << 22),
    ("f32", ("periodic",), MILLION[:2], 1, 1 << 18),
    ("f16", ("periodic",), MILLION[:3], 1, 1 << 18)])
def test_form_by_size(storage, kinds, sizes, launches, least):
    check(storage, kinds, sizes, launches, least)


@pytest.mark.parametrize("storage", ("f16", "bf16r"))
@pytest.mark.parametrize("kinds", (("periodic",), ("half", "periodic")))
def test_narrow_member(storage, kinds):
    """A lattice too narrow for four nodes per thread in a batch of 2^18 to 2^20 nodes."""
    check(storage, kinds, [(5, 9000), (515, 511)], 1, 1 << 18)


@pytest.mark.parametrize("storage", ("f16", "bf16"))
@pytest.mark.parametrize("kinds,size,count,npt", [
    (("half",), (64, 700), 7, 2), (("channel", "half"), (200, 250), 6, 2), (("half",), (420, 180), 6, 4),
    (("channel",), (64, 700), 7, 4), (("periodic",), (64, 700), 7, 4)])
def test_shape_where_the_sources_stay_inside(storage, kinds, size, count, npt):
    """Members without a frame keep row-segment tiles: two nodes per thread where
    four would leave more lanes idle at the rows' ends."""
    b = Batch(members(kinds, [size] * count, storage), storage=storage).start()
    assert 1 << 18 <= b.nodes < 1 << 20
    assert b.npt == npt and (b.bc_chunks == -1) == ("half" in kinds)
