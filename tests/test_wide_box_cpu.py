"""wide_box of a compiled geometry: whether its boundary nodes off the frame fill
more than an eighth of the lattice."""
import numpy as np
import pytest

from lattice_boltzmann_parallel_solver_gb300.geometry import BOUNCE, CompiledGeometry


def mask(nx, ny, *spans):
    m = np.zeros((nx, ny), dtype=bool)
    for xs, ys in spans:
        m[xs, ys] = True
    return m


EVERY = slice(None)


@pytest.mark.parametrize("name,spans,wide", [
    ("none", None, False), ("wall", [(EVERY, 0)], False), ("walls and plate", [(EVERY, 0), (EVERY, -1), (20, slice(10, 15))], False),
    ("half a side", [(0, slice(0, 10))], True), ("corners of the inside", [(1, 1), (62, 28)], True),
    ("an eighth", [(slice(10, 26), slice(5, 20))], False), ("a column more", [(slice(10, 27), slice(5, 20))], True)])
def test_wide_box(name, spans, wide):
    nx, ny = 64, 30  # 1920 nodes, an eighth of them 240 = 16 x 15
    sources = [] if spans is None else [(mask(nx, ny, *spans), 2, BOUNCE, 0.0)]
    assert CompiledGeometry(nx, ny, sources, device="cpu").wide_box == wide
