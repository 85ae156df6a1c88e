"""The frame of a compiled geometry (one descriptor per side and corner, the box
of the other boundary nodes) against its mask and descriptors."""
import numpy as np
import pytest

from lattice_boltzmann_parallel_solver_gb300.geometry import BOUNCE, CONST, OUTLET, CompiledGeometry


def rows(nx, ny, *ys):
    m = np.zeros((nx, ny), dtype=bool)
    m[:, list(ys)] = True
    return m


def cols(nx, ny, *xs):
    m = np.zeros((nx, ny), dtype=bool)
    m[list(xs), :] = True
    return m


def spot(nx, ny, xs, ys):
    m = np.zeros((nx, ny), dtype=bool)
    m[xs, ys] = True
    return m


def shapes(nx, ny):
    yield "empty", [], None
    yield "walls", [(rows(nx, ny, 0), 2, BOUNCE, 0.0), (rows(nx, ny, -1), 4, BOUNCE, 0.1)], True
    yield "box", [(cols(nx, ny, 0), 1, BOUNCE, 0.0), (cols(nx, ny, -1), 3, BOUNCE, 0.0), (rows(nx, ny, 0), 2, BOUNCE, 0.0),
                  (rows(nx, ny, -1), 4, BOUNCE, 0.2)], True
    yield "channel", [(cols(nx, ny, 0), i, CONST, 0.1 * i) for i in range(9)] + \
        [(cols(nx, ny, -1), 3, OUTLET, 0.0), (spot(nx, ny, slice(2, 4), slice(1, 3)), 1, BOUNCE, 0.0)], True
    yield "part of a side", [(spot(nx, ny, slice(1, nx // 2), 0), 2, BOUNCE, 0.0)], False
    yield "mixed side", [(rows(nx, ny, 0), 2, BOUNCE, 0.0), (spot(nx, ny, slice(1, 2), 0), 5, BOUNCE, 0.0)], nx <= 3
    yield "corner only", [(spot(nx, ny, 0, ny - 1), 8, BOUNCE, 0.0)], True
    yield "inner nodes to the edge", [(spot(nx, ny, slice(1, nx - 1), slice(1, ny - 1)), 6, BOUNCE, 0.0)], True


@pytest.mark.parametrize("nx,ny", [(5, 5), (6, 9), (33, 7), (64, 40)])
def test_frame_agrees_with_the_descriptors(nx, ny):
    for name, sources, framed in shapes(nx, ny):
        g = CompiledGeometry(nx, ny, sources, device="cpu")
        assert bool(g.struct.frame) == bool(framed), name
        if not framed:
            continue
        d = g.desc.numpy()
        f = list(g.struct.frame_desc)
        assert (d[0, 1:-1] == f[0]).all() and (d[-1, 1:-1] == f[1]).all()
        assert (d[1:-1, 0] == f[2]).all() and (d[1:-1, -1] == f[3]).all()
        assert [d[0, 0], d[0, -1], d[-1, 0], d[-1, -1]] == f[4:]
        x0, x1, y0, y1 = g.struct.inner_box
        inner = np.zeros((ny, nx), dtype=bool)
        if x0 <= x1:
            inner[y0:y1 + 1, x0:x1 + 1] = True
        assert not (d[1:-1, 1:-1].astype(bool) & ~inner[1:-1, 1:-1]).any()


def test_narrow_lattices_have_no_frame():
    for nx, ny in ((2, 9), (9, 2), (1, 5)):
        assert CompiledGeometry(nx, ny, [(rows(nx, ny, 0), 2, BOUNCE, 0.0)], device="cpu").struct.frame == 0
