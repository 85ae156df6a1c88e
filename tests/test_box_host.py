"""The box of boundary nodes the kernels get (host code compiled alone): empty for
a lattice without boundary nodes, whether or not it comes with a frame, so that no
chunk of it is taken for one with nodes of the boundary-node pass; the frame's box;
the whole lattice for a mask without a frame."""
import os
import subprocess

from lattice_boltzmann_parallel_solver_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_box(tmp_path):
    lib = _build.build()
    exe = str(tmp_path / "box")
    subprocess.check_call([_build._nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", _build.CSRC, "-o", exe,
                           os.path.join(HERE, "host", "box.cu"), lib, "-Xlinker", "-rpath=" + os.path.dirname(lib)])
    rows = [tuple(int(v) for v in line.split())
            for line in subprocess.check_output([exe], text=True).splitlines()]
    assert len(rows) == 4
    for x0, x1, y0, y1, first, last in rows[:2]:
        assert x0 > x1 and y0 > y1 and first == last == 0
    assert rows[2] == (0, 7, 0, 5, 0, 0)
    assert rows[3] == (2, 4, 1, 3, 1, 8)
