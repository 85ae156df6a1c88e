"""The fixed-point boundary tables (set_fx_tables, host code compiled alone) equal
each constant converted by itself, for sets of numbers, of zeros of either sign and of
both."""
import os
import subprocess

from lattice_boltzmann_parallel_solver_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tables(tmp_path):
    lib = _build.build()
    exe = str(tmp_path / "fx_tables")
    subprocess.check_call([_build._nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", _build.CSRC, "-o", exe,
                           os.path.join(HERE, "host", "fx_tables.cu"), lib, "-Xlinker", "-rpath=" + os.path.dirname(lib)])
    assert subprocess.check_output([exe], text=True).split() == ["0"]
