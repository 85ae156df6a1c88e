"""The interface's version follows its structs: the library's number is the
header's, and each number stands for one layout."""
import ctypes
import os
import re

from lattice_boltzmann_parallel_solver_gb300 import _build, _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# (sizeof lbm_geometry, sizeof lbm_batch_lattice, sizeof lbm_run_options) by version
SIZES = {10000: (2416, 112, 40), 10100: (2472, 112, 40)}


def test_version_stands_for_the_layout():
    _build.build()
    version = _lib.load().lbm_version()
    header = open(os.path.join(ROOT, "include", "lbm_gb300.h")).read()
    assert int(re.search(r"#define LBM_VERSION (\d+)", header).group(1)) == version
    assert SIZES[version] == tuple(ctypes.sizeof(c) for c in (_lib.Geometry, _lib.BatchLattice, _lib.RunOptions))
