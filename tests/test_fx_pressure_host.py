"""The fixed-point pressure rewrite (fx::pressure_q in lbm_fx.cuh) compiled for
the host, against long double: within one unit of 2^-56 (half a unit from the
last rounding; the products before it carry three more bits and are off by less
than two of their units each) at small and large velocities and pressure
differences, and refused outside the range its products take."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    out = str(tmp_path_factory.mktemp("fxp") / "fx_pressure")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "fx_host", "fx_pressure.cpp"),
                           "-o", out])
    return out


@pytest.mark.parametrize("um,dr,least,most", [(1e-4, 1e-3, 20000, 20000), (0.05, 0.01, 20000, 20000),
                                              (0.17, 0.1, 19000, 20000), (0.17, 0.45, 5000, 19999), (0.9, 0.1, 1, 12000)])
def test_against_long_double(exe, um, dr, least, most):
    worst, accepted = subprocess.run([exe, "7", repr(um), repr(dr)], capture_output=True, text=True, check=True).stdout.split()
    assert float(worst) <= 1.0
    assert least <= int(accepted) <= most
