"""A captured graph as the first use of a kernel in its process: float64 steps, which
ask for their kernel's resident blocks once, and a batch whose pass is a launch of its
own, against plain stepping."""
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu


def run(code):
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(code)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-1] == "same"


@pytest.mark.parametrize("kind", ("poiseuille", "channel", "periodic"))
def test_float64_lattice(kind):
    run("""
        import torch
        from lattice_boltzmann_parallel_solver_gb300 import Lattice, scenarios
        from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
        nx, ny, kind = 603, 162, "%s"
        b = {"poiseuille": lambda: BU.poiseuille_flow_boundary_conditions(nx, ny, 1.002 / 3, 1 / 3), "periodic": lambda: None,
             "channel": lambda: BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, 20, walls=True, plate_offset=1)}[kind]()
        state = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=1)
        a = Lattice(nx, ny, 1.3, b, storage="f64").set_state(*state).step_graph(31, chunk=10)
        c = Lattice(nx, ny, 1.3, b, storage="f64").set_state(*state).step(31)
        assert all(torch.equal(x, y) for x, y in zip(a.read(), c.read()))
        print("same")
        """ % kind)


@pytest.mark.parametrize("storage,count", [("f64", 4), ("f32", 34), ("fx64", 18)])
def test_batch(storage, count):
    run("""
        import torch
        from lattice_boltzmann_parallel_solver_gb300 import scenarios
        from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
        from lattice_boltzmann_parallel_solver_gb300.batch import Batch, Member
        nx, ny = 512, 500
        state = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=1)
        b = BU.von_karman_boundary_conditions(nx, ny, 1.0, 0.1, 20, walls=True, plate_offset=1)
        def batch():
            return Batch([Member(nx, ny, 1.0 + 0.01 * j, b, steps=22, f0=state[0], rho0=state[1], u0=state[2], probe=(9, 0))
                          for j in range(%d)], storage="%s").start()
        a, c = batch().run_graph(chunk=5), batch().run()
        for j in range(len(a.members)):
            assert all(torch.equal(x, y) for x, y in zip(a.read(j), c.read(j)))
            assert torch.equal(a.probe_trace(j), c.probe_trace(j))
        print("same")
        """ % (count, storage))
