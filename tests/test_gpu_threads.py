"""Two lattices of one storage and different sizes stepped by two host threads on
two streams: each ends as it does alone (their several-steps launches share a
kernel and ask for different amounts of shared memory)."""
import threading

import pytest
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice, scenarios

pytestmark = pytest.mark.gpu

SIZES = ((300, 200), (200, 150), (64, 64))


def lattice(n, storage):
    nx, ny = SIZES[n]
    f, rho, u = scenarios.von_karman_start(nx, ny, u_in=0.05, noise=1e-2, seed=n)
    return Lattice(nx, ny, 1.3, None, storage=storage, seed=n).set_state(f, rho, u)


@pytest.mark.parametrize("storage", ("fx64", "f32"))
def test_lattices_in_two_threads(storage):
    rounds, steps = 60, 150
    alone = [lattice(n, storage).step(1 + rounds * steps).read()[0] for n in range(len(SIZES))]
    lats = [lattice(n, storage).step(1) for n in range(len(SIZES))]
    torch.cuda.synchronize()
    errors, go = [], threading.Barrier(len(SIZES))

    def work(lat):
        try:
            s = torch.cuda.Stream()
            go.wait(60)
            with torch.cuda.stream(s):
                for _ in range(rounds):
                    lat.step(steps)
            s.synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(lat,)) for lat in lats]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    assert all(torch.equal(a, lat.read()[0]) for a, lat in zip(alone, lats))
