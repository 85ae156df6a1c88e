"""Where float64 steps overlap their launches: the rule (host code compiled alone)
against a small simulation of what it guards, the most blocks that one SM gets."""
import os
import random
import subprocess

from lattice_boltzmann_parallel_solver_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 152


def most_on_one_sm(blocks, slots):
    """Blocks of an overlapping launch that one SM may get: the free slots beside
    the launch before it, emptiest SM first, and if these do not take all of it,
    every slot of an SM that comes free."""
    loads = [blocks // SMS + (i < blocks % SMS) for i in range(SMS)]
    if blocks > slots * SMS:
        return None  # several waves: nothing is spread evenly to begin with
    free = sum(slots - n for n in loads)
    if free < blocks:
        return slots
    mine = [0] * SMS
    for _ in range(blocks):
        i = min(range(SMS), key=lambda j: loads[j] + mine[j])
        mine[i] += 1
    return max(mine)


def test_rule(tmp_path):
    rng = random.Random(1)
    cases = [(486, 5), (360, 4), (360, 5), (612, 5), (300, 3), (160, 3), (330, 3), (100, 1), (152, 1), (304, 2), (305, 2),
             (152, 2), (153, 2), (76, 1), (228, 3), (229, 3), (304, 3)]
    cases += [(rng.randint(1, 1200), rng.randint(1, 8)) for _ in range(60)]
    lib = _build.build()
    exe = str(tmp_path / "overlap")
    subprocess.check_call([_build._nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", _build.CSRC, "-o", exe,
                           os.path.join(HERE, "host", "overlap.cu"), lib, "-Xlinker", "-rpath=" + os.path.dirname(lib)])
    args = [str(v) for b, s in cases for v in (b, s, SMS)]
    got = [int(v) for v in subprocess.check_output([exe, *args], text=True).split()]
    for (b, s), pays in zip(cases, got):
        most = most_on_one_sm(b, s)
        even = -(-b // SMS)
        assert pays == (most is None or most <= even), (b, s, most, even)
