"""What the step calls launch, on the host alone: csrc/ensc_capi.cu compiled
against a fake CUDA runtime and fake kernels (tests/host/) that act on a control
block and partial sums in host memory.

- Every call runs its cycles, no more and no fewer: whole graphs, then up to half
  a graph's cycles one by one.
- A resident launch that the runtime refuses leaves the handle on the per-phase
  kernels with all cycles run and nothing of the earlier runs in the energies.
"""
import os
import subprocess

import pytest

from enscdynamics_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host") / "step_launches")
    cmd = [build.nvcc()] + build.ARCH + ["-std=c++17", "-O1", "--expt-relaxed-constexpr", "-cudart", "none",
                                         "-I" + build.INCLUDE, "-I" + build.CSRC,
                                         os.path.join(HERE, "host", "step_launches.cu"),
                                         os.path.join(HERE, "host", "fake_cudart.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    return [x.split() for x in out.stdout.splitlines()]


def test_a_call_is_whole_graphs_and_single_cycles(lines):
    rows = [tuple(map(int, x[1:])) for x in lines if x[0] == "split"]
    assert len(rows) == 38
    for chunk, n, cycles, graphs, singles, arms in rows:
        assert cycles == n and arms == 1, (chunk, n)
        rest = n % chunk
        one_by_one = 2 * rest <= chunk
        assert singles == (rest if one_by_one else 0), (chunk, n)
        assert graphs == n // chunk + (0 if one_by_one else 1), (chunk, n)


def test_resident_calls_run_their_cycles(lines):
    rows = [tuple(map(int, x[1:])) for x in lines if x[0] == "resident"]
    assert len(rows) == 4
    for n, cycles, runs, longest, graphs, singles in rows:
        assert cycles == n and graphs == 0 and singles == 0
        assert runs == -(-n // longest) and longest <= 4096


def test_a_refused_resident_launch_leaves_no_kinetic_energy_behind(lines):
    rows = [x[1:] for x in lines if x[0] == "refused"]
    assert len(rows) == 12
    for good, cycles, kinetic, internal, per_cycle in rows:
        n = 7 * int(good) + 40
        assert int(cycles) == n and int(per_cycle) == 4
        # 1 + cycles in three equal parts, added up: two roundings of the parts' sum
        assert abs(float(kinetic) - (1.0 + n)) <= 3 * 2.0 ** -52 * (1.0 + n)
        assert float(internal) == n
