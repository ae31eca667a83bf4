"""Kinetic energy of mixed resident runs: formed from the FP64 velocities of the
last update, as in a batch (which runs the per-phase kernels), however the run
ends.  Both sum the same terms in another order.  Only one element moves, so 24
terms are not zero and the bound is that of 23 additions of positive terms on
either side; velocities of the stored 40 bits would be off by about 1e-13.

The meshes are disjoint elements: the one-cluster form with one and with two
nodes per thread, and the grid form with two nodes per thread and several such
groups per thread."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = [1, 31, 250, 600, 9600]


def separate_elements(ne):
    from enscdynamics_b200 import mesh as M
    one = M.box_mesh(1, 1, 1, 0.01, 0.01, 0.01)
    at = 0.02 * np.arange(ne)[:, None, None] * np.array([1.0, 0.0, 0.0])
    x0 = (one.x0[None] + at).reshape(-1, 3)
    conn = (one.conn.reshape(1, 8) + 8 * np.arange(ne)[:, None]).astype(np.uint32)
    v0 = np.zeros(x0.shape)
    v0[-8:] = np.random.default_rng(7).normal(0.0, 1.0, (8, 3))
    return x0, conn, v0


@pytest.mark.parametrize("ne", MESHES)
@pytest.mark.parametrize("stop", ["cycles", "end", "pause"])
def test_kinetic_energy_equals_the_batch(ne, stop):
    from enscdynamics_b200 import capi
    from enscdynamics_b200 import mesh as M
    x0, conn, v0 = separate_elements(ne)
    code, val = np.zeros(x0.shape, dtype=np.int8), np.zeros(x0.shape)
    m, c = M.Material(70e9, 0.33, 2700.0), M.Controls()
    with capi.Stepper(x0, conn, v0, material=m, controls=c, precision=capi.MIXED) as s:
        s.set_bcs(code, val)
        dt = s.step(1)["dt_i"]
        rep = {"cycles": lambda: s.step(4), "end": lambda: s.step(99, 3.6 * dt),
               "pause": lambda: s.step_until(99, math.inf, 3.6 * dt)}[stop]()
        assert rep["status"] == 0 and 4 <= rep["total_cycles"] <= 6 and s.kernels_per_cycle == 0
        e = s.energy()
    with capi.Batch(max_instances=1, max_elements=ne, max_nodes=8 * ne, budget_bytes=1 << 30,
                    precision=capi.MIXED) as b:
        sl = b.add(x0, conn, v0, material=m, controls=c)
        b.set_bcs(sl, code, val)
        b.arm(sl, rep["total_cycles"], 3.6 * dt if stop == "end" else math.inf)
        b.run(rep["total_cycles"])
        b.sync()
        assert b.report(sl)["time"] == rep["time"]
        ref = b.energy(sl)
    assert e["kinetic"] > 0.0
    assert abs(e["kinetic"] - ref["kinetic"]) <= 2 * 23 * 2.0 ** -53 * ref["kinetic"]
