"""Resident runs on the paths that the size sweep of test_gpu_resident.py does
not reach: two nodes per thread with further groups of nodes per thread on a
grid, step calls of more cycles than one launch takes, and runs beside other
handles' kernels.  States are compared bit for bit.  Energies are sums of the
same terms in another order: 2e-12 of the energy that changes hands, at most
the kinetic energy at the start, leaves room for some 10,000 roundings of it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(dims, plastic=True):
    from enscdynamics_b200 import workloads as W
    return W.block(*dims, *(0.01 * d for d in dims), seed=sum(dims), plastic=plastic)


def stepper(p, precision):
    from enscdynamics_b200 import capi
    s = capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls,
                     precision=(capi.FP64, capi.MIXED)[precision])
    s.set_bcs(p.bc_code, p.bc_value)
    return s


def equal(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ne", [20000, 30001])
def test_more_nodes_than_the_grid_takes_at_once(ne, precision):
    """A row of elements has 4 nodes per element: more than two per thread."""
    from enscdynamics_b200 import capi
    p = problem((ne, 1, 1))
    with stepper(p, precision) as s:
        reps = [s.step(n) for n in (5, 7)]
        assert s.kernels_per_cycle == 0 and reps[-1]["total_cycles"] == 12 and reps[-1]["status"] == 0
        got, e = s.download(), s.energy()
    with capi.Batch(max_instances=1, max_elements=p.mesh.n_elements, max_nodes=p.mesh.n_nodes, budget_bytes=1 << 30,
                    precision=(capi.FP64, capi.MIXED)[precision]) as b:
        sl = b.add(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls)
        b.set_bcs(sl, p.bc_code, p.bc_value)
        b.arm(sl, 12)
        b.run(12)
        b.sync()
        equal(got, b.download(sl))
        ref = b.energy(sl)
    for k in e:
        assert abs(e[k] - ref[k]) <= 2e-12 * max(abs(ref[k]), e["kinetic0"]), k


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", [(5, 3, 3), (16, 16, 9)])
def test_a_call_of_several_launches(dims, precision):
    """One cluster, and a grid: 4100 cycles in one call and in four."""
    p = problem(dims, plastic=False)
    ends = []
    for calls in ((4100,), (1000, 1, 3000, 99)):
        with stepper(p, precision) as s:
            cycles = sum(s.step(n)["cycles"] for n in calls)
            rep = s.step(0)
            assert cycles == rep["total_cycles"] == 4100 and rep["status"] == 0 and s.kernels_per_cycle == 0
            ends.append((s.download(), (rep["time"], rep["dt_i"], rep["dt_i_1"], rep["dt_stable_min"]), s.energy()))
    equal(ends[0][0], ends[1][0])
    assert ends[0][1] == ends[1][1]
    a, b = ends[0][2], ends[1][2]
    for k in a:
        assert abs(a[k] - b[k]) <= 2e-12 * max(abs(b[k]), a["kinetic0"]), k


def test_beside_other_handles():
    """Two resident grids, a cluster run and a per-phase handle, each stepped by
    a thread of its own on its own stream."""
    jobs = [((41, 22, 21), 0), ((41, 22, 21), 1), ((20, 4, 4), 0), ((90, 60, 40), 1)]
    probs = [problem(d) for d, _ in jobs]
    alone = []
    for p, (_, precision) in zip(probs, jobs):
        with stepper(p, precision) as s:
            for _ in range(4):
                s.step(100)
            alone.append(s.download())
    hs = [stepper(p, precision) for p, (_, precision) in zip(probs, jobs)]
    assert [h.kernels_per_cycle for h in hs] == [0, 0, 0, 4]
    errors = []

    def run(h):
        try:
            for _ in range(4):
                assert h.step(100)["cycles"] == 100
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(h,)) for h in hs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for h, ref in zip(hs, alone):
        equal(h.download(), ref)
        h.close()
