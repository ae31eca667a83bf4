"""Resident runs (one launch for all cycles of a small or medium mesh): the
FP64 state equals the CPU restatement bit for bit and the mixed state equals
the same solve in a batch (which runs the per-phase kernels), at the sizes
where the launch form changes -- one element, partial tiles, the largest
one-cluster mesh and the next size, a grid with one tile per warp, several
tiles per warp, and a mesh that does not fit on chip -- and through the
total-time clamp.  Equality is exact, so no tolerance enters."""
import numpy as np
import pytest

from enscdynamics_b200 import capi
from enscdynamics_b200 import mesh as M
from enscdynamics_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (31, 1, 1), (33, 1, 1), (43, 3, 1), (16, 16, 8), (683, 3, 1), (41, 22, 21), (61, 37, 19)]


def problem(dims, plastic=True, total_time=1.0):
    p = W.block(*dims, *(0.01 * d for d in dims), seed=sum(dims), plastic=plastic)
    p.controls.total_time = total_time
    return p


def run_single(p, precision, cycles, **kw):
    with capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls, precision=precision,
                      **kw) as s:
        s.set_bcs(p.bc_code, p.bc_value)
        reps = [s.step(n) for n in cycles]
        return s.download(), reps[-1], s.energy(), s.kernels_per_cycle


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("plastic", [False, True])
def test_fp64_equals_the_oracle(dims, plastic):
    import pyoracle
    p = problem(dims, plastic)
    m, c = p.material, p.controls
    o = pyoracle.Oracle(p.mesh.x0, p.mesh.conn, p.v0, p.bc_code, p.bc_value, E=m.E, nu=m.nu, rho=m.rho, c_dr=c.c_dr,
                        c_cr=c.c_cr, factor=c.factor, cvisl=c.cvisl, cvisq=c.cvisq, total_time=c.total_time,
                        yield0=m.yield_stress, hardening=m.hardening)
    o.run(12)
    got, rep, e, launches = run_single(p, capi.FP64, (5, 7))
    assert launches == 0 and rep["total_cycles"] == 12 and rep["status"] == 0
    for k in ("x", "u", "v", "sigma", "qia"):
        assert np.array_equal(got[k].reshape(-1), getattr(o, k)), k
    assert (rep["time"], rep["dt_i"], rep["dt_i_1"]) == (o.time, *o.dt)
    assert abs(e["kinetic"] - o.energy[0]) <= 1e-12 * o.energy[0]


@pytest.mark.parametrize("dims", SIZES)
def test_mixed_equals_the_batch(dims):
    p = problem(dims)
    got, rep, e, launches = run_single(p, capi.MIXED, (5, 7))
    assert launches == 0 and rep["total_cycles"] == 12
    with capi.Batch(max_instances=1, max_elements=p.mesh.n_elements, max_nodes=p.mesh.n_nodes,
                    budget_bytes=1 << 30, precision=capi.MIXED) as b:
        sl = b.add(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls)
        b.set_bcs(sl, p.bc_code, p.bc_value)
        b.arm(sl, 12)
        b.run(12)
        b.sync()
        ref, eb = b.download(sl), b.energy(sl)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    for k in e:
        assert abs(e[k] - eb[k]) <= 1e-12 * max(abs(eb[k]), e["kinetic0"]), k


@pytest.mark.parametrize("dims", [(33, 1, 1), (683, 3, 1)])
def test_total_time_clamp_and_stop(dims):
    import pyoracle
    dt = run_single(problem(dims, False), capi.FP64, (4,))[1]["dt_i"]
    p = problem(dims, False, total_time=9.4 * dt)
    m, c = p.material, p.controls
    o = pyoracle.Oracle(p.mesh.x0, p.mesh.conn, p.v0, p.bc_code, p.bc_value, E=m.E, nu=m.nu, rho=m.rho, c_dr=c.c_dr,
                        c_cr=c.c_cr, factor=c.factor, cvisl=c.cvisl, cvisq=c.cvisq, total_time=c.total_time)
    n = o.run(1000, c.total_time)
    with capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=m, controls=c) as s:
        s.set_bcs(p.bc_code, p.bc_value)
        rep = s.step(1000, c.total_time)
        got = s.download()
    assert rep["cycles"] == n and rep["done"] == 1 and rep["time"] == o.time
    for k in ("x", "u", "v", "sigma"):
        assert np.array_equal(got[k].reshape(-1), getattr(o, k)), k


def test_a_mesh_beyond_the_chip_uses_the_phase_kernels():
    for n, launches in ((60_000, 0), (400_000, 4)):
        k = M.box_mesh(n, 1, 1, 0.01 * n, 0.01, 0.01)
        with capi.Stepper(k.x0, k.conn, None, material=M.Material(70e9, 0.33, 2700.0),
                          controls=M.Controls()) as s:
            assert s.kernels_per_cycle == launches
            assert s.step(2)["cycles"] == 2
