"""Force hand-off of meshes whose nodes repeat local slots, and caller's own
B0^T: FP64 states equal the CPU restatement bit for bit, alone and in a batch.

Fans of kites around an axis, the axis in slot 0 of every element of a layer:
4 kites in 2 and more layers put exactly 8 elements on an axis node (rows of
the force array per node), 5 kites 10 (node lists).  The permuted block runs
the per-phase kernels of one instance.  Mixed precision equals its batch bit
for bit, and the FP64 state within FP32 round-off."""
import numpy as np
import pytest

from enscdynamics_b200 import capi
from enscdynamics_b200 import mesh as M
from enscdynamics_b200 import workloads as W

pytestmark = pytest.mark.gpu

MAT = M.Material(210e9, 0.3, 7850.0, 150e6, 2e9)
CTL = M.Controls(c_dr=0.013, c_cr=0.05, factor=0.71, cvisl=0.06, cvisq=1.2, total_time=1.0)
FANS = [(4, 1), (4, 2), (4, 19), (5, 2), (5, 19)]


def fan(m, layers):
    """m kites around the z axis per layer: centre, spoke i, corner i, spoke i + 1."""
    a = 2 * np.pi * np.arange(m) / m
    b = a + np.pi / m
    ring = np.concatenate([[[0.0, 0.0]], 0.1 * np.c_[np.cos(a), np.sin(a)], 0.13 * np.c_[np.cos(b), np.sin(b)]])
    n2 = len(ring)
    x0 = np.concatenate([np.c_[ring, np.full(n2, 0.1 * l)] for l in range(layers + 1)])
    conn = np.array([[l * n2 + q for l in (k, k + 1) for q in (0, 1 + i, 1 + m + i, 1 + (i + 1) % m)]
                     for k in range(layers) for i in range(m)], dtype=np.uint32)
    return x0, conn


def permuted_block(dims):
    """A block whose odd elements start their numbering a quarter turn further."""
    m = W.block(*dims, *(0.01 * d for d in dims), seed=1, plastic=True).mesh
    conn = np.array(m.conn, dtype=np.uint32)
    conn[1::2] = conn[1::2][:, [1, 2, 3, 0, 5, 6, 7, 4]]
    return np.asarray(m.x0), conn


def start(x0):
    rng = np.random.default_rng(3)
    v0 = rng.normal(0.0, 20.0, x0.shape)
    code = np.zeros(x0.shape, dtype=np.int8)
    code[x0[:, 2] == 0.0, 2] = 1
    return v0, code, np.zeros(x0.shape)


def oracle(x0, conn, cycles, setup=None):
    import pyoracle
    v0, code, val = start(x0)
    o = pyoracle.Oracle(x0, conn, v0, code, val, E=MAT.E, nu=MAT.nu, rho=MAT.rho, c_dr=CTL.c_dr, c_cr=CTL.c_cr,
                        factor=CTL.factor, cvisl=CTL.cvisl, cvisq=CTL.cvisq, total_time=CTL.total_time,
                        yield0=MAT.yield_stress, hardening=MAT.hardening, setup=setup)
    if cycles:
        o.run(cycles)
    return o


def single(x0, conn, cycles, precision=capi.FP64, **setup):
    v0, code, val = start(x0)
    with capi.Stepper(x0, conn, v0, material=MAT, controls=CTL, precision=precision, **setup) as s:
        s.set_bcs(code, val)
        assert s.step(cycles)["status"] == 0
        return s.download()


def batched(x0, conn, cycles, precision=capi.FP64, **setup):
    v0, code, val = start(x0)
    with capi.Batch(max_instances=1, max_elements=len(conn), max_nodes=len(x0), budget_bytes=1 << 30,
                    precision=precision) as b:
        sl = b.add(x0, conn, v0, material=MAT, controls=CTL, **setup)
        b.set_bcs(sl, code, val)
        b.arm(sl, cycles)
        b.run(cycles)
        b.sync()
        return b.download(sl)


def assert_oracle(got, o):
    for k in ("x", "u", "v", "sigma", "qia", "eps_p"):
        assert np.array_equal(got[k].reshape(-1), getattr(o, k)), k


@pytest.mark.parametrize("m,layers", FANS)
def test_fans_equal_the_oracle(m, layers):
    x0, conn = fan(m, layers)
    assert M.check_slot_clashes(conn, len(x0)) > 0
    assert np.bincount(conn.reshape(-1)).max() == m * min(layers, 2)
    o = oracle(x0, conn, 25)
    assert_oracle(single(x0, conn, 25), o)
    assert_oracle(batched(x0, conn, 25), o)


@pytest.mark.parametrize("dims", [(4, 3, 2), (83, 41, 36)])
def test_permuted_block_equals_the_oracle(dims):
    x0, conn = permuted_block(dims)
    assert M.check_slot_clashes(conn, len(x0)) > 0
    o = oracle(x0, conn, 6)
    assert_oracle(single(x0, conn, 6), o)
    assert_oracle(batched(x0, conn, 6), o)


@pytest.mark.parametrize("mesh", [fan(4, 19), permuted_block((83, 41, 36))])
def test_mixed_rows_equal_the_batch(mesh):
    x0, conn = mesh
    got, ref, f64 = single(x0, conn, 6, capi.MIXED), batched(x0, conn, 6, capi.MIXED), single(x0, conn, 6)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    # six cycles of FP32 element arithmetic: 6 x 32 roundings of 2^-24, doubled
    for k in ("u", "v"):
        assert np.abs(got[k] - f64[k]).max() <= 2.3e-5 * np.abs(f64[k]).max(), k


@pytest.mark.parametrize("plastic_dims", [(3, 2, 1), (11, 9, 7)])
def test_callers_own_b0_equals_the_oracle(plastic_dims):
    """Constants whose bits no 9 numbers reproduce: B0^T moved by an ulp here
    and there, so the 24-number tiles run."""
    x0, conn = permuted_block(plastic_dims)
    o = oracle(x0, conn, 0)
    rng = np.random.default_rng(5)
    bt = np.where(rng.integers(0, 2, o.bt.size) == 1, np.nextafter(o.bt, np.inf), o.bt)
    setup = dict(bt=bt.reshape(-1, 24), vol0=o.vol0.copy(), inv_mass=o.inv_mass.copy())
    o = oracle(x0, conn, 12, setup)
    setup["inv_mass"] = setup["inv_mass"].reshape(-1, 3)
    assert_oracle(single(x0, conn, 12, **setup), o)
    assert_oracle(batched(x0, conn, 12, **setup), o)


@pytest.mark.parametrize("dims", [(5, 4, 3), (9, 8, 33), (83, 41, 36)])
def test_shuffled_elements_equal_the_oracle(dims):
    """Elements numbered at random: they are stored in an order that follows
    the nodes, and every element field comes back in the caller's numbering."""
    x0, conn = permuted_block(dims)
    conn = np.ascontiguousarray(conn[np.random.default_rng(9).permutation(len(conn))])
    o = oracle(x0, conn, 6)
    assert_oracle(single(x0, conn, 6), o)
    assert_oracle(batched(x0, conn, 6), o)
    got, ref = single(x0, conn, 6, capi.MIXED), batched(x0, conn, 6, capi.MIXED)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    v0, code, val = start(x0)
    with capi.Stepper(x0, conn, v0, material=MAT, controls=CTL) as s:
        s.set_bcs(code, val)
        clk = s.step(4)
        mid = s.download()
    with capi.Stepper(x0, conn, v0, material=MAT, controls=CTL) as s:
        s.set_bcs(code, val)
        s.upload_state(mid, clk["time"], clk["dt_i"], clk["dt_i_1"], clk["dt_stable_min"])
        s.step(2)
        assert_oracle(s.download(), o)
