"""Resident runs in one cluster: shared memory of another block is written only
after a barrier of the cluster that follows the launch, which is what says that
the other block runs.  Read from the source, since a lost store would depend on
the timing of a launch."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "enscdynamics_b200", "csrc")


def run_cycles_body():
    with open(os.path.join(CSRC, "ensc_run.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    at = text.index("void run_cycles(")
    start = end = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[start:end]


def test_a_cluster_barrier_comes_before_the_first_remote_store():
    body = run_cycles_body()
    loop = body.index("while (sh.go)")
    stores = [m.start() for m in re.finditer(r"\bst_cluster(32)?\(", body)]
    assert stores and min(stores) > loop  # launches with no cycle to run store nothing
    head = body[:loop]
    assert len(re.findall(r"if \(CLUSTER\) cluster_arrive\(\);", head)) == 1
    assert len(re.findall(r"if \(CLUSTER\) cluster_wait\(\);", head)) == 1
    assert head.index("cluster_arrive()") < head.index("cluster_wait()")
    # no block leaves between the two
    assert "return" not in head[head.index("cluster_arrive()"):]


@pytest.mark.gpu
@pytest.mark.parametrize("ne,clusters", [(33, 4), (250, 16)])
def test_blocks_without_a_tile_equal_the_oracle(ne, clusters):
    """Elements that share no node need more blocks for their nodes than for
    their tiles; a launch per cycle takes the launch's first barrier each time."""
    import pyoracle
    from enscdynamics_b200 import capi
    from enscdynamics_b200 import mesh as M
    one = M.box_mesh(1, 1, 1, 0.01, 0.01, 0.01)
    x0 = np.concatenate([one.x0 + [0.02 * i, 0.0, 0.0] for i in range(ne)])
    conn = np.concatenate([one.conn + 8 * i for i in range(ne)]).astype(np.uint32)
    assert 128 * clusters >= len(x0) > 64 * clusters and (ne + 31) // 32 <= 2 * clusters
    v0 = np.random.default_rng(ne).normal(0.0, 5.0, x0.shape)
    code, val = np.zeros(x0.shape, dtype=np.int8), np.zeros(x0.shape)
    m, c = M.Material(70e9, 0.33, 2700.0), M.Controls()
    o = pyoracle.Oracle(x0, conn, v0, code, val, E=m.E, nu=m.nu, rho=m.rho, c_dr=c.c_dr, c_cr=c.c_cr,
                        factor=c.factor, cvisl=c.cvisl, cvisq=c.cvisq, total_time=c.total_time)
    o.run(5)
    with capi.Stepper(x0, conn, v0, material=m, controls=c) as s:
        s.set_bcs(code, val)
        for _ in range(5):
            s.step(1)
        got = s.download()
    for k in ("x", "u", "v", "sigma", "qia"):
        assert np.array_equal(got[k].reshape(-1), getattr(o, k)), k
