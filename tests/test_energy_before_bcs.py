"""Cycles that run before a handle's first boundary conditions keep their work
in the energy sums: the report is the same, to the bit, as when the energies are
read (and so folded) before the conditions are set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", [(16, 8, 8), (41, 22, 21), (90, 60, 40)])
def test_work_done_before_the_first_conditions_is_kept(dims, precision):
    from enscdynamics_b200 import capi
    from enscdynamics_b200 import workloads as W
    p = W.block(*dims, *(0.01 * d for d in dims), seed=4, plastic=True)
    reports = []
    for read in (False, True):
        with capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls,
                          precision=(capi.FP64, capi.MIXED)[precision]) as s:
            s.step(24)
            mid = s.energy() if read else None
            s.set_bcs(p.bc_code, p.bc_value)
            start = s.energy()
            s.step(3)
            reports.append((start, s.energy()))
    assert reports[0] == reports[1]
    assert mid["internal"] > 0.0 and reports[0][0]["internal"] == mid["internal"]
    assert reports[0][0]["kinetic"] == reports[0][0]["kinetic0"] > 0.0
    assert all(np.isfinite(v) for e in reports[0] for v in e.values())
