"""A step call in a stream under capture is refused, whatever the launch form of
the mesh (resident in a cluster, resident on the grid, per-phase kernels one by
one or as a graph): the cycles would be recorded and not run.  The capture and
the handle stay usable."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 8, 8), (41, 22, 21), (90, 40, 40)])
@pytest.mark.parametrize("cycles", [1, 4, 64])
def test_step_calls_are_refused_under_capture(dims, cycles):
    import torch
    from enscdynamics_b200 import capi
    from enscdynamics_b200 import workloads as W
    p = W.block(*dims, *(0.01 * d for d in dims), seed=2, plastic=False)
    st = torch.cuda.Stream()
    with capi.Stepper(p.mesh.x0, p.mesh.conn, p.v0, material=p.material, controls=p.controls,
                      stream=st.cuda_stream) as s:
        s.set_bcs(p.bc_code, p.bc_value)
        s.step(3)
        torch.cuda.synchronize()
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st, capture_error_mode="thread_local"):
            for call in (lambda: s.step_until_async(cycles, math.inf, math.inf), lambda: s.step(cycles)):
                with pytest.raises(capi.EnscError) as e:
                    call()
                assert e.value.code == -3 and "StreamCaptureUnsupported" in str(e.value)
        torch.cuda.synchronize()
        assert s.step(2)["total_cycles"] == 5
