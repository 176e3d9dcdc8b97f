"""The FP32 step with the split vertical velocity next to the side stream's stages."""
import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_implicit_diffusion_costs_the_split_velocity_its_own_time_only():
    """The implicit diffusion adds two short stages to a step with the split velocity and the limiter: its
    factors, which run beside the edge stages, and the solve.  Measured 1.00 times the step with explicit
    diffusion; 1.69 where the long column kernel of the split velocity shared the SMs with the side stream.
    The line is half way, on the fastest of five runs of each."""
    mesh = M.sphere_mesh(6, M.stretched_zbar(47, 5.0, 250.0), seed=3)
    f = O.ensure_f64(M.split_vertical_velocity(mesh, M.make_forcing(mesh, "sphere", seed=11, dt=600.0), 0.5))
    tr = [np.ascontiguousarray(t, dtype=np.float64) for t in M.make_tracers(mesh, "sphere", ntr=2, seed=4)]
    stream = torch.cuda.Stream()
    ms = []
    for ivd in (True, False):
        ctx = G.Context(mesh, G.PREC_FP32, max_tracers=2)
        ctx.set_stream(stream.cuda_stream)
        ctx.set_wsplit(True)
        ctx.state_setup([G.tra_cfg(i_vert_diff=ivd, id=k + 1) for k in range(2)])
        ctx.forcing_upload(f)
        for k in range(2):
            ctx.tracer_upload(k, tr[k], tr[k])
        ctx.run_steps(f.dt, 4)
        assert ctx.status() == 0
        best = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            ctx.run_steps(f.dt, 10)
            b.record(stream)
            assert ctx.status() == 0
            b.synchronize()
            best.append(a.elapsed_time(b) / 10)
        ms.append(min(best))
        ctx.close()
    assert ms[0] <= 1.34 * ms[1], ms
