"""FP32 diffusion on a mesh whose gradient_sca does not add up to zero over an element: the element's
gradient is the sum of its weighted node values, as in the oracle, not a sum of weighted differences."""
import copy

import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O
from tests.conftest import wet_mask
from tests.test_oracle import _ki

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntr", [2, 3])
@pytest.mark.parametrize("redi", [False, True])
def test_weights_that_do_not_add_up(channel_seamount, ntr, redi):
    """Upwind advection, which takes no gradient; the FP32 form's 1e-5, and the diffusive part within 5 %
    plus the error of the two steps."""
    m = copy.copy(channel_seamount)
    m.gradient_sca = m.gradient_sca.copy()
    g = m.gradient_sca.reshape(m.elem2D, 6)
    g[::7, 1] += 0.02 * np.abs(g[::7, :3]).max(axis=1)
    g[3::11, 5] -= 0.01 * np.abs(g[3::11, 3:]).max(axis=1)
    f = O.ensure_f64(M.make_forcing(channel_seamount, "channel", seed=3, dt=600.0))
    T = [t.astype(np.float32).astype(np.float64) for t in M.make_tracers(m, "channel", ntr=ntr, seed=4)]
    Ki, S = _ki(m, 2e5), M.make_slopes(m, smax=5e-3, s_cr=4e-3) if redi else None
    out = []
    for on in (True, False):
        ctx = G.Context(m, G.PREC_FP32, max_tracers=ntr)
        ctx.state_setup([G.tra_cfg("UPW1", "UPW1", "FCT", id=k + 1) for k in range(ntr)])
        ctx.forcing_upload(f)
        if on:
            ctx.set_hdiff(Ki)
            if redi:
                ctx.set_redi(S)
        for k in range(ntr):
            ctx.tracer_upload(k, T[k], T[k])
        ctx.run_steps(f.dt, 1)
        assert ctx.status() == 0
        out.append([ctx.tracer_download(k)[0] for k in range(ntr)])
    om, wet, c = O.OracleMesh(m), wet_mask(m), O.cfg_struct("UPW1", "UPW1", "FCT")
    for k in range(ntr):
        a, b = T[k].copy(), T[k].copy()
        om.tracer_step_ex(f, c, a, np.zeros_like(a), T[k].copy(), Ki=Ki, slope=S)
        om.tracer_step_ex(f, c, b, np.zeros_like(b), T[k].copy())
        scale = np.abs(a[wet]).max()
        ea, eb = np.abs(out[0][k] - a)[wet].max(), np.abs(out[1][k] - b)[wet].max()
        assert ea <= 1e-5 * scale and eb <= 1e-5 * scale, (k, ea / scale, eb / scale)
        d64, d32 = (a - b)[wet], (out[0][k] - out[1][k])[wet]
        assert np.abs(d64).max() > 1e-4 * scale, k
        assert np.abs(d32 - d64).max() <= 0.05 * np.abs(d64).max() + ea + eb, k
