"""The Redi terms of the FP32 form on a mesh whose nod_in_elem2D lists leave out elements of some nodes:
the node gradient of the vertical projection is over the listed elements, as in the oracle, not over the
edges around the node."""
import copy

import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O
from tests.conftest import wet_mask
from tests.test_oracle import _ki

pytestmark = pytest.mark.gpu


def _short_lists(mesh):
    m = copy.copy(mesh)
    ptr, num = mesh.nod_in_elem2D_ptr, np.diff(mesh.nod_in_elem2D_ptr)
    # an element of the full depth of the node's levels stays in the list
    short = [n for n in range(2, mesh.nod2D, 5) if num[n] >= 5]
    keep = np.ones(mesh.nod_in_elem2D.size, dtype=bool)
    keep[[ptr[n + 1] - 1 for n in short]] = False
    drop = np.zeros(mesh.nod2D, dtype=np.int64)
    drop[short] = 1
    m.nod_in_elem2D_ptr = (ptr - np.concatenate([[0], np.cumsum(drop)])).astype(ptr.dtype)
    m.nod_in_elem2D = np.ascontiguousarray(mesh.nod_in_elem2D[keep])
    return m


@pytest.mark.parametrize("ntr", [2, 3])
def test_fp32_redi_over_the_listed_elements(channel_seamount, ntr):
    """Upwind advection without the limiter, whose other uses of the lists differ by form; the FP32 form's
    1e-5, and the part of the step that the lists change within 5 % plus the error of the two steps."""
    mesh = channel_seamount
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    T = [t.astype(np.float32).astype(np.float64) for t in M.make_tracers(mesh, "channel", ntr=ntr, seed=4)]
    Ki, S = _ki(mesh, 2e6), M.make_slopes(mesh, smax=5e-3, s_cr=4e-3)
    c, wet, got, want = O.cfg_struct("UPW1", "UPW1", "NON"), wet_mask(mesh), [], []
    for m in (_short_lists(mesh), mesh):
        ctx = G.Context(m, G.PREC_FP32, max_tracers=ntr)
        ctx.state_setup([G.tra_cfg("UPW1", "UPW1", "NON", id=k + 1) for k in range(ntr)])
        ctx.forcing_upload(f)
        ctx.set_hdiff(Ki)
        ctx.set_redi(S)
        for k in range(ntr):
            ctx.tracer_upload(k, T[k], T[k])
        ctx.run_steps(f.dt, 1)
        assert ctx.status() == 0
        got.append([ctx.tracer_download(k)[0] for k in range(ntr)])
        om, ref = O.OracleMesh(m), []
        for k in range(ntr):
            a = T[k].copy()
            om.tracer_step_ex(f, c, a, np.zeros_like(a), T[k].copy(), Ki=Ki, slope=S)
            ref.append(a)
        want.append(ref)
    for k in range(ntr):
        scale = np.abs(want[0][k][wet]).max()
        e = [np.abs(got[q][k] - want[q][k])[wet].max() for q in (0, 1)]
        assert max(e) <= 1e-5 * scale, (k, e, scale)
        d64, d32 = (want[0][k] - want[1][k])[wet], (got[0][k] - got[1][k])[wet]
        assert np.abs(d64).max() > 5e-6 * scale, k  # thirty times the form's own error
        assert np.abs(d32 - d64).max() <= 0.05 * np.abs(d64).max() + e[0] + e[1], k
