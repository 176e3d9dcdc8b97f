"""Horizontal diffusion of the FP32 form on a mesh whose edge_tri names, for some edges, an element that
does not contain the edge's ends.  The mesh check accepts it (the index is an element, its levels lie
inside both columns), and the flux is then that element's own gradient, as in the oracle."""
import copy

import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O
from tests.conftest import wet_mask
from tests.test_oracle import _ki

KH = 2e5


def _misnamed(mesh):
    """A copy of mesh in which every fifth edge's first or second element is another element, not deeper
    and not starting higher than the edge's columns; the edges changed."""
    m = copy.copy(mesh)
    m.edge_tri = mesh.edge_tri.copy()
    rng = np.random.default_rng(12)
    changed = []
    for e in range(3, mesh.edge2D, 5):
        side = int(rng.integers(2)) if mesh.edge_tri[e, 1] >= 0 else 0
        other = mesh.edge_tri[e, 1 - side]
        top = max(mesh.ulevels_nod2D[n] for n in mesh.edges[e])
        bot = min(mesh.nlevels_nod2D[n] for n in mesh.edges[e])
        ok = (mesh.ulevels >= top) & (mesh.nlevels <= bot)
        if other >= 0:  # the two wet ranges still meet
            ok &= (np.minimum(mesh.nlevels, mesh.nlevels[other]) - 1 >= np.maximum(mesh.ulevels, mesh.ulevels[other]))
        ok &= ~(np.isin(mesh.elem2D_nodes, mesh.edges[e]).sum(axis=1) == 2)
        cand = np.flatnonzero(ok)
        if cand.size:
            m.edge_tri[e, side] = rng.choice(cand)
            changed.append(e)
    return m, np.array(changed)


def test_mesh_is_accepted_and_node_sums_leave_the_mesh(basin_irregular):
    """The mesh passes the host check, and the sum of an element's nodes less the edge's ends is then no
    node of that element, mostly not even a node: an index no kernel may form."""
    m, changed = _misnamed(basin_irregular)
    G.mesh_check(m)
    assert changed.size > 50
    el = m.edge_tri[changed]
    s = m.elem2D_nodes.sum(axis=1)[el] - m.edges[changed].sum(axis=1)[:, None]
    bad = (el >= 0) & ((s < 0) | (s >= m.nod2D))
    assert bad.any()


def _run(ctx_step, ctx, f, cfgs, T, Ki, S):
    ctx.state_setup(cfgs)
    ctx.forcing_upload(f)
    if Ki is not None:
        ctx.set_hdiff(Ki)
    if S is not None:
        ctx.set_redi(S)
    for k, t in enumerate(T):
        ctx.tracer_upload(k, t, t)
    ctx_step()
    return [ctx.tracer_download(k)[0] for k in range(len(T))]


def _check(m, f, ocfgs, T, Ki, S, got, off):
    """got within the FP32 form's 1e-5 of the oracle; its diffusive part (against the step without) within 5 %
    of the oracle's plus the error of the two steps."""
    om, wet = O.OracleMesh(m), wet_mask(m)
    for k, c in enumerate(ocfgs):
        a, b = T[k].copy(), T[k].copy()
        om.tracer_step_ex(f, c, a, np.zeros_like(a), T[k].copy(), Ki=Ki, slope=S)
        om.tracer_step_ex(f, c, b, np.zeros_like(b), T[k].copy())
        scale = np.abs(a[wet]).max()
        ea, eb = np.abs(got[k] - a)[wet].max(), np.abs(off[k] - b)[wet].max()
        assert ea <= 1e-5 * scale and eb <= 1e-5 * scale, (k, ea / scale, eb / scale)
        d64, d32 = (a - b)[wet], (got[k] - off[k])[wet]
        assert np.abs(d64).max() > 1e-4 * scale, k
        assert np.abs(d32 - d64).max() <= 0.05 * np.abs(d64).max() + ea + eb, k


def _setup(basin, ntr):
    m, _ = _misnamed(basin)
    f = O.ensure_f64(M.make_forcing(basin, "basin", seed=3, dt=600.0))
    T = [t.astype(np.float32).astype(np.float64) for t in M.make_tracers(basin, "basin", ntr=ntr, seed=4)]
    # without the limiter: its bounds are over the elements in the oracle, over the edges in the FP32 form
    cfgs = [G.tra_cfg("MUSCL", "QR4C", "NON", 0.0, 1.0, id=k + 1) for k in range(ntr)]
    ocfgs = [O.cfg_struct("MUSCL", "QR4C", "NON", 0.0, 1.0) for _ in range(ntr)]
    return m, f, T, cfgs, ocfgs


@pytest.mark.gpu
@pytest.mark.parametrize("redi", [False, True])
@pytest.mark.parametrize("ntr", [2, 3])
def test_fp32_step_takes_the_named_elements(basin_irregular, ntr, redi):
    m, f, T, cfgs, ocfgs = _setup(basin_irregular, ntr)
    Ki, S = _ki(m, KH), M.make_slopes(m, smax=5e-3, s_cr=4e-3) if redi else None
    got = []
    for hd in (True, False):
        ctx = G.Context(m, G.PREC_FP32, max_tracers=ntr)
        got.append(_run(lambda: ctx.run_steps(f.dt, 1), ctx, f, cfgs, T, Ki if hd else None, S if hd else None))
        assert ctx.status() == 0
    _check(m, f, ocfgs, T, Ki, S, *got)


@pytest.mark.gpu
def test_batch_takes_the_named_elements(basin_irregular):
    """Two instances, one with such edges and one without, as their own contexts give them."""
    ntr = 2
    m, f, T, cfgs, ocfgs = _setup(basin_irregular, ntr)
    meshes = [m, basin_irregular]
    ctxs = [G.Context(q, G.PREC_FP32, max_tracers=ntr) for q in meshes]
    for c, q in zip(ctxs, meshes):
        c.state_setup(cfgs)
        c.forcing_upload(f)
        c.set_hdiff(_ki(q, KH))
        for k, t in enumerate(T):
            c.tracer_upload(k, t, t)
    batch = G.Batch(ctxs)
    batch.run_steps(f.dt, 1)
    for c, q in zip(ctxs, meshes):
        alone = G.Context(q, G.PREC_FP32, max_tracers=ntr)
        want = _run(lambda: alone.run_steps(f.dt, 1), alone, f, cfgs, T, _ki(q, KH), None)
        for k in range(ntr):
            v = c.tracer_download(k)[0]
            wet = wet_mask(q)
            scale = np.abs(want[k][wet]).max()
            assert np.abs(v - want[k])[wet].max() <= 1e-6 * scale, k
