"""The FP64 form's tiled kernels at the sizes where they can go wrong: entity counts that leave a
partial tile, tiles of 4 and of 8, columns around a warp's 32 levels, and the general expressions
behind the short ones (adv_ph /= 0, adv_pv /= 1); bit for bit against the oracle."""
import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O
from tests.conftest import perturbed_old

pytestmark = pytest.mark.gpu

# nx, ny, layers, partial cells, tracers: (horizontal, vertical, limiter, adv_ph, adv_pv), ab
CASES = [
    (5, 7, 4, False, [("MUSCL", "QR4C", "FCT", 0.0, 1.0)], 2),
    (5, 7, 5, False, [("MFCT", "QR4C", "FCT", 0.4, 0.3), ("UPW1", "CDIFF", "FCT", 0.0, 1.0)], 3),
    (7, 11, 31, True, [("MUSCL", "QR4C", "FCT", 0.0, 1.0)] * 2, 2),
    (9, 13, 32, True, [("MFCT", "CDIFF", "NON", 0.0, 1.0), ("MUSCL", "UPW1", "FCT", 1.0, 0.0)], 2),
    (9, 13, 33, True, [("MUSCL", "QR4C", "FCT", 0.25, 0.5)] * 3, 3),
    (11, 17, 65, True, [("MUSCL", "QR4C", "FCT", 0.0, 1.0), ("MFCT", "PPM", "FCT", 0.0, 1.0)], 2),
    (101, 97, 21, True, [("MUSCL", "QR4C", "FCT", 0.0, 1.0)] * 2, 2),
]


@pytest.mark.parametrize("nx,ny,layers,partial,schemes,ab", CASES)
def test_step_bitwise(nx, ny, layers, partial, schemes, ab):
    mesh = M.channel_mesh(nx, ny, 5000.0, M.stretched_zbar(layers, 10.0, 200.0), seamounts=2 if partial else 0, seed=5,
                          partial_cells=partial)
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    n = len(schemes)
    tr = M.make_tracers(mesh, "channel", ntr=n, seed=4)
    om = O.OracleMesh(mesh)
    ctx = G.Context(mesh, G.PREC_FP64, max_tracers=n)
    rng = np.random.default_rng(2)
    To = [np.array(t, copy=True) for t in tr]
    Oo = [np.ascontiguousarray(np.stack([perturbed_old(t, rng) for _ in range(ab - 1)], axis=-1)) for t in To]
    Tg, Og = [t.copy() for t in To], [o.copy() for o in Oo]
    gcfg = [G.tra_cfg(h, v, l, ph, pv, ab, True, k + 1) for k, (h, v, l, ph, pv) in enumerate(schemes)]
    ocfg = [O.cfg_struct(h, v, l, ph, pv, ab) for h, v, l, ph, pv in schemes]
    for step in range(2):
        for k in range(n):
            om.tracer_step(f, ocfg[k], To[k], np.zeros_like(To[k]), Oo[k])
        ctx.tracer_step(f, gcfg, Tg, Og)
        for k in range(n):
            assert np.array_equal(Tg[k], To[k]), f"step {step} tracer {k}"
            assert np.array_equal(Og[k], Oo[k]), f"step {step} tracer {k}: previous levels"
    assert ctx.status() == 0


@pytest.mark.parametrize("nx,ny,layers,ntr", [(5, 7, 4, 1), (8, 4, 32, 2), (7, 9, 33, 3), (11, 13, 65, 5),
                                              (6, 7, 217, 2), (6, 7, 218, 2)])
def test_vertical_diffusion_tiles_bitwise(nx, ny, layers, ntr):
    """Tiles of 32 columns (a last one of fewer), up to four tracers to a pass, and the deepest
    column a tile holds next to the first that takes a thread per column."""
    mesh = M.channel_mesh(nx, ny, 5000.0, M.stretched_zbar(layers, 5.0, 20.0), seamounts=1, seed=5, partial_cells=True)
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    rng = np.random.default_rng(6)
    tr = [np.ascontiguousarray(t) for t in M.make_tracers(mesh, "channel", ntr=ntr, seed=4)]
    om = O.OracleMesh(mesh)
    ctx = G.Context(mesh, G.PREC_FP64, max_tracers=ntr)
    To, Tg = [t.copy() for t in tr], [t.copy() for t in tr]
    Oo = [perturbed_old(t, rng) for t in To]
    Og = [o.copy() for o in Oo]
    for k in range(ntr):
        om.tracer_step(f, O.cfg_struct(), To[k], np.zeros_like(To[k]), Oo[k])
    ctx.tracer_step(f, [G.tra_cfg(id=k + 1) for k in range(ntr)], Tg, Og)
    for k in range(ntr):
        assert np.array_equal(Tg[k], To[k]), f"tracer {k}"
    # the drop-ins, with a surface flux: one tracer through a context and without one
    f.bc_surface = np.linspace(-1e-3, 1e-3, mesh.nod2D)
    want, got = tr[0].copy(), tr[0].copy()
    om.diff_ver_part_impl_ale(f, want)
    ctx.vdiff_impl(f, G.tra_cfg(), got)
    assert np.array_equal(got, want)


def test_element_lists_beside_the_edges_bitwise():
    """A mesh whose nod_in_elem2D lists leave out an element of some nodes: the bounds of those nodes
    come from the listed elements, not from the neighbours over the edges, as in the oracle."""
    mesh = M.channel_mesh(9, 13, 5000.0, M.stretched_zbar(33, 10.0, 200.0), seamounts=2, seed=5, partial_cells=True)
    ptr, keep = mesh.nod_in_elem2D_ptr, np.ones(mesh.nod_in_elem2D.size, dtype=bool)
    short = [n for n in range(5, mesh.nod2D, 7) if ptr[n + 1] - ptr[n] == 6]
    keep[[ptr[n + 1] - 1 for n in short]] = False
    drop = np.zeros(mesh.nod2D, dtype=np.int64)
    drop[short] = 1
    mesh.nod_in_elem2D_ptr = (ptr - np.concatenate([[0], np.cumsum(drop)])).astype(np.int32)
    mesh.nod_in_elem2D = np.ascontiguousarray(mesh.nod_in_elem2D[keep])
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    T = np.ascontiguousarray(M.make_tracers(mesh, "channel", ntr=1, seed=4)[0])
    rng = np.random.default_rng(8)
    T *= 1.0 + 0.05 * rng.standard_normal(T.shape)
    TAB = np.ascontiguousarray(T * (1.0 + 1e-3 * rng.standard_normal(T.shape)))
    om, cfg = O.OracleMesh(mesh), O.cfg_struct()
    om.init_tracers_AB(cfg, T.copy(), np.zeros_like(T), T.copy())
    om.do_oce_adv_tra(f, cfg, T, TAB)
    ctx = G.Context(mesh, G.PREC_FP64)
    dh, dv = ctx.adv_tra(f, G.tra_cfg(), T, TAB)
    lev = np.arange(1, mesh.nl)[None, :]
    wet = (lev >= mesh.ulevels_nod2D[:, None]) & (lev <= mesh.nlevels_nod2D[:, None] - 1)
    assert np.array_equal(dh[wet], om.work["del_ttf_advhoriz"][wet])
    assert np.array_equal(dv[wet], om.work["del_ttf_advvert"][wet])


@pytest.mark.parametrize("hor,ver,lim,ph,pv", [("MUSCL", "QR4C", "FCT", 0.0, 1.0), ("MFCT", "CDIFF", "FCT", 0.0, 1.0),
                                               ("UPW1", "UPW1", "FCT", 0.0, 1.0), ("MUSCL", "QR4C", "NON", 0.3, 0.4),
                                               ("MFCT", "QR4C", "FCT", 0.0, 0.7)])
@pytest.mark.parametrize("bad", [(np.nan,), (np.inf, -np.inf), (np.nan, np.inf), (1e300, -1e300),
                                 (1e-310, -1e-310, 0.0)], ids=["nan", "inf", "mixed", "huge", "tiny"])
def test_values_outside_the_normal_range_bitwise(hor, ver, lim, ph, pv, bad):
    """Not-a-number, infinite, huge and denormal values reach the same results through the short
    expressions (a product that drops out, integer maxima, quotients by reciprocals) as in the oracle."""
    mesh = M.sphere_mesh(4, M.stretched_zbar(33, 5.0, 250.0), seed=9)
    f = O.ensure_f64(M.make_forcing(mesh, "sphere", seed=3, dt=600.0))
    rng = np.random.default_rng(5)
    T = np.array(M.make_tracers(mesh, "sphere", ntr=1, seed=4)[0], copy=True)
    T *= 1.0 + 0.02 * rng.standard_normal(T.shape)
    TAB = np.ascontiguousarray(T * (1.0 + 1e-3 * rng.standard_normal(T.shape)))
    lev = np.arange(1, mesh.nl)[None, :]
    wet = (lev >= mesh.ulevels_nod2D[:, None]) & (lev <= mesh.nlevels_nod2D[:, None] - 1)
    idx = np.argwhere(wet)
    for q, (n, k) in enumerate(idx[rng.choice(len(idx), 12, replace=False)]):
        (T if q % 2 else TAB)[n, k] = bad[q % len(bad)]
    om, cfg = O.OracleMesh(mesh), O.cfg_struct(hor, ver, lim, ph=ph, pv=pv)
    om.init_tracers_AB(cfg, T.copy(), np.zeros_like(T), T.copy())
    om.do_oce_adv_tra(f, cfg, T, TAB)
    ctx = G.Context(mesh, G.PREC_FP64)
    dh, dv = ctx.adv_tra(f, G.tra_cfg(hor, ver, lim, ph, pv), T, TAB)
    assert np.array_equal(dh[wet], om.work["del_ttf_advhoriz"][wet], equal_nan=True)
    assert np.array_equal(dv[wet], om.work["del_ttf_advvert"][wet], equal_nan=True)
