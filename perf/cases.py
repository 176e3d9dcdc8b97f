"""Performance cases of the tracer-transport step: the calls that programs of this library make.

A case is one mesh, one set of tracers with their schemes, and one way of calling the library:

``loop``      the time loop of a model whose other components live on the GPU: every pass brings new
              velocities, diffusivities and surface fluxes (device arrays), runs ``steps`` tracer steps
              on the resident state and reads every tracer into the model's own device arrays
``call``      ``fesom_gpu_tracer_step`` on the caller's own FP64 arrays, on the device (an OpenACC build
              passes device addresses) or in page-locked host memory (a CPU build)
``routines``  the routine-level drop-ins in the order of the reference's tracer loop: init_tracers_AB,
              do_oce_adv_tra, diff_ver_part_impl_ale, FP64 device arrays, one tracer
``noalloc``   the allocation-free implicit vertical diffusion on the caller's device arrays
``batch``     independent meshes of uneven size stepped together

Meshes come from this package's generators (channel and sphere, flat, seamount or partial-cell
bottoms), as do the velocities; tracer values are drawn on the device from the seed.  ``exact`` states
the same step in FP64 torch, written from the formulas.
"""
from __future__ import annotations

import collections
import ctypes as C
import dataclasses
import math

import numpy as np
import torch

from fesom2_gb300 import batch as BA
from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M

DT = 600.0          # seconds, the time step of every configuration of this repository
R_EARTH = 6367500.0
K_HOR = 3000.0      # m^2/s at 100 km resolution, the reference's global setting


def _case(name, call, prec, mesh, size, layers, tracers, hor="MUSCL", ver="QR4C", lim="FCT", ab=2, redi=False,
          steps=1, where="device", bottom="partial"):
    return dict(name=name, call=call, prec=prec, mesh=mesh, size=size, layers=layers, tracers=tracers, hor=hor,
                ver=ver, lim=lim, ab=ab, redi=redi, steps=steps, where=where, bottom=bottom)


def listed():
    return [
        # A regional toy channel (the size of the reference's Soufflet test, 2.9k nodes): the calls are
        # short, launches and latency count.  First the FP64 drop-in routines, then the FP32 time loop.
        _case("routines_toy_fp64", "routines", "fp64", "channel", 27, 40, 1, bottom="flat"),
        _case("loop_toy_fp32", "loop", "fp32", "channel", 27, 40, 2, bottom="flat"),
        # The allocation-free vertical diffusion of a caller that owns all device memory, near the
        # largest mesh its fixed scratch takes (odd number of layers, seamounts: ragged columns).
        _case("noalloc_vdiff_fp64", "noalloc", "fp64", "channel", 70, 47, 1, bottom="seamounts"),
        # The 100 x 400 channel of the first configuration, T and S: as an FP64 time loop, and called
        # with FP64 arrays in host memory as a Fortran CPU build does (FP32 on the device).
        _case("loop_channel_fp64", "loop", "fp64", "channel", 100, 40, 2, bottom="flat"),
        _case("call_channel_host", "call", "fp32", "channel", 100, 40, 2, where="host", bottom="flat"),
        # The same call with device addresses, in FP64, on a partial-cell sphere with an odd number of
        # layers: three tracers, third-order Adams-Bashforth, MFCT, centred vertical differences.
        _case("call_ragged_fp64", "call", "fp64", "sphere", 6, 61, 3, hor="MFCT", ver="CDIFF", ab=3),
        # The refined seamount channel of the second configuration (640k nodes, 60 layers), T and S.
        _case("loop_seamounts_fp32", "loop", "fp32", "channel", 400, 60, 2, bottom="seamounts"),
        # The land-masked sphere of the third configuration, T and S: the FP64 form and the FP32 form.
        _case("loop_sphere_fp64", "loop", "fp64", "sphere", 7, 48, 2),
        _case("loop_sphere_fp32", "loop", "fp32", "sphere", 7, 48, 2, steps=2),
        # A global set-up with the reference's default physics: MFCT, horizontal diffusion with Redi
        # slopes renewed every step; T, S and five passive tracers.
        _case("loop_redi_fp32", "loop", "fp32", "sphere", 7, 47, 7, hor="MFCT", redi=True),
        # Ocean biogeochemistry: T, S and 22 passive tracers on 450k nodes, 70 layers.
        _case("loop_biogeo_fp32", "loop", "fp32", "sphere", 8, 70, 24, steps=2),
        # An ensemble of uneven basins stepped in one launch per stage (the fifth configuration's draw
        # at a sixteenth of its node counts).
        _case("batch_uneven_fp32", "batch", "fp32", "mixed", 16, 0, 0, steps=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["loop", "loop", "loop", "loop", "call", "routines", "noalloc", "batch"])
    if call == "batch":
        return _pure(_case("", "batch", "fp32", "mixed", rng.randint(3, 16), 0, 0, steps=rng.randint(1, 3)))
    c = _case("", call, "fp64", "channel", 0, rng.randint(20, 80), 1)
    if call == "noalloc":
        # 3 (layers + 1) nodes stays below the fixed scratch: 4 size^2 nodes
        top = math.sqrt(4194304 / (3 * (c["layers"] + 1) * 4)) * 0.98
        c.update(size=int(_log(rng, 20, top)), bottom=rng.choice(["flat", "seamounts"]))
        return _pure(c)
    if call == "routines":
        c.update(size=int(_log(rng, 20, 150)), bottom="flat", hor=rng.choice(["MUSCL", "MFCT", "UPW1"]),
                 ver=rng.choice(["QR4C", "QR4C", "CDIFF", "UPW1"]), ab=rng.choice([2, 2, 3]))
        return _pure(c)
    c["prec"] = rng.choice(["fp32", "fp32", "fp64"])
    c.update(hor=rng.choice(["MUSCL", "MUSCL", "MFCT", "UPW1"]), ver=rng.choice(["QR4C", "QR4C", "CDIFF", "UPW1"]),
             lim=rng.choice(["FCT", "FCT", "FCT", "NON"]), ab=rng.choice([2, 2, 3]))
    budget = 5.0e8 if c["prec"] == "fp32" else 2.5e7   # tracer values of one step: the largest listed case's
    if call == "call":
        budget = 2.0e7
        c["where"] = rng.choice(["device", "device", "host"])
    if rng.random() < 0.5:
        c.update(mesh="channel", size=int(_log(rng, 25, 350)), bottom=rng.choice(["flat", "seamounts"]))
        nodes = 4 * c["size"] ** 2
    else:
        c.update(mesh="sphere", size=rng.randint(4, 8 if c["prec"] == "fp32" and call == "loop" else 7))
        nodes = 7 * 4 ** c["size"]
    while nodes * c["layers"] > budget / 2:
        c["layers"] = max(20, c["layers"] // 2)
        if c["layers"] == 20:
            break
    top = max(1, min(24, int(budget / (nodes * c["layers"]))))
    c["tracers"] = max(1, min(top, int(_log(rng, 1, top + 1))))
    if call == "loop":
        c["redi"] = c["mesh"] == "sphere" and c["size"] <= 7 and rng.random() < 0.35
        c["steps"] = rng.choice([1, 1, 2])
    return _pure(c)


def _pure(c):
    return {k: v for k, v in c.items() if k != "name"}


# ---------------------------------------------------------------------------
# meshes (kept between preparations: a program makes its mesh once)
# ---------------------------------------------------------------------------
_meshes = collections.OrderedDict()


def _mesh(key, make):
    if key in _meshes:
        _meshes.move_to_end(key)
    else:
        while len(_meshes) >= 2:
            _meshes.popitem(last=False)
        _meshes[key] = make()
    return _meshes[key]


def _make_mesh(kind, size, layers, bottom):
    if kind == "sphere":
        m = M.sphere_mesh(size, M.stretched_zbar(layers, 5.0, 250.0), seed=3)
    elif bottom == "flat":
        m = M.channel_mesh(size, 4 * size, 5000.0, -100.0 * np.arange(layers + 1))
    else:
        m = M.channel_mesh(size, 4 * size, 5000.0, M.stretched_zbar(layers, 10.0, 200.0),
                           seamounts=max(1, size // 33), seed=1, partial_cells=True)
    return m, M.make_forcing(m, kind, seed=11, dt=DT)


def _meshes_of(case):
    """[(mesh, forcing, kind, tracer count)] of a case: one mesh, or the instances of a batch."""
    if case["call"] == "batch":
        def make():
            out = []
            for s in BA.instance_specs()[:case["size"]]:
                m, kind, f, _ = BA.make_instance(dataclasses.replace(s, tracers=1), 1.0 / 16.0)
                out.append((m, f, kind, s.tracers))
            return out
        return _mesh(("batch", case["size"]), make)
    key = tuple(case[k] for k in ("mesh", "size", "layers", "bottom"))
    m, f = _mesh(key, lambda: _make_mesh(*key))
    return [(m, f, case["mesh"], case["tracers"])]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _fields(case, m, f, kind, ntr, seed, dev, dtype):
    """Velocities, diffusivity, surface fluxes and tracers of one mesh on `dev`: the mesh's flow and
    mixing with seeded strengths, T and S with their vertical and meridional structure and noise,
    lognormal passive tracers."""
    g = torch.Generator(device=dev).manual_seed(int(seed))
    r = np.random.default_rng(seed)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    amp, mix = float(r.uniform(0.5, 1.0) * r.choice([-1.0, 1.0])), float(r.uniform(0.5, 2.0))
    N2, L1 = m.nod2D, m.nl - 1
    uv, w = (t(f.uv) * amp).to(dtype), (t(f.w) * amp).to(dtype)
    Kv = (t(f.Kv) * mix).to(dtype)
    wet = torch.arange(L1, device=dev)[None, :] < t(m.nlevels_nod2D - 1)[:, None]
    d, lat = -t(m.Z_3d_n), t(m.coord_nod2D[:, 1])[:, None]
    if kind == "channel":
        y = lat * R_EARTH
        T = 20.0 - 0.002 * d + 2.0 * torch.tanh((y - 0.5 * (y.min() + y.max())) / 100e3)
        S, noise = torch.full_like(d, 35.0), 0.01
    else:
        T = 2.0 + 26.0 * torch.cos(lat) ** 2 * torch.exp(-d / 1000.0)
        S, noise = 34.0 + 1.5 * torch.cos(2 * lat).expand_as(d), 0.1
    ab = case["ab"]
    val = torch.zeros((ntr, N2, L1), device=dev, dtype=dtype)
    old = torch.zeros((ntr, N2, L1, ab - 1), device=dev, dtype=dtype)
    for k in range(ntr):
        z = torch.randn((N2, L1), generator=g, device=dev, dtype=torch.float32)
        v = (T + noise * z) if k == 0 else (S + noise * z) if k == 1 else torch.exp(z)
        val[k] = torch.where(wet, v, 0.0).to(dtype)
        for j in range(ab - 1):  # the earlier levels differ by a step's worth of change
            z = torch.randn((N2, L1), generator=g, device=dev, dtype=torch.float32)
            old[k, :, :, j] = (val[k] * (1.0 + 1e-3 * z)).to(dtype)
    bc = 1e-4 * torch.randn((ntr, N2), generator=g, device=dev, dtype=torch.float32)
    if case["hor"] != "UPW1" and case["lim"] == "FCT":
        bc[2:] = bc[2:].abs()  # passive tracers gain at the surface
    x = dict(uv=uv, w=w, Kv=Kv, bc=bc.to(dtype).contiguous(), values=val, old=old)
    if case["redi"]:
        res = torch.sqrt(t(m.areasvol[:, :1]))
        x["Ki"] = (K_HOR * (res / 100e3) ** 2 * wet).double().contiguous()
        s = torch.randn((2, 24), generator=g, device=dev, dtype=torch.float64)
        lon = t(m.coord_nod2D[:, 0])[:, None]
        prof = 1.5e-3 * torch.exp(-d / 1500.0)
        sx = prof * torch.sin(2 * lat + 3 * lon + s[0, 0])
        sy = prof * torch.cos(3 * lat - 2 * lon + s[1, 0])
        x["slope"] = torch.stack([sx, sy, torch.sqrt(sx * sx + sy * sy)], 2).mul(wet[:, :, None]).contiguous()
    return x


def _host(a):
    h = G.host_array(tuple(a.shape), np.float64)
    h[...] = a.cpu().numpy()
    return h


class Unit:
    """One mesh with its context, inputs and the arrays its results go to."""


def _chk(u, rc):
    if rc:
        raise RuntimeError(u.ctx.L.fesom_gpu_last_error(u.ctx.h).decode())


def _p(a):
    return None if a is None else C.c_void_p(a.ctypes.data if isinstance(a, np.ndarray) else a.data_ptr())


def _unit(case, m, f, kind, ntr, seed):
    u = Unit()
    fp32 = case["prec"] == "fp32"
    own = torch.float32 if fp32 and case["call"] in ("loop", "batch") else torch.float64
    u.x = _fields(case, m, f, kind, ntr, seed, "cuda", own)
    u.ntr = ntr
    u.cfgs = (G.TraCfg * ntr)(*[G.tra_cfg(case["hor"], case["ver"], case["lim"], 0.0, 1.0, case["ab"], True,
                                          k + 1 if k < 2 else 99 + k) for k in range(ntr)])
    if case["call"] == "noalloc":
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        u.N2, u.nl = m.nod2D, m.nl
        u.arrays = [t(m.nlevels_nod2D.astype(np.int32)), t(m.ulevels_nod2D.astype(np.int32)), t(m.zbar_n_bot),
                    t(m.hnode_new), t(m.area), t(m.areasvol)]
        return u
    u.ctx = G.Context(m, G.PREC_FP32 if fp32 else G.PREC_FP64, max_tracers=ntr)
    x = u.x
    if case["call"] == "routines":
        u.out = {k: torch.empty_like(x["values"][0]) for k in ("valuesAB", "dttf_h", "dttf_v")}
        u.star = x["values"][0].clone()
        return u
    if case["call"] == "call":
        if case["where"] == "host":
            u.x = x = {k: _host(v) for k, v in x.items()}
        at = (lambda a: a.ctypes.data) if case["where"] == "host" else (lambda a: a.data_ptr())
        u.vp = (C.c_void_p * ntr)(*[at(x["values"][k]) for k in range(ntr)])
        u.op = (C.c_void_p * ntr)(*[at(x["old"][k]) for k in range(ntr)])
        return u
    u.ctx.state_setup(list(u.cfgs))
    if case["redi"]:
        _chk(u, u.ctx.L.fesom_gpu_set_hdiff(u.ctx.h, _p(x["Ki"])))
    up = u.ctx.L.fesom_gpu_tracer_upload_f32 if fp32 else u.ctx.L.fesom_gpu_tracer_upload
    for k in range(ntr):
        _chk(u, up(u.ctx.h, k, _p(x["values"][k]), _p(x["old"][k])))
    u.out = torch.empty_like(x["values"])
    return u


def _forcing(u, fp32):
    x, L = u.x, u.ctx.L
    up = L.fesom_gpu_forcing_upload_f32 if fp32 else L.fesom_gpu_forcing_upload
    _chk(u, up(u.ctx.h, _p(x["uv"]), _p(x["w"]), None, _p(x["w"]), _p(x["Kv"]), _p(x["bc"])))


def _read(u, fp32):
    down = u.ctx.L.fesom_gpu_tracer_download_f32 if fp32 else u.ctx.L.fesom_gpu_tracer_download
    for k in range(u.ntr):
        _chk(u, down(u.ctx.h, k, _p(u.out[k]), None))
    return u.out


def prepare(case, seed):
    units = [_unit(case, m, f, kind, ntr, seed + 1000 * i)
             for i, (m, f, kind, ntr) in enumerate(_meshes_of(case))]
    s = dict(case=case, units=units)
    if case["call"] == "batch":
        for u in units:
            _forcing(u, True)
        s["batch"] = G.Batch([u.ctx for u in units])
    torch.cuda.synchronize()
    return s


def run(s):
    case, u = s["case"], s["units"][0]
    fp32 = case["prec"] == "fp32"
    if case["call"] == "loop":
        _forcing(u, fp32)
        if case["redi"]:
            _chk(u, u.ctx.L.fesom_gpu_set_redi(u.ctx.h, _p(u.x["slope"])))
        u.ctx.run_steps(DT, case["steps"])
        return _read(u, fp32)
    if case["call"] == "batch":
        for v in s["units"]:
            _forcing(v, True)
        s["batch"].run_steps(DT, case["steps"])
        return [_read(v, True) for v in s["units"]]
    x = u.x
    if case["call"] == "call":
        _chk(u, u.ctx.L.fesom_gpu_tracer_step(u.ctx.h, u.ntr, u.cfgs, DT, _p(x["uv"]), _p(x["w"]), None, _p(x["w"]),
                                              _p(x["Kv"]), _p(x["bc"]), u.vp, u.op))
        return [x["values"], x["old"]]
    if case["call"] == "noalloc":
        err = C.create_string_buffer(256)
        lev, ulev, bot, hn, ar, av = u.arrays
        rc = G.load().fesom_gpu_vdiff_impl_noalloc(
            C.c_int32(u.N2), C.c_int32(u.nl), _p(lev), _p(ulev), _p(bot), _p(hn), _p(ar), _p(av), _p(x["Kv"]),
            _p(x["bc"]), C.c_double(DT), _p(x["values"]), C.c_void_p(torch.cuda.current_stream().cuda_stream), err, 256)
        if rc:
            raise RuntimeError(err.value.decode())
        return x["values"]
    L, h, o, cfg = u.ctx.L, u.ctx.h, u.out, C.byref(u.cfgs[0])
    _chk(u, L.fesom_gpu_init_tracers_ab(h, cfg, _p(x["values"]), _p(o["valuesAB"]), _p(x["old"])))
    _chk(u, L.fesom_gpu_adv_tra(h, DT, _p(x["uv"]), _p(x["w"]), None, _p(x["w"]), cfg, _p(x["values"]),
                                _p(o["valuesAB"]), _p(o["dttf_h"]), _p(o["dttf_v"])))
    _chk(u, L.fesom_gpu_vdiff_impl(h, DT, cfg, _p(x["Kv"]), _p(x["bc"]), _p(u.star)))
    return dict(o, old=x["old"], star=u.star)


def work(case):
    """Inputs read once, outputs written once: every tracer's values and previous levels in, its new
    values out, the velocities, diffusivity, mesh geometry once; operations of the default schemes."""
    nbytes = flops = 0.0
    for m, _, _, ntr in _meshes_of(case):
        N3 = float(np.sum(m.nlevels_nod2D - m.ulevels_nod2D))
        T3 = float(np.sum(m.nlevels - m.ulevels))
        E3 = 1.5 * T3
        s = 4 if case["prec"] == "fp32" else 8
        n = case["steps"]
        if case["call"] == "noalloc":
            nbytes, flops = s * N3 * 6, 30.0 * N3
            continue
        io = (8 if case["call"] == "call" else s)
        shared = s * (3 * T3 + 10 * N3 + (4 * N3 if case["redi"] else 0))
        nbytes += ntr * io * (1 + case["ab"]) * N3 + shared
        flops += n * ntr * (120.0 * N3 + 45.0 * E3 + (80.0 * N3 if case["redi"] else 0))
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same step in FP64 torch
# ---------------------------------------------------------------------------
class Exact:
    def __init__(self, m, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.N2, self.E2, self.T2, self.L1, self.dev = m.nod2D, m.edge2D, m.elem2D, m.nl - 1, dev
        L1 = self.L1
        lev = torch.arange(L1, device=dev)[None, :]
        self.lev = lev
        self.tri = t(m.elem2D_nodes).long()
        e = t(m.edges).long()
        self.n1, self.n2 = e[:, 0], e[:, 1]
        et = t(m.edge_tri).long()
        self.el1, has2 = et[:, 0], et[:, 1] >= 0
        self.el2 = et[:, 1].clamp(min=0)
        self.nlt, self.nln = t(m.nlevels).long(), t(m.nlevels_nod2D).long()
        self.twet = lev < (self.nlt - 1)[:, None]
        self.nwet = lev < (self.nln - 1)[:, None]
        self.w1 = self.twet[self.el1]
        self.w2 = self.twet[self.el2] & has2[:, None]
        self.ecd = t(m.edge_cross_dxdy)
        self.helem, self.gs = t(m.helem), t(m.gradient_sca)
        self.earea = t(m.elem_area)
        cos = t(m.elem_cos)
        a = R_EARTH * torch.where(has2, 0.5 * (cos[self.el1] + cos[self.el2]), cos[self.el1])
        dxy = t(m.edge_dxdy)
        self.px, self.py = (dxy[:, 0] * a)[:, None], (dxy[:, 1] * R_EARTH)[:, None]
        self.area, self.av = t(m.area), t(m.areasvol)[:, :L1]
        self.av = torch.where(self.nwet, self.av, 1.0)
        self.h, self.hn = (torch.where(self.nwet, t(x), 1.0) for x in (m.hnode, m.hnode_new))
        self.Z, self.zb, self.bot = t(m.Z_3d_n), t(m.zbar_3d_n), t(m.zbar_n_bot)
        # the up and down triangles of each edge and the boundary layers are the mesh's own set-up
        # arrays (muscl_adv_init), integers that the call may be given
        nbl, updn = G.mesh_check(m)
        updn = t(updn).long()
        nlmin = t(m.nlevels_nod2D_min).long()
        gmax = torch.minimum(nlmin[self.n1], nlmin[self.n2])
        inner = (updn[:, 0] >= 0) & (updn[:, 1] >= 0)
        self.inner = inner[:, None] & (lev < (gmax - 1)[:, None])
        self.up, self.dn = updn[:, 0].clamp(min=0), updn[:, 1].clamp(min=0)
        nbl = t(nbl).long()
        self.c1 = (lev + 1 <= nbl[self.n1][:, None]).double()
        self.c2 = (lev + 1 <= nbl[self.n2][:, None]).double()

    def nodes(self, elem):
        """Sum over the elements around each node of an element field."""
        out = torch.zeros((self.N2, self.L1), dtype=torch.float64, device=self.dev)
        v = torch.where(self.twet, elem, 0.0)
        for k in range(3):
            out.index_add_(0, self.tri[:, k], v)
        return out

    def grad(self, T):
        a, b, c = (T[self.tri[:, k]] for k in range(3))
        g = self.gs
        return (g[:, 0:1] * a + g[:, 1:2] * b + g[:, 2:3] * c, g[:, 3:4] * a + g[:, 4:5] * b + g[:, 5:6] * c)

    def divergence(self, F):
        out = torch.zeros((self.N2, self.L1), dtype=torch.float64, device=self.dev)
        out.index_add_(0, self.n1, F)
        return out.index_add_(0, self.n2, -F)

    def vflux(self, uv):
        v = torch.zeros((self.E2, self.L1), dtype=torch.float64, device=self.dev)
        for el, wet, k, sg in ((self.el1, self.w1, 0, 1.0), (self.el2, self.w2, 2, -1.0)):
            c = (uv[el, :, 0] * self.ecd[:, k + 1:k + 2] - uv[el, :, 1] * self.ecd[:, k:k + 1]) * self.helem[el]
            v += sg * torch.where(wet, c, 0.0)
        return v

    def upwind_edge(self, T, vf):
        return -(T[self.n1] * vf.clamp(min=0) + T[self.n2] * vf.clamp(max=0))

    def hor(self, case, T, TA, vf):
        if case["hor"] == "UPW1":
            return self.upwind_edge(TA, vf)
        gx, gy = self.grad(T)
        ea = self.earea[:, None]
        vol = self.nodes(ea.expand(-1, self.L1))
        vol = torch.where(vol > 0, vol, 1.0)
        mx, my = self.nodes(gx * ea) / vol, self.nodes(gy * ea) / vol
        pick = lambda tri, node, q, mean: torch.where(self.inner, q[tri], mean[node])  # noqa: E731
        s1 = self.px * pick(self.up, self.n1, gx, mx) + self.py * pick(self.up, self.n1, gy, my)
        s2 = self.px * pick(self.dn, self.n2, gx, mx) + self.py * pick(self.dn, self.n2, gy, my)
        del gx, gy
        t1, t2 = TA[self.n1], TA[self.n2]
        c1, c2 = (self.c1, self.c2) if case["hor"] == "MUSCL" else (1.0, 1.0)
        d = 2.0 * (t2 - t1)
        return -(vf.clamp(min=0) * (t1 + (d + s1) / 6.0 * c1) + vf.clamp(max=0) * (t2 - (d + s2) / 6.0 * c2))

    def ifaces(self, top, inner):
        """An interface field (N2, nl): `top` at the surface, `inner` at wet interior interfaces, 0 below."""
        out = torch.zeros((self.N2, self.L1 + 1), dtype=torch.float64, device=self.dev)
        out[:, :self.L1] = torch.where(self.nwet, inner, 0.0)
        out[:, 0] = top
        return out

    @staticmethod
    def above(x):
        return torch.cat([x[:, :1], x[:, :-1]], 1)

    def ver_upw(self, T, W):
        w, ar = W[:, :self.L1], self.area[:, :self.L1]
        return self.ifaces(-(w * T * ar)[:, 0], -(T * w.clamp(min=0) + self.above(T) * w.clamp(max=0)) * ar)

    def ver(self, case, TA, W):
        if case["ver"] == "UPW1":
            return self.ver_upw(TA, W)
        w, ar = W[:, :self.L1], self.area[:, :self.L1]
        up = self.above(TA)
        cen = -(0.5 * (up + TA) * w * ar)
        if case["ver"] == "CDIFF":
            return self.ifaces(-(w * TA * ar)[:, 0], cen)
        Z = self.Z
        Zu, Zuu, Zd = self.above(Z), self.above(self.above(Z)), torch.cat([Z[:, 1:], Z[:, -1:]], 1)
        uu, dn = self.above(up), torch.cat([TA[:, 1:], TA[:, -1:]], 1)
        inn = (self.lev >= 2) & (self.lev < (self.nln - 2)[:, None])
        dz = lambda q: torch.where(inn, q, 1.0)  # noqa: E731
        qc, qu, qd = (up - TA) / dz(Zu - Z), (TA - dn) / dz(Z - Zd), (uu - up) / dz(Zuu - Zu)
        zb = self.zb[:, :self.L1]
        m1 = TA + (2.0 * qc + qu) * (zb - Z) / 3.0
        m2 = up + (2.0 * qc + qd) * (zb - Zu) / 3.0
        return self.ifaces(-(w * TA * ar)[:, 0], torch.where(inn, -0.5 * (m1 + m2) * w * ar, cen))

    def diffusion(self, T, Ki, slope):
        """Horizontal diffusion with the Redi slopes and its explicit vertical projection, per unit dt."""
        gx, gy = self.grad(T)
        L1 = self.L1
        tz = torch.zeros((self.N2, L1 + 1), dtype=torch.float64, device=self.dev)
        dz = 0.5 * (self.h[:, :-1] + self.h[:, 1:])
        tz[:, 1:L1] = torch.where(self.nwet[:, 1:], (T[:, :-1] - T[:, 1:]) / dz, 0.0)
        tz = 0.5 * (tz[:, :L1] + tz[:, 1:])
        Kh = 0.5 * (Ki[self.n1] + Ki[self.n2])
        sx, sy = (0.5 * ((tz * slope[:, :, k])[self.n1] + (tz * slope[:, :, k])[self.n2]) for k in (0, 1))
        ecd = lambda k: self.ecd[:, k:k + 1]  # noqa: E731
        h1, h2 = self.helem[self.el1], self.helem[self.el2]
        gx1, gy1, gx2, gy2 = gx[self.el1], gy[self.el1], gx[self.el2], gy[self.el2]
        both = self.w1 & self.w2
        f1 = (-ecd(0) * (gy1 + sy) + ecd(1) * (gx1 + sx)) * h1
        f2 = (ecd(2) * (gy2 + sy) - ecd(3) * (gx2 + sx)) * h2
        f3 = ((ecd(2) - ecd(0)) * (0.5 * (gy1 + gy2) + sy) - (ecd(3) - ecd(1)) * (0.5 * (gx1 + gx2) + sx)) * 0.5 * (h1 + h2)
        F = Kh * torch.where(both, f3, torch.where(self.w1, f1, torch.where(self.w2, f2, 0.0)))
        out = self.divergence(F) / self.av
        del f1, f2, f3, F
        ea = self.earea[:, None]
        p = (slope[:, :, 0] * self.nodes(gx * ea) + slope[:, :, 1] * self.nodes(gy * ea)) / 3.0 / self.av * Ki
        zbar, z = self.depths(self.h)
        zu, pu = self.above(z), self.above(p)
        v = ((zu - zbar[:, :L1]) * pu + (zbar[:, :L1] - z) * p) / torch.where(self.nwet & (self.lev > 0), zu - z, 1.0)
        vd = self.ifaces(torch.zeros(self.N2, dtype=torch.float64, device=self.dev), v * self.area[:, :L1])
        return out + (vd[:, :L1] - vd[:, 1:]) / self.av

    def depths(self, h):
        """Interface and mid depths summed from the bottom up."""
        hw = torch.where(self.nwet, h, 0.0)
        zbar = torch.cat([torch.flip(torch.cumsum(torch.flip(hw, [1]), 1), [1]),
                          torch.zeros((self.N2, 1), dtype=torch.float64, device=self.dev)], 1) + self.bot[:, None]
        return zbar, zbar[:, 1:] + 0.5 * hw

    def vdiff(self, T, Kv, bc):
        """Implicit vertical diffusion: the tridiagonal systems of all columns level by level."""
        L1 = self.L1
        h = self.hn
        r = torch.zeros((self.N2, L1 + 1), dtype=torch.float64, device=self.dev)   # Kv dt area / dz per interface
        r[:, 1:L1] = torch.where(self.nwet[:, 1:], Kv[:, 1:L1] * DT * self.area[:, 1:L1] * 2.0 / (h[:, :-1] + h[:, 1:]), 0.0)
        a, c = r[:, :L1] / self.av, r[:, 1:] / self.av
        up, dn = self.above(T), torch.cat([T[:, 1:], T[:, -1:]], 1)
        rhs = a * (up - T) + c * (dn - T)
        rhs[:, 0] += bc
        b = torch.where(self.nwet, a + c + h, 1.0)
        rhs = torch.where(self.nwet, rhs, 0.0)
        cp, tp = torch.empty_like(T), torch.empty_like(T)
        cp[:, 0], tp[:, 0] = -c[:, 0] / b[:, 0], rhs[:, 0] / b[:, 0]
        for k in range(1, L1):
            den = b[:, k] + a[:, k] * cp[:, k - 1]
            cp[:, k], tp[:, k] = -c[:, k] / den, (rhs[:, k] + a[:, k] * tp[:, k - 1]) / den
        for k in range(L1 - 2, -1, -1):
            tp[:, k] -= cp[:, k] * tp[:, k + 1]
        return torch.where(self.nwet, T + tp, T)

    def ab(self, case, T, old):
        return 1.6 * T - 0.6 * old[..., 0] if case["ab"] == 2 else (23.0 * T - 16.0 * old[..., 0] + 5.0 * old[..., 1]) / 12.0

    def advect(self, case, T, TA, vf, W):
        """The horizontal and vertical advective increments (del_ttf_advhoriz, del_ttf_advvert)."""
        fct, L1, av = case["lim"] == "FCT", self.L1, self.av
        Fh, Fv = self.hor(case, T, TA, vf), self.ver(case, TA, W)
        base = torch.zeros_like(T)
        if fct:
            lo_h, lo_v = self.upwind_edge(T, vf), self.ver_upw(T, W)
            LO = (T * self.h + (self.divergence(lo_h) + lo_v[:, :L1] - lo_v[:, 1:]) * DT / av) / self.hn
            LO = torch.where(self.nwet, LO, 0.0)
            Fh, Fv = Fh - lo_h, Fv - lo_v
            base = LO * self.hn - T * self.h
            del lo_h, lo_v
            ext = []
            for op, pick, fill in ((torch.maximum, "amax", -math.inf), (torch.minimum, "amin", math.inf)):
                q = op(LO, T)
                q = op(op(q[self.tri[:, 0]], q[self.tri[:, 1]]), q[self.tri[:, 2]])
                q = torch.where(self.twet, q, fill)
                x = torch.full((self.N2, L1), fill, dtype=torch.float64, device=self.dev)
                for k in range(3):
                    x.index_reduce_(0, self.tri[:, k], q, pick)
                mid = op(op(self.above(x), x), torch.cat([x[:, 1:], x[:, -1:]], 1))
                ins = (self.lev > 0) & (self.lev < (self.nln - 2)[:, None])
                ext.append(torch.where(ins, mid, x) - LO)
                del q, x, mid
            P = torch.zeros_like(T).index_add_(0, self.n1, Fh.clamp(min=0)).index_add_(0, self.n2, (-Fh).clamp(min=0))
            N = torch.zeros_like(T).index_add_(0, self.n1, Fh.clamp(max=0)).index_add_(0, self.n2, (-Fh).clamp(max=0))
            P += Fv[:, :L1].clamp(min=0) + (-Fv[:, 1:]).clamp(min=0)
            N += Fv[:, :L1].clamp(max=0) + (-Fv[:, 1:]).clamp(max=0)
            rp = torch.where(self.nwet, (ext[0] / (P * DT / av / self.hn + 1e-16)).clamp(max=1.0), 1.0)
            rm = torch.where(self.nwet, (ext[1] / (N * DT / av / self.hn - 1e-16)).clamp(max=1.0), 1.0)
            del ext, P, N
            Fh = Fh * torch.where(Fh >= 0, torch.minimum(rp[self.n1], rm[self.n2]), torch.minimum(rm[self.n1], rp[self.n2]))
            up = lambda r: torch.cat([torch.full_like(r[:, :1], math.inf), r[:, :-1]], 1)  # noqa: E731
            lim = torch.where(Fv[:, :L1] >= 0, torch.minimum(up(rm), rp), torch.minimum(up(rp), rm))
            Fv = torch.cat([Fv[:, :L1] * lim, Fv[:, L1:]], 1)
        wet = lambda q: torch.where(self.nwet, q, 0.0)  # noqa: E731
        return wet(self.divergence(Fh) * DT / av), wet(base + (Fv[:, :L1] - Fv[:, 1:]) * DT / av)

    def step(self, case, T, old, vf, W, Kv, bc, Ki=None, slope=None):
        dh, dv = self.advect(case, T, self.ab(case, T, old), vf, W)
        d = dh + dv
        if Ki is not None:
            d = d + DT * self.diffusion(T, Ki, slope)
        T2 = torch.where(self.nwet, T + (d + T * (self.h - self.hn)) / self.hn, T)
        return self.vdiff(T2, Kv, bc)

    def k33(self, Kv, Ki, slope):
        zbar, z = self.depths(self.hn)
        s = slope[:, :, 2] ** 2 * Ki
        zu, zb, L1 = self.above(z), zbar[:, :self.L1], self.L1
        ins = self.nwet & (self.lev > 0)
        ty = ((zb - z) * self.above(s) + (zu - zb) * s) / torch.where(ins, zu - z, 1.0)
        out = Kv.clone()
        out[:, :L1] += torch.where(ins, ty, 0.0)
        return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    outs = []
    for i, (m, f, kind, ntr) in enumerate(_meshes_of(case)):
        own = torch.float32 if case["prec"] == "fp32" and case["call"] in ("loop", "batch") else torch.float64
        x = _fields(case, m, f, kind, ntr, seed + 1000 * i, dev, own)
        E = Exact(m, dev)
        if case["call"] == "noalloc":
            return E.vdiff(x["values"][0], x["Kv"], x["bc"][0])[None]
        vf, W, Kv = E.vflux(x["uv"].double()), x["w"].double(), x["Kv"].double()
        if case["call"] == "routines":
            T = x["values"][0]
            TA = E.ab(case, T, x["old"][0])
            dh, dv = E.advect(case, T, TA, vf, W)
            old = x["old"].clone()
            old[0, :, :, 1:] = x["old"][0, :, :, :-1]
            old[0, :, :, 0] = T
            return dict(valuesAB=TA, dttf_h=dh, dttf_v=dv, old=old, star=E.vdiff(T, Kv, x["bc"][0]))
        K = E.k33(Kv, x["Ki"], x["slope"]) if case["redi"] else Kv
        vals, olds = [], []
        for k in range(ntr):
            T, old = x["values"][k].double(), x["old"][k].double()
            for _ in range(case["steps"]):
                new = E.step(case, T, old, vf, W, K, x["bc"][k].double(), x.get("Ki"), x.get("slope"))
                old = torch.cat([T[..., None], old[..., :-1]], -1)
                T = new
            vals.append(T)
            olds.append(old)
        if case["call"] == "call":
            return [torch.stack(vals), torch.stack(olds)]
        outs.append(torch.stack(vals))
        del x, E
    return outs if case["call"] == "batch" else outs[0]
