"""FP32 contexts on the caller's device arrays, which kernels read and write as they are: the forcing in
one launch (w and w_e one array or two, w_i given or not, bases off a 16-byte boundary, tracers that
leave slots of a group empty) and tracers into and out of their slots.  A step from them equals the step
from host arrays bit for bit."""
import ctypes as C

import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


@pytest.mark.parametrize("ntr,ab,shift,split_w,flux", [(1, 2, 0, False, True), (3, 3, 1, True, False),
                                                        (5, 2, 3, True, True), (6, 3, 0, False, False)])
def test_device_arrays_equal_host_arrays(ntr, ab, shift, split_w, flux):
    mesh = M.channel_mesh(9, 13, 5000.0, M.stretched_zbar(33, 10.0, 200.0), seamounts=2, seed=5, partial_cells=True)
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    rng = np.random.default_rng(7)
    f32 = lambda a: np.ascontiguousarray(a, dtype=np.float32)  # noqa: E731
    uv, w, Kv = f32(f.uv), f32(f.w), f32(f.Kv)
    we = f32(0.5 * w) if split_w else w
    wi = f32(w - we) if split_w else None
    bc = f32(1e-4 * rng.standard_normal((ntr, mesh.nod2D))) if flux else None
    val = [f32(t) for t in M.make_tracers(mesh, "channel", ntr=ntr, seed=4)]
    old = [f32(v[..., None] * (1.0 + 1e-3 * rng.standard_normal(v.shape + (ab - 1,)))) for v in val]

    def on_device(a):
        if a is None:
            return None
        t = torch.empty(a.size + shift, dtype=torch.float32, device="cuda")
        t[shift:] = torch.from_numpy(a.reshape(-1)).cuda()
        return t[shift:]

    outs = []
    for dev in (False, True):
        put = on_device if dev else (lambda a: a)
        ctx = G.Context(mesh, G.PREC_FP32, max_tracers=ntr)
        ctx.set_wsplit(split_w)
        ctx.state_setup([G.tra_cfg(id=k + 1, ab_order=ab) for k in range(ntr)])
        duv, dw, dKv, dbc, dwi = put(uv), put(w), put(Kv), put(bc), put(wi)
        dwe = put(we) if split_w else dw
        assert ctx.L.fesom_gpu_forcing_upload_f32(ctx.h, _p(duv), _p(dw), _p(dwi), _p(dwe), _p(dKv), _p(dbc)) == 0
        keep = [(put(v), put(o)) for v, o in zip(val, old)]
        for k, (v, o) in enumerate(keep):
            assert ctx.L.fesom_gpu_tracer_upload_f32(ctx.h, k, _p(v), _p(o)) == 0
        ctx.run_steps(f.dt, 2)
        res = []
        for k in range(ntr):
            n = val[k].size
            if dev:
                a = torch.full((n + shift + 4,), 7.0, dtype=torch.float32, device="cuda")
                b = torch.full((n * (ab - 1) + shift + 4,), 7.0, dtype=torch.float32, device="cuda")
                assert ctx.L.fesom_gpu_tracer_download_f32(ctx.h, k, _p(a[shift:]), _p(b[shift:])) == 0
                assert ctx.status() == 0
                for t, m in ((a, n), (b, n * (ab - 1))):  # nothing written beside the array
                    assert (t[:shift] == 7.0).all() and (t[shift + m:] == 7.0).all()
                res += [a[shift:shift + n].cpu().numpy(), b[shift:shift + n * (ab - 1)].cpu().numpy()]
            else:
                a, b = np.empty(n, np.float32), np.empty(n * (ab - 1), np.float32)
                assert ctx.L.fesom_gpu_tracer_download_f32(ctx.h, k, _p(a), _p(b)) == 0
                assert ctx.status() == 0
                res += [a, b]
        outs.append(res)
        ctx.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
