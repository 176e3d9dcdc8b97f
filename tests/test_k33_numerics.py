"""K33 = Kv + Ty of the FP32 form (k32_k33: sums of two FP32 numbers, rounded once) against exact rational
arithmetic and against FP64 arithmetic along the column, restated in numpy FP32 and FP64.  Sampled over
meshes of 20 to 80 layers and the tapered slopes and diffusivities of the Redi configurations, both give the FP32
number nearest to the exact value."""
from fractions import Fraction as F

import numpy as np
import pytest

from fesom2_gb300 import mesh as M

f32 = np.float32


def _nearest(x: F):
    """The FP32 number nearest to x (ties to even)."""
    if x == 0:
        return f32(0)
    s, x = (-1 if x < 0 else 1), abs(x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    e -= F(2) ** e > x
    q = max(e - 23, -149)
    y = x / F(2) ** q
    n, r = divmod(y.numerator, y.denominator)
    n += 2 * r > y.denominator or (2 * r == y.denominator and n & 1)
    return f32(s * float(n) * 2.0 ** q)


def _fma(a, b, c):
    return _nearest(F(float(a)) * F(float(b)) + F(float(c)))


def _two_prod(a, b):
    p = f32(a * b)
    return p, _fma(a, b, -p)


def _two_sum(a, b):
    s = f32(a + b)
    t = f32(s - a)
    return s, f32(f32(a - f32(s - t)) + f32(b - t))


def _mul(x, b):
    h, l = _two_prod(x[0], b)
    return h, _fma(x[1], b, l)


def _pairs(kv, hu, hc, sa, sb, ka, kb):
    x, y = _mul(_mul(_two_prod(sa, sa), ka), hc), _mul(_mul(_two_prod(sb, sb), kb), hu)
    m, d = _two_sum(x[0], y[0]), _two_sum(hu, hc)
    ml = f32(m[1] + f32(x[1] + y[1]))
    q = f32(m[0] / d[0])
    r = f32(_fma(-q, d[1], f32(_fma(-q, d[0], m[0]) + ml)) / d[0])
    t = _two_sum(kv, q)
    return f32(t[0] + f32(t[1] + r))


@pytest.mark.parametrize("layers,nsub,seed", [(20, 4, 1), (47, 4, 2), (80, 3, 3)])
def test_pairs_are_as_near_as_fp64(layers, nsub, seed):
    rng = np.random.default_rng(seed)
    m = M.sphere_mesh(nsub, M.stretched_zbar(layers, 5.0, 250.0), seed=3)
    S = M.make_slopes(m, smax=5e-3, s_cr=4e-3)[:, :, 2].astype(f32)
    Ki = np.broadcast_to(3000.0 * m.areasvol[:, :1] / 1e10, S.shape).astype(f32)
    hn, bot = m.hnode_new.astype(f32), m.zbar_n_bot.astype(f32)
    Kv = (10.0 ** rng.uniform(-6, -1, (m.nod2D, m.nl))).astype(f32)
    far64 = far = 0.0
    count = 0
    for n in rng.choice(m.nod2D, 12, replace=False):
        top, last = m.ulevels_nod2D[n], m.nlevels_nod2D[n]
        zb = float(bot[n])
        Zc = zb + float(hn[n, last - 2]) / 2.0
        for nz in range(last - 1, top, -1):
            hu, hc, sa, sb = hn[n, nz - 2], hn[n, nz - 1], S[n, nz - 2], S[n, nz - 1]
            ka, kb, kv = Ki[n, nz - 2], Ki[n, nz - 1], Kv[n, nz - 1]
            zbn = zb + float(hc)
            Zu = zbn + float(hu) / 2.0
            zinv = 1.0 / (Zu - Zc)
            Ty = (zbn - Zc) * zinv * float(sa) ** 2 * float(ka) + (Zu - zbn) * zinv * float(sb) ** 2 * float(kb)
            zb, Zc = zbn, Zu
            hu_, hc_ = F(float(hu)), F(float(hc))
            exact = F(float(kv)) + (hc_ * F(float(sa)) ** 2 * F(float(ka)) + hu_ * F(float(sb)) ** 2 * F(float(kb))) / (hu_ + hc_)
            err = [abs(float((F(float(v)) - exact) / exact)) for v in (f32(float(kv) + Ty), _pairs(kv, hu, hc, sa, sb, ka, kb))]
            # half an ulp of the rounding plus the pairs' own 2^-44
            assert err[1] <= 2.0 ** -24 + 2.0 ** -44, (n, nz, err)
            far64, far = max(far64, err[0]), max(far, err[1])
            count += 1
    assert count > 100 and far <= far64 + 2.0 ** -44, (far, far64)
