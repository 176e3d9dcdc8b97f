// fp64_stages.cuh -- the advection stages of the FP64 form.
//
// All of these kernels are bound by the FP64 unit (72-98 % of its one warp instruction in 19 cycles per
// SM; DRAM under 10 %), so they are built to issue as few FP64 warp instructions as possible for the
// reference's bits:
//   * comparisons, maxima, absolute values and selections run on integers (fp64_arith.cuh);
//   * v + |v| and v - |v| are 2v or 0: an upwind sum T1 (v + |v|) + T2 (v - |v|) is one product of
//     the upwind value, and 0.5 * (T * 2v) is T * v; both only while the operand that drops out
//     is finite (0 * inf is a NaN the reference would produce), else the full expression;
//   * divisions by shared or constant divisors take 3 or 4 instructions instead of 9;
//   * the wet levels of a tile of entities are dealt to the threads one after another (Tile), so
//     every warp but a tile's last is full.  A warp per column left 27 to 50 % of the lanes idle
//     (47 layers are 32 + 15 lanes), and an FP64 instruction costs its 19 cycles however many
//     lanes take part.
#pragma once
#include <type_traits>

#include "fesom_internal.h"
#include "fp64_arith.cuh"
#include "tile.cuh"
#include "tracer_kernels.cuh"

namespace fesom {

// -(0.5 (a (v + |v|) + b (v - |v|))), the upwind flux of a (v > 0) and b (v < 0)
__device__ __forceinline__ double upwind64(double a, double b, double v) {
    const bool neg = neg64(v);
    const double x = neg ? b : a, y = neg ? a : b;
    if (nonfinite64(y) || nonfinite64(v)) {
        const double av = fabs(v);
        return -(0.5 * (a * (v + av) + b * (v - av)));
    }
    return -(x * v);
}

// ===========================================================================
// init_tracers_AB: valuesAB and the valuesold shift (src/oce_tracer_mod.F90:46-123)
// ===========================================================================
static __global__ void k_ab(DTracers<double> tr, size_t n, int ab) {
    const double ca = 0.5 + kABEpsilon, cb = 1.5 + kABEpsilon;
    for (int t = 0; t < tr.ntr; t++) {
        double *T = tr.T + t * tr.sN, *TAB = tr.TAB + t * tr.sN;
        double *O = tr.Told + t * tr.sN * (ab - 1);
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
            const double v = T[i];
            if (ab == 2) {
                TAB[i] = -(ca * O[i]) + cb * v;
                O[i] = v;
            } else {
                const double2 o = reinterpret_cast<double2 *>(O)[i];
                // 16 o1 is exact: one rounding, as in 5 o2 - 16 o1
                TAB[i] = div_3x2k<12>(__fma_rn(-16.0, o.x, 5.0 * o.y) + 23.0 * v);
                reinterpret_cast<double2 *>(O)[i] = make_double2(v, o.x);
            }
        }
    }
}

// ===========================================================================
// tracer_gradient_elements (src/oce_tracer_mod.F90:147-188): a tile of elements
// ===========================================================================
static __global__ void __launch_bounds__(kTileThreads)
k_trxy(DTopo tp, DGeom<double> g, DTracers<double> tr, int tile) {
    __shared__ Tile S;
    __shared__ int nod[kTileMax][3];
    const int L1 = tp.L1, el0 = blockIdx.x * tile;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, el = el0 + j;
        const bool ok = j < tile && el < tp.T2;
        if (ok)
            for (int k = 0; k < 3; k++) nod[j][k] = tp.t_n[3 * el + k];
        S.fill(j, ok ? tp.t_ulev[el] : 1, ok ? tp.t_nlev[el] - tp.t_ulev[el] : 0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
        const int j = S.find(i), el = el0 + j, nz = S.top[j] + i - S.pre[j];
        const size_t a = ix1(nz, nod[j][0], L1), b = ix1(nz, nod[j][1], L1), c = ix1(nz, nod[j][2], L1);
        const double *gs = g.gs + 6 * (size_t)el;
        const double g0 = gs[0], g1 = gs[1], g2 = gs[2], g3 = gs[3], g4 = gs[4], g5 = gs[5];
        for (int t = 0; t < tr.ntr; t++) {
            const double *T = tr.T + t * tr.sN;
            const double ta = T[a], tb = T[b], tc = T[c];
            reinterpret_cast<double2 *>(tr.trxy + t * tr.sT)[ix1(nz, el, L1)] =
                make_double2(g0 * ta + g1 * tb + g2 * tc, g3 * ta + g4 * tb + g5 * tc);
        }
    }
}

// ===========================================================================
// Edge fluxes: adv_tra_hor_upw1 (LO, values) and adv_tra_hor_muscl / _mfct /
// _upw1 (HO, valuesAB) with fill_up_dn_grad inlined
// (src/oce_adv_tra_hor.F90:64-834, src/oce_muscl_adv.F90:356-525).
// Writes FLO (FCT only) and ADh = HO - LO (FCT) or HO (no limiter).
//
// With adv_ph = 0 only the upwind end's reconstruction has a weight, so only it is formed (the
// downwind one enters as 0 times a finite number); adv_ph /= 0, or a value or gradient at either
// end that is not finite, takes the full expression.
// Bound by FP64 issue.  FP64 instructions per edge-layer (FCT, MUSCL): 13 per tracer and 10
// shared by the tracers, against about 70 per tracer: 4.84 -> 1.46 ms on the sphere of 7 subdivisions,
// 48 levels, 2 tracers (1.70 before the node means were set aside and the registers bounded).
// ===========================================================================
// whether the gradient of node's reconstruction at nz (triangle el, or the node mean) is not finite
__device__ __forceinline__ bool grad_bad(const DTopo &tp, const double *txy, bool tri, int el, int node, int nz) {
    const double2 *xy = reinterpret_cast<const double2 *>(txy);
    if (tri) {
        const double2 v = xy[ix1(nz, el, tp.L1)];
        return nonfinite64(v.x) || nonfinite64(v.y);
    }
    bool bad = false;
    for (int k = tp.nie_ptr[node]; k < tp.nie_ptr[node + 1]; k++) {
        const int e = tp.nie_idx[k];
        if (tp.t_nlev[e] - 1 < nz || nz < tp.t_ulev[e]) continue;
        const double2 v = xy[ix1(nz, e, tp.L1)];
        bad = bad || nonfinite64(v.x) || nonfinite64(v.y);
    }
    return bad;
}

// both reconstructions and the flux of adv_tra_hor_muscl / _mfct for any adv_ph
static __device__ __noinline__ double edge_ho_full(const DTopo &tp, const DGeom<double> &g, const double *txy,
                                                   const DCfg &c, bool tri, int up, int dn, int n1, int n2, int nz,
                                                   double t1, double t2, double vf, double ca, double cb, bool in1,
                                                   bool in2, double fin) {
    double g1, g2, g3, g4;
    if (tri) {
        g1 = txy[2 * ix1(nz, up, tp.L1)];
        g3 = txy[2 * ix1(nz, up, tp.L1) + 1];
        g2 = txy[2 * ix1(nz, dn, tp.L1)];
        g4 = txy[2 * ix1(nz, dn, tp.L1) + 1];
    } else {
        node_mean_grad(tp, g, txy, n1, nz, g1, g3);
        node_mean_grad(tp, g, txy, n2, nz, g2, g4);
    }
    double q2 = (2.0 * (t2 - t1) + ca * g2 + cb * g4) / 6.0, q1 = (2.0 * (t2 - t1) + ca * g1 + cb * g3) / 6.0;
    if (c.hor == 0) {
        q2 = q2 * (in2 ? 1.0 : 0.0);
        q1 = q1 * (in1 ? 1.0 : 0.0);
    }
    const double Tm2 = t2 - q2, Tm1 = t1 + q1, no = c.ph, avf = fabs(vf);
    const double cHO = (vf + avf) * Tm1 + (vf - avf) * Tm2;
    return -(0.5 * (1.0 - no) * cHO) - vf * no * 0.5 * (Tm1 + Tm2) - fin;
}

struct EdgeData {
    int n1, n2, el1, el2, nu1, nl1, nu2, nl2, up, dn, gmin, gmax, nbl1, nbl2;
    double dX1, dY1, dX2, dY2, ca, cb;  // ca = edge_dxdy(1) a, cb = edge_dxdy(2) r_earth
};

// The edge-layers whose gradients are node means (the last layers over a slope, every layer at a
// coast: 2 % of a sphere's) cost five times the others' instructions, and lie in half of the
// warps: they are set aside and take their own passes, full warps again.
static __global__ void __launch_bounds__(kTileThreads, 8)
k_edge_flux(DTopo tp, DGeom<double> g, DForcing<double> f, DTracers<double> tr, int tile, int any_ho) {
    extern __shared__ int aside[];
    __shared__ int n_aside;
    __shared__ Tile S;
    __shared__ EdgeData Ed[kTileMax];
    const int L1 = tp.L1, e0 = blockIdx.x * tile;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, e = e0 + j;
        const bool ok = j < tile && e < tp.E2;
        if (ok) {
            EdgeData &E = Ed[j];
            const int el1 = tp.e_t1[e], el2 = tp.e_t2[e], n1 = tp.e_n1[e], n2 = tp.e_n2[e];
            E.n1 = n1;
            E.n2 = n2;
            E.el1 = el1;
            E.el2 = el2;
            E.nl1 = tp.t_nlev[el1] - 1;
            E.nu1 = tp.t_ulev[el1];
            E.dX1 = g.ecd[4 * (size_t)e];
            E.dY1 = g.ecd[4 * (size_t)e + 1];
            double a = kREarth * g.elem_cos[el1];
            E.nl2 = E.nu2 = 0;
            E.dX2 = E.dY2 = 0.0;
            if (el2 >= 0) {
                E.dX2 = g.ecd[4 * (size_t)e + 2];
                E.dY2 = g.ecd[4 * (size_t)e + 3];
                E.nl2 = tp.t_nlev[el2] - 1;
                E.nu2 = tp.t_ulev[el2];
                a = 0.5 * (a + kREarth * g.elem_cos[el2]);
            }
            E.ca = g.edxy[2 * (size_t)e] * a;
            E.cb = g.edxy[2 * (size_t)e + 1] * kREarth;
            E.up = tp.e_up[e];
            E.dn = tp.e_dn[e];
            const bool inner = E.up >= 0 && E.dn >= 0;
            E.gmin = inner ? max(tp.n_ulevmax[n1], tp.n_ulevmax[n2]) : 1;
            E.gmax = inner ? min(tp.n_nlevmin[n1], tp.n_nlevmin[n2]) - 1 : 0;
            E.nbl1 = tp.n_nbl[n1];
            E.nbl2 = tp.n_nbl[n2];
        }
        S.fill(j, ok ? tp.e_lo[e] : 1, ok ? tp.e_hi[e] - tp.e_lo[e] + 1 : 0);
    }
    if (threadIdx.x == 32) n_aside = 0;
    __syncthreads();
    auto layer = [&](int i, auto pass) {
        constexpr bool means = decltype(pass)::value;
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j];
        const EdgeData &E = Ed[j];
        const bool tri = nz >= E.gmin && nz <= E.gmax;
        if (!means && !tri && any_ho) {
            aside[atomicAdd(&n_aside, 1)] = i;
            return;
        }
        const size_t ke = ix1(nz, e0 + j, L1), k1 = ix1(nz, E.n1, L1), k2 = ix1(nz, E.n2, L1);
        // segment rule of the reference's five loops (A..E)
        const int fnl12 = min(E.nl1, E.nl2), fnu12 = max(E.nu1, E.nu2);
        int seg = 0;
        if (nz >= E.nu1 && nz <= fnu12 - 1) seg = 1;
        else if (E.nu2 > 0 && nz >= E.nu2 && nz <= fnu12 - 1) seg = 2;
        else if (nz >= fnu12 && nz <= fnl12) seg = 3;
        else if (nz >= fnl12 + 1 && nz <= E.nl1) seg = 1;
        else if (nz >= fnl12 + 1 && nz <= E.nl2) seg = 2;
        double vf = 0.0;
        if (seg & 1) {
            const size_t k = ix1(nz, E.el1, L1);
            const double2 v = reinterpret_cast<const double2 *>(f.uv)[k];
            vf = (-(v.y * E.dX1) + v.x * E.dY1) * g.helem[k];
        }
        if (seg & 2) {
            const size_t k = ix1(nz, E.el2, L1);
            const double2 v = reinterpret_cast<const double2 *>(f.uv)[k];
            const double v2 = (v.y * E.dX2 - v.x * E.dY2) * g.helem[k];
            vf = (seg == 3) ? vf + v2 : v2;
        }
        const bool neg = neg64(vf), vbad = nonfinite64(vf);
        for (int t = 0; t < tr.ntr; t++) {
            const DCfg c = tr.cfg[t];
            double flo = 0.0, ad = 0.0;
            if (seg) {
                const double *T = tr.T + t * tr.sN, *TA = tr.TAB + t * tr.sN;
                const double t1 = TA[k1], t2 = TA[k2];
                if (c.lim) flo = upwind64(T[k1], T[k2], vf);
                if (c.hor == 2) {
                    ad = upwind64(t1, t2, vf) - flo;
                } else {
                    const double *txy = tr.trxy + t * tr.sT;
                    // short: the upwind reconstruction alone, while everything it leaves out is finite
                    bool full = c.ph != 0.0 || vbad || nonfinite64(t1) || nonfinite64(t2) ||
                                grad_bad(tp, txy, !means, neg ? E.up : E.dn, neg ? E.n1 : E.n2, nz);
                    if (!full) {
                        double2 gr;
                        if (means) node_mean_grad(tp, g, txy, neg ? E.n2 : E.n1, nz, gr.x, gr.y);
                        else gr = reinterpret_cast<const double2 *>(txy)[ix1(nz, neg ? E.dn : E.up, L1)];
                        // 2 (t2 - t1) is exact: one rounding in the fused sum, as in the reference's
                        double q = div_3x2k<6>(__fma_rn(2.0, t2 - t1, E.ca * gr.x) + E.cb * gr.y);
                        if (c.hor == 0 && (neg ? E.nbl2 : E.nbl1) < nz) q = q * 0.0;
                        const double Tm = (neg ? t2 : t1) + (neg ? -q : q);
                        ad = -(Tm * vf) - flo;
                        full = nonfinite64(Tm);  // adv_ph (Tm1 + Tm2) is then 0 * inf
                    }
                    if (full)
                        ad = edge_ho_full(tp, g, txy, c, !means, E.up, E.dn, E.n1, E.n2, nz, t1, t2, vf, E.ca, E.cb,
                                          E.nbl1 >= nz, E.nbl2 >= nz, flo);
                }
            }
            if (c.lim) tr.FLO[t * tr.sE + ke] = flo;
            tr.ADh[t * tr.sE + ke] = ad;
        }
    };
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) layer(i, std::false_type{});
    __syncthreads();
    for (int q = threadIdx.x; q < n_aside; q += kTileThreads) layer(aside[q], std::true_type{});
}

// ===========================================================================
// Node columns, stage 1: LO solution (edge gather of the upwind fluxes,
// adv_tra_ver_upw1 with w_e, src/oce_adv_tra_driver.F90:122-250) and the
// vertical high-order flux minus the LO flux (adv_tra_ver_qr4c / _upw1 / _cdiff / _ppm with w,
// src/oce_adv_tra_ver.F90:244-695).  Without a limiter only the HO vertical
// flux (with w_e) is formed.
//
// Two passes over a tile of nodes: the upwind flux and the gradient quotient
// (T(nz-1) - T(nz)) / (Z(nz-1) - Z(nz)) of every interface once into shared memory, then the
// layers, which read both neighbours' (the quotient was formed three times, the flux twice).
// Every centred or surface flux is -(0.5 (A + B) W area) - fin with A, B chosen per interface;
// the factor 0.5 is exact, so it is applied in the last, fused operation.  51.8 -> 18.2 M FP64 warp
// instructions on the sphere of 7 subdivisions, 48 levels, 2 tracers: 3.09 -> 1.11 ms.
// ===========================================================================
// the upwind flux of adv_tra_ver_upw1 through interface nz above layer nz (top: the surface)
__device__ __forceinline__ double ver_upw64(double T0, double Tu, double W, double ar, bool top) {
    if (top) return -(W * T0 * ar);
    const bool neg = neg64(W);
    const double x = neg ? Tu : T0, y = neg ? T0 : Tu;
    if (nonfinite64(y) || nonfinite64(W)) {
        const double aW = fabs(W);
        return -(0.5 * (T0 * (W + aW) + Tu * (W - aW)) * ar);
    }
    return -(x * W * ar);
}

static __global__ void __launch_bounds__(kTileThreads, 7)
k_node_lo(DTopo tp, DGeom<double> g, DForcing<double> f, DTracers<double> tr, double dt, int tile) {
    extern __shared__ __align__(16) double sm64[];
    __shared__ Tile S;
    const int L1 = tp.L1, nl = tp.nl, n0 = blockIdx.x * tile;
    double *fl = sm64, *qc = sm64 + (size_t)tile * L1;
    if (threadIdx.x < 32) {
        const int n = n0 + threadIdx.x;
        const bool ok = threadIdx.x < tile && n < tp.N2;
        S.fill(threadIdx.x, ok ? tp.n_ulev[n] : 1, ok ? tp.n_nlev[n] - tp.n_ulev[n] : 0);
    }
    for (int t = 0; t < tr.ntr; t++) {
        const DCfg c = tr.cfg[t];
        const bool fct = c.lim != 0;
        const double *T = tr.T + t * tr.sN, *TA = tr.TAB + t * tr.sN, *FLO = tr.FLO + t * tr.sE;
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            const bool top = i == S.pre[j];
            const size_t k = ix1(nz, n, L1), kv = ixn(nz, n, nl);
            if (fct) fl[i] = ver_upw64(T[k], top ? 0.0 : T[k - 1], f.we[kv], g.area[kv], top);
            if (c.ver == 0 && !top) qc[i] = (TA[k - 1] - TA[k]) / (g.Z3[k - 1] - g.Z3[k]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            const int nzmin = S.top[j], nzmax = nzmin + S.pre[j + 1] - S.pre[j];
            const bool top = nz == nzmin, bot = nz == nzmax - 1;
            const size_t k = ix1(nz, n, L1), kv = ixn(nz, n, nl);
            double fin = 0.0;
            if (fct) {
                fin = fl[i];
                const double f1 = bot ? 0.0 : fl[i + 1];
                double acc = 0.0;
                for (int q = tp.ne_ptr[n]; q < tp.ne_ptr[n + 1]; q++) {
                    const int code = tp.ne_idx[q], e = code >= 0 ? code : ~code;
                    if (nz < tp.e_lo[e] || nz > tp.e_hi[e]) continue;
                    const double x = FLO[ix1(nz, e, L1)];
                    acc = acc + (code >= 0 ? x : -x);
                }
                const double h = T[k] * g.hnode[k];
                tr.LO[t * tr.sN + k] = sdiv64(h + sdiv64((acc + (fin - f1)) * dt, g.areasvol[kv], g.rav[kv]),
                                              g.hnode_new[k], g.rhn[k]);
                // with the split vertical velocity the LO part of the antidiffusive flux is the
                // upwind flux of the full w (oce_adv_tra_driver.F90:323-334)
                if (f.wsplit) fin = ver_upw64(T[k], top ? 0.0 : T[k - 1], f.w[kv], g.area[kv], top);
            }
            const double *pw = fct ? f.w : f.we;
            double v;
            if (c.ver == 3) {
                v = ver_ppm_flux(TA, pw, g.area, g.hnode_new, g.hnode, dt, nz, n, nzmin, nzmax, L1, nl, fin);
            } else {
                const double W = pw[kv], ar = g.area[kv], t0 = TA[k];
                if (c.ver == 1) {
                    v = ver_upw64(t0, top ? 0.0 : TA[k - 1], W, ar, top) - fin;
                } else {
                    double A = top ? t0 : TA[k - 1], B = t0;
                    const bool inner = c.ver == 0 && nz >= nzmin + 2 && !bot;
                    if (inner) {
                        const double zb = g.zbar3[kv], q0 = qc[i];
                        // 2 qc is exact: one rounding in the fused sum, as in the reference's
                        A = A + div_3x2k<3>(__fma_rn(2.0, q0, qc[i - 1]) * (zb - g.Z3[k - 1]));
                        B = B + div_3x2k<3>(__fma_rn(2.0, q0, qc[i + 1]) * (zb - g.Z3[k]));
                    }
                    if (inner && (c.pv != 1.0 || nonfinite64(W) || nonfinite64(A) || nonfinite64(B))) {
                        const double no = c.pv, aW = fabs(W);
                        const double Tmean = (W + aW) * B + (W - aW) * A;
                        v = (-(0.5 * (1.0 - no) * Tmean) - no * (0.5 * (B + A)) * W) * ar - fin;
                    } else {
                        const double P = (A + B) * W * ar;
                        v = __fma_rn(-0.5, P, -fin);
                        // a two-layer column writes its middle interface twice (nzmin+1, nzmax-1)
                        if (c.ver == 0 && bot && nz == nzmin + 1) v = -(0.5 * P) - v;
                    }
                }
            }
            tr.ADv[t * tr.sNI + kv] = v;
            if (bot) tr.ADv[t * tr.sNI + kv + 1] = 0.0;
        }
    }
}

// ===========================================================================
// FCT bounds a1-a3 and b1 + b2: the bounds of a node-layer over the node's elements and the
// adjacent layers, the sums of positive / negative antidiffusive fluxes (vertical, then edges in
// ascending order) and the ratios R+ / R- (src/oce_adv_tra_fct.F90:124-405), in one kernel.
//
// The maximum over the node's wet elements is the maximum over the node and the neighbours whose
// edge is wet (each wet element is the wet side of two of the node's edges), plus -bignumber
// where an element of the node is dry: 7 values instead of 18.  Maxima run on integer keys in
// shared memory; only the sums and quotients are FP64 instructions (about 45 per node-layer and
// tracer, 165 in two kernels before; 4.17 -> 0.74 ms on the sphere of 7 subdivisions, 2 tracers).  A mesh whose edges do not cover its elements' sides, or a
// value that is not a number, takes the elements themselves with the FP64 comparisons.
// ===========================================================================
// max / min over the elements of node n at layer nz in the order of the reference's loop
static __device__ __noinline__ void bounds_elements(const DTopo &tp, const double *T, const double *LO, int n, int nz,
                                                    double &mx, double &mn) {
    const int L1 = tp.L1, k0 = tp.nie_ptr[n], k1 = tp.nie_ptr[n + 1];
    mx = mn = 0.0;
    for (int k = k0; k < k1; k++) {
        const int el = tp.nie_idx[k];
        double amx = -kBigNumber, amn = kBigNumber;
        if (nz >= tp.t_ulev[el] && nz <= tp.t_nlev[el] - 1) {
            const size_t a = ix1(nz, tp.t_n[3 * el], L1), b = ix1(nz, tp.t_n[3 * el + 1], L1),
                         c = ix1(nz, tp.t_n[3 * el + 2], L1);
            amx = rmax(rmax(rmax(LO[a], T[a]), rmax(LO[b], T[b])), rmax(LO[c], T[c]));
            amn = rmin(rmin(rmin(LO[a], T[a]), rmin(LO[b], T[b])), rmin(LO[c], T[c]));
        }
        mx = k == k0 ? amx : rmax(mx, amx);
        mn = k == k0 ? amn : rmin(mn, amn);
    }
}

// rmin(1, b / fl); b and fl of one sign, |b| >= |fl|: the quotient rounds to 1 or more
__device__ __forceinline__ double ratio1(double b, double fl) {
    const unsigned long long ub = (unsigned long long)__double_as_longlong(b),
                             uf = (unsigned long long)__double_as_longlong(fl);
    if ((long long)(ub ^ uf) >= 0 && (ub << 1) >= (uf << 1) && !nonfinite64(b) && !zero64(fl)) return 1.0;
    return rmin(1.0, b / fl);
}

static __global__ void __launch_bounds__(kTileThreads, 12)
k_bounds_rpm(DTopo tp, DGeom<double> g, DTracers<double> tr, double dt, int tile) {
    extern __shared__ __align__(16) long long smk[];
    __shared__ Tile S;
    __shared__ int wlo[kTileMax], whi[kTileMax];  // the levels at which every element of the node is wet
    const int L1 = tp.L1, nl = tp.nl, n0 = blockIdx.x * tile;
    long long *kmx = smk, *kmn = smk + (size_t)tile * L1;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, n = n0 + j;
        const bool ok = j < tile && n < tp.N2;
        if (ok) {
            int lo = 1, hi = nl;
            for (int k = tp.nie_ptr[n]; k < tp.nie_ptr[n + 1]; k++) {
                const int el = tp.nie_idx[k];
                lo = max(lo, tp.t_ulev[el]);
                hi = min(hi, tp.t_nlev[el] - 1);
            }
            wlo[j] = lo;
            whi[j] = hi;
        }
        S.fill(j, ok ? tp.n_ulev[n] : 1, ok ? tp.n_nlev[n] - tp.n_ulev[n] : 0);
    }
    for (int t = 0; t < tr.ntr; t++) {
        if (!tr.cfg[t].lim) continue;
        const double *T = tr.T + t * tr.sN, *LO = tr.LO + t * tr.sN;
        const double *ADv = tr.ADv + t * tr.sNI, *ADh = tr.ADh + t * tr.sE;
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            const bool dry = nz < wlo[j] || nz > whi[j];
            const size_t k = ix1(nz, n, L1);
            const double lo0 = LO[k], t0 = T[k];
            bool bad = nan64(lo0) || nan64(t0), wet = false;
            const long long a = key64(lo0), b = key64(t0);
            long long mx = max(a, b), mn = min(a, b);
            for (int q = tp.ne_ptr[n]; q < tp.ne_ptr[n + 1]; q++) {
                const int code = tp.ne_idx[q], e = code >= 0 ? code : ~code;
                if (nz < tp.e_lo[e] || nz > tp.e_hi[e]) continue;
                wet = true;
                const size_t m = ix1(nz, code >= 0 ? tp.e_n2[e] : tp.e_n1[e], L1);
                const double lm = LO[m], tm = T[m];
                bad = bad || nan64(lm) || nan64(tm);
                const long long ka = key64(lm), kb = key64(tm);
                mx = max(mx, max(ka, kb));
                mn = min(mn, min(ka, kb));
            }
            if (dry) {
                const long long big = __double_as_longlong(kBigNumber), nbig = key64(-kBigNumber);
                mx = wet ? max(mx, nbig) : nbig;
                mn = wet ? min(mn, big) : big;
            }
            if (bad || !tp.ring_ok) {
                double x, y;
                bounds_elements(tp, T, LO, n, nz, x, y);
                mx = key64(x);
                mn = key64(y);
            }
            kmx[i] = mx;
            kmn[i] = mn;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            const bool end = i == S.pre[j] || i == S.pre[j + 1] - 1;
            const size_t k = ix1(nz, n, L1), kv = ixn(nz, n, nl);
            long long mx = kmx[i], mn = kmn[i];
            if (!end) {
                const long long xu = kmx[i - 1], xd = kmx[i + 1], yu = kmn[i - 1], yd = kmn[i + 1];
                if (nan64(unkey64(xu)) || nan64(unkey64(mx)) || nan64(unkey64(xd)) || nan64(unkey64(yu)) ||
                    nan64(unkey64(mn)) || nan64(unkey64(yd))) {
                    mx = key64(rmax(rmax(unkey64(xu), unkey64(mx)), unkey64(xd)));
                    mn = key64(rmin(rmin(unkey64(yu), unkey64(mn)), unkey64(yd)));
                } else {
                    mx = max(max(xu, mx), xd);
                    mn = min(min(yu, mn), yd);
                }
            }
            const double lo = LO[k], bx = unkey64(mx) - lo, bn = unkey64(mn) - lo;
            // sums of the fluxes into (P) and out of (M) the layer; a flux adds to one of them
            double P = 0.0, M = 0.0;
            bool bad = false;
            auto add = [&](double x) {
                bad = bad || nan64(x);
                const bool neg = neg64(x);
                const double s = (neg ? M : P) + x;
                P = neg ? P : s;
                M = neg ? s : M;
            };
            add(ADv[kv]);
            add(-ADv[kv + 1]);
            for (int q = tp.ne_ptr[n]; q < tp.ne_ptr[n + 1]; q++) {
                const int code = tp.ne_idx[q], e = code >= 0 ? code : ~code;
                if (nz < tp.e_lo[e] || nz > tp.e_hi[e]) continue;
                const double x = ADh[ix1(nz, e, L1)];
                add(code >= 0 ? x : -x);
            }
            if (bad) P = M = __longlong_as_double(0x7ff8000000000000ll);  // both sums take a NaN flux
            const double av = g.areasvol[kv], hn = g.hnode_new[k];
            const double2 ra = g.rav[kv], rh = g.rhn[k];
            const double fp = sdiv64(sdiv64(P * dt, av, ra), hn, rh) + kFluxEps;
            const double fm = sdiv64(sdiv64(M * dt, av, ra), hn, rh) - kFluxEps;
            tr.bmax[t * tr.sN + k] = ratio1(bx, fp);
            tr.bmin[t * tr.sN + k] = ratio1(bn, fm);
        }
    }
}

// ===========================================================================
// FCT b3 limiting + oce_tra_adv_flux2dtracer (src/oce_adv_tra_fct.F90:425-500,
// src/oce_adv_tra_driver.F90:494-646) + (mode 1) the del_ttf sum and the T*
// update of diff_tracers_ale (src/oce_ale_tracer.F90:319-321, 743-754).
// The limited edge flux is formed at each end node from R+/R- of both ends; a limited interface
// flux once, in a first pass over the tile.  About 60 FP64 instructions per node-layer and
// tracer (118 before: six of its divisions are by areasvol, at 4 instead of 9 each): 2.96 -> 1.23 ms on
// the sphere of 7 subdivisions, 48 levels, 2 tracers, at the FP64 unit's rate.
// ===========================================================================
static __global__ void __launch_bounds__(kTileThreads)
k_update(DTopo tp, DGeom<double> g, DTracers<double> tr, double dt, int mode, int tile) {
    extern __shared__ __align__(16) double sm64[];
    __shared__ Tile S;
    const int L1 = tp.L1, nl = tp.nl, n0 = blockIdx.x * tile;
    if (threadIdx.x < 32) {
        const int n = n0 + threadIdx.x;
        const bool ok = threadIdx.x < tile && n < tp.N2;
        S.fill(threadIdx.x, ok ? tp.n_ulev[n] : 1, ok ? tp.n_nlev[n] - tp.n_ulev[n] : 0);
    }
    for (int t = 0; t < tr.ntr; t++) {
        const bool fct = tr.cfg[t].lim != 0;
        double *T = tr.T + t * tr.sN;
        const double *ADv = tr.ADv + t * tr.sNI, *ADh = tr.ADh + t * tr.sE;
        const double *Rp = tr.bmax + t * tr.sN, *Rm = tr.bmin + t * tr.sN;
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            double x = ADv[ixn(nz, n, nl)];
            if (fct) {
                const size_t k = ix1(nz, n, L1);
                const bool in = !neg64(x) || zero64(x);  // x >= 0 (a NaN stays one under any factor)
                double ae = in ? Rp[k] : Rm[k];
                if (i != S.pre[j]) ae = min64(in ? Rm[k - 1] : Rp[k - 1], ae);
                x = ae * x;
            }
            sm64[i] = x;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
            const int j = S.find(i), n = n0 + j, nz = S.top[j] + i - S.pre[j];
            const size_t k = ix1(nz, n, L1), kv = ixn(nz, n, nl);
            const double av = g.areasvol[kv], h = g.hnode[k], hn = g.hnode_new[k], t0 = T[k];
            const double2 ra = g.rav[kv];
            const double f0 = sm64[i], f1 = i + 1 < S.pre[j + 1] ? sm64[i + 1] : ADv[kv + 1];
            double dv = sdiv64((f0 - f1) * dt, av, ra);
            if (fct) dv = (-(t0 * h) + tr.LO[t * tr.sN + k] * hn) + dv;
            double dh = 0.0;
            for (int q = tp.ne_ptr[n]; q < tp.ne_ptr[n + 1]; q++) {
                const int code = tp.ne_idx[q], e = code >= 0 ? code : ~code;
                if (nz < tp.e_lo[e] || nz > tp.e_hi[e]) continue;
                double x = ADh[ix1(nz, e, L1)];
                if (fct) {
                    const bool in = !neg64(x) || zero64(x), own = code >= 0;
                    const size_t m = ix1(nz, own ? tp.e_n2[e] : tp.e_n1[e], L1);
                    // x >= 0: R+ of edges(1,e), R- of edges(2,e); x < 0 the other way round
                    const double rn = in == own ? Rp[k] : Rm[k], rm = in == own ? Rm[m] : Rp[m];
                    x = min64(own ? rn : rm, own ? rm : rn) * x;
                }
                x = sdiv64(x * dt, av, ra);
                dh = dh + (code >= 0 ? x : -x);
            }
            if (mode == 0) {
                tr.dttf_h[t * tr.sN + k] = dh;
                tr.dttf_v[t * tr.sN + k] = dv;
            } else {
                double del = dh + dv;
                // diff_tracers_ale: horizontal, then explicit vertical diffusion
                if (tr.HD) del = hdiff_add(tp, tr.HD + t * tr.sE, del, n, nz, L1, dt, av);
                if (tr.VX && !tr.cfg[t].ivd) del = del + tr.VX[t * tr.sN + k];
                // Redi: diff_ver_part_redi_expl (:623)
                if (tr.RV) del = del + tr.RV[t * tr.sN + k];
                del = del + t0 * (h - hn);
                const double tn = t0 + sdiv64(del, hn, g.rhn[k]);
                T[k] = tn;
                if (nonfinite64(tn)) atomicOr(tr.status, 1u);
            }
        }
    }
}

// ===========================================================================
// diff_ver_part_impl_ale (src/oce_ale_tracer.F90:1071-1430): a tile of columns per block, the
// tracers with implicit vertical diffusion NT at a time
// ===========================================================================
template <int NT>
static __global__ void __launch_bounds__(kVThreads) k_vdiff_tile(VArgs P, DTracers<double> tr, const double *bc,
                                                                 int wsplit) {
    extern __shared__ __align__(16) double sm64[];
    __shared__ VTile S;
    const int n0 = blockIdx.x * P.cols;
    if (threadIdx.x < 32) {
        const int n = n0 + threadIdx.x;
        const bool ok = threadIdx.x < P.cols && n < P.N2;
        S.fill(threadIdx.x, ok ? P.ulev[n] : 1, ok ? P.nlev[n] - P.ulev[n] : 0);
    }
    // the implicit part of a split vertical velocity joins the solve without a limiter (:961)
    for (int w = 0; w <= (wsplit ? 1 : 0); w++) {
        int t = 0;
        while (t < tr.ntr) {
            VTracer q[NT];
            int nt = 0;
#pragma unroll
            for (int k = 0; k < NT; k++) {
                while (t < tr.ntr && !(tr.cfg[t].ivd && (wsplit && !tr.cfg[t].lim) == (w != 0))) t++;
                q[k] = VTracer{nullptr, nullptr};
                if (t < tr.ntr) {
                    q[k] = VTracer{tr.T + t * tr.sN, bc ? bc + (size_t)t * P.N2 : nullptr};
                    nt = k + 1;
                    t++;
                }
            }
            if (!nt) break;
            __syncthreads();
            vdiff_tile<NT>(P, S, n0, sm64, q, nt, w != 0);
        }
    }
}
// shared-memory limits, once per context
template <int NT>
static cudaError_t vdiff_prepare() {
    return cudaFuncSetAttribute(k_vdiff_tile<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVSmemMax);
}
cudaError_t fp64_prepare() {
    cudaError_t e = vdiff_prepare<1>();
    if (e == cudaSuccess) e = vdiff_prepare<2>();
    if (e == cudaSuccess) e = vdiff_prepare<3>();
    if (e == cudaSuccess) e = vdiff_prepare<4>();
    return e;
}

// ===========================================================================
// launches
// ===========================================================================
template <>
void Launch<double>::ab(const DTopo &tp, DTracers<double> &tr, int ab, cudaStream_t s) {
    const size_t n = (size_t)tp.L1 * tp.N2;
    k_ab<<<(int)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, s>>>(tr, n, ab);
}
template <>
void Launch<double>::trxy(const DTopo &tp, const DGeom<double> &g, DTracers<double> &tr, cudaStream_t s) {
    const int t = tile_size(tp.T2, 0);
    k_trxy<<<(tp.T2 + t - 1) / t, kTileThreads, 0, s>>>(tp, g, tr, t);
}
template <>
void Launch<double>::edge_flux(const DTopo &tp, const DGeom<double> &g, const DForcing<double> &f, DTracers<double> &tr,
                               int any_ho, cudaStream_t s) {
    const size_t b = sizeof(int) * tp.L1;
    const int t = tile_size(tp.E2, b);
    k_edge_flux<<<(tp.E2 + t - 1) / t, kTileThreads, t * b, s>>>(tp, g, f, tr, t, any_ho);
}
template <>
void Launch<double>::node_lo(const DTopo &tp, const DGeom<double> &g, const DForcing<double> &f, DTracers<double> &tr,
                             double dt, int, cudaStream_t s) {
    const size_t b = 2 * sizeof(double) * tp.L1;
    const int t = tile_size(tp.N2, b);
    k_node_lo<<<(tp.N2 + t - 1) / t, kTileThreads, t * b, s>>>(tp, g, f, tr, dt, t);
}
template <>
void Launch<double>::bounds_rpm(const DTopo &tp, const DGeom<double> &g, DTracers<double> &tr, double dt,
                                cudaStream_t s) {
    const size_t b = 2 * sizeof(double) * tp.L1;
    const int t = tile_size(tp.N2, b);
    k_bounds_rpm<<<(tp.N2 + t - 1) / t, kTileThreads, t * b, s>>>(tp, g, tr, dt, t);
}
template <>
void Launch<double>::update(const DTopo &tp, const DGeom<double> &g, DTracers<double> &tr, double dt, int, int mode,
                            cudaStream_t s) {
    const size_t b = sizeof(double) * tp.L1;
    const int t = tile_size(tp.N2, b);
    k_update<<<(tp.N2 + t - 1) / t, kTileThreads, t * b, s>>>(tp, g, tr, dt, mode, t);
}
template <>
void Launch<double>::vdiff(const DTopo &tp, const DGeom<double> &g, const DForcing<double> &f, DTracers<double> &tr,
                           double dt, double *scratch, cudaStream_t s) {
    if (vtile_smem(tp.L1, kVCols, 1) > kVSmemMax || vdiff_by_column(tp.N2, tp.L1)) {
        k_vdiff<double><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, tr, dt, scratch);
        return;
    }
    // as many tracers at a time as share the coefficients with two blocks resident per SM
    int nt = std::min(tr.ntr, 4);
    while (nt > 1 && vtile_smem(tp.L1, kVCols, nt) > kVSmemMax / 2) nt--;
    const int cols = vtile_cols(tp.N2, nt, tp.L1);
    const VArgs P{tp.N2, tp.nl,      cols, tp.n_nlev, tp.n_ulev, g.zbar_n_bot, g.hnode_new,
                  g.area, g.areasvol, f.Kv, f.wi,      g.rav,     dt};
    const int nb = (tp.N2 + cols - 1) / cols;
    const size_t sm = vtile_smem(tp.L1, cols, nt);
    if (nt == 1) k_vdiff_tile<1><<<nb, kVThreads, sm, s>>>(P, tr, f.bc, f.wsplit);
    else if (nt == 2) k_vdiff_tile<2><<<nb, kVThreads, sm, s>>>(P, tr, f.bc, f.wsplit);
    else if (nt == 3) k_vdiff_tile<3><<<nb, kVThreads, sm, s>>>(P, tr, f.bc, f.wsplit);
    else k_vdiff_tile<4><<<nb, kVThreads, sm, s>>>(P, tr, f.bc, f.wsplit);
}
// reciprocals of a divisor array (DGeom::rav, rhn)
static __global__ void k_recip(const double *y, double2 *out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = recip64(y[i]);
}
void recip_table(const double *y, double2 *out, size_t n, cudaStream_t s) {
    k_recip<<<(int)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, s>>>(y, out, n);
}

}  // namespace fesom
