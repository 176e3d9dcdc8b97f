// fp64_stages.cuh -- the advection stages of the FP64 form.
//
// All of these kernels are bound by the FP64 pipe (84-87 % busy before and after; DRAM under
// 10 %), so they are built to issue as few FP64 warp instructions as possible for the
// reference's bits:
//   * comparisons, maxima, absolute values and selections run on integers (fp64_arith.cuh);
//   * v + |v| and v - |v| are 2v or 0: an upwind sum T1 (v + |v|) + T2 (v - |v|) is one product of
//     the upwind value, and 0.5 * (T * 2v) is T * v; both only while the operand that drops out
//     is finite (0 * inf is a NaN the reference would produce), else the full expression;
//   * divisions by shared or constant divisors take 3 or 4 instructions instead of 8;
//   * the wet levels of a tile of entities are dealt to the threads one after another (Tile), so
//     every warp but a tile's last is full.  A warp per column left 27 to 50 % of the lanes idle
//     (47 layers are 32 + 15 lanes), and an FP64 instruction costs its 16 cycles however many
//     lanes take part.
#pragma once
#include "fesom_internal.h"
#include "fp64_arith.cuh"
#include "tracer_kernels.cuh"

namespace fesom {

constexpr int kTileThreads = 128;
constexpr int kTileMax = 8;  // entities per tile

// the wet levels of a tile's entities as items 0 .. total-1: entity j holds the items
// pre[j] .. pre[j+1]-1, levels top[j], top[j] + 1, ...
struct Tile {
    int total;
    int pre[kTileMax + 1], top[kTileMax];
    // one warp, lane j < kTileMax with the level count of entity j (0 past the tile's end)
    __device__ __forceinline__ void fill(int lane, int first_level, int levels) {
        int s = lane < kTileMax ? levels : 0;
#pragma unroll
        for (int o = 1; o < kTileMax; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        if (lane < kTileMax) {
            pre[lane + 1] = s;
            top[lane] = first_level;
            if (lane == 0) pre[0] = 0;
            if (lane == kTileMax - 1) total = s;
        }
    }
    __device__ __forceinline__ int find(int i) const {
        int j = i >= pre[4] ? 4 : 0;
        j += i >= pre[j + 2] ? 2 : 0;
        return j + (i >= pre[j + 1] ? 1 : 0);
    }
};

// entities per tile: 8, or 4 where 8 would leave less than eight blocks per SM (a mesh of 2.9k
// nodes: 4.8 blocks per SM instead of 2.4, so the SMs finish together); fewer where the tile's
// shared memory (`bytes` per entity) would pass 48 KB
static inline int tile_size(int n, size_t bytes) {
    int t = n >= 152 * 8 * kTileMax ? kTileMax : 4;
    while (t > 1 && t * bytes > 46 * 1024) t >>= 1;
    return t;
}

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
// shared by the tracers, against about 70 per tracer.  A step of the sphere of 7 subdivisions
// with 48 levels and 2 tracers: 17.5 ms with k_ab, k_trxy and k_edge_flux at 5.5 ms before, 14.1
// ms with the three at 2.1 ms.
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

static __global__ void __launch_bounds__(kTileThreads)
k_edge_flux(DTopo tp, DGeom<double> g, DForcing<double> f, DTracers<double> tr, int tile) {
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
    __syncthreads();
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j];
        const EdgeData &E = Ed[j];
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
        const bool tri = nz >= E.gmin && nz <= E.gmax;
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
                    if (c.ph == 0.0 && !vbad && !nonfinite64(t1) && !nonfinite64(t2) &&
                        !grad_bad(tp, txy, tri, neg ? E.up : E.dn, neg ? E.n1 : E.n2, nz)) {
                        double2 gr;
                        if (tri) gr = reinterpret_cast<const double2 *>(txy)[ix1(nz, neg ? E.dn : E.up, L1)];
                        else node_mean_grad(tp, g, txy, neg ? E.n2 : E.n1, nz, gr.x, gr.y);
                        // 2 (t2 - t1) is exact: one rounding in the fused sum, as in the reference's
                        double q = div_3x2k<6>(__fma_rn(2.0, t2 - t1, E.ca * gr.x) + E.cb * gr.y);
                        if (c.hor == 0 && (neg ? E.nbl2 : E.nbl1) < nz) q = q * 0.0;
                        const double Tm = (neg ? t2 : t1) + (neg ? -q : q);
                        ad = -(Tm * vf) - flo;
                    } else {
                        ad = edge_ho_full(tp, g, txy, c, tri, E.up, E.dn, E.n1, E.n2, nz, t1, t2, vf, E.ca, E.cb,
                                          E.nbl1 >= nz, E.nbl2 >= nz, flo);
                    }
                }
            }
            if (c.lim) tr.FLO[t * tr.sE + ke] = flo;
            tr.ADh[t * tr.sE + ke] = ad;
        }
    }
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
                               int, cudaStream_t s) {
    const int t = tile_size(tp.E2, 0);
    k_edge_flux<<<(tp.E2 + t - 1) / t, kTileThreads, 0, s>>>(tp, g, f, tr, t);
}

}  // namespace fesom
