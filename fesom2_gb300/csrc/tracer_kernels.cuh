// tracer_kernels.cuh -- sm_103a kernels of the FESOM2 tracer-transport step, FP64 form.
//
// Instantiated with R = double (kernels_fp64.cu, built with --fmad=false): the
// reference's FP64 arithmetic in the reference's evaluation order, so the results
// match the serial Fortran loops bit for bit.  The FP32 form has its own kernels
// (kernels_fp32_batched.cu) and takes only the content sums from here
// (kernels_fp32.cu).  The advection stages and the column solve of the step
// are in fp64_stages.cuh and vdiff_column.cuh; here are the vertical PPM flux, the
// diffusion and Redi kernels, the split velocity's solve and the column solve of
// columns too deep for shared memory.
//
// Mapping: edge and node kernels run one warp per entity with the lanes over
// the levels of the column (the reference's arrays are level-contiguous, so
// every lane load is coalesced); solves run one thread per column.  Node sums
// are gathers over the node's ascending edge list instead of the reference's
// edge scatters: the terms are added in the same order, without atomics, so
// sums are deterministic.
#pragma once
#include <cuda_runtime.h>

#include "fesom_internal.h"
#include "vdiff_column.cuh"

namespace fesom {

constexpr int kWarpsPerBlock = 4;
constexpr int kThreads = 32 * kWarpsPerBlock;

template <typename R> __device__ __forceinline__ R rmax(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R rmin(R a, R b) { return a < b ? a : b; }
template <typename R> __device__ __forceinline__ R rabs(R a) { return fabs(a); }
template <> __device__ __forceinline__ float rabs<float>(float a) { return fabsf(a); }

__device__ __forceinline__ size_t ix1(int nz, int n, int L1) { return (size_t)n * L1 + (nz - 1); }
__device__ __forceinline__ size_t ixn(int nz, int n, int nl) { return (size_t)n * nl + (nz - 1); }

// ===========================================================================
// tracer_gradient_z (src/oce_tracer_mod.F90:192-232): warp per node, lanes over levels;
// tr_z(nz) = (T(nz-1) - T(nz)) / (0.5 (hnode(nz-1) + hnode(nz))) inside the column, zero at
// the first and last interface; the interfaces outside [nzmin, nzmax] are left as they are
// ===========================================================================
template <typename R>
__global__ void __launch_bounds__(kThreads) k_trz(DTopo tp, DGeom<R> g, const R *__restrict__ T, R *__restrict__ trz) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L1 = tp.L1, nl = tp.nl;
    for (int n = blockIdx.x * kWarpsPerBlock + warp; n < tp.N2; n += gridDim.x * kWarpsPerBlock) {
        const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
        for (int nz = nzmin + 1 + lane; nz <= nzmax - 1; nz += 32) {
            const R dz = R(0.5) * (g.hnode[ix1(nz - 1, n, L1)] + g.hnode[ix1(nz, n, L1)]);
            trz[ixn(nz, n, nl)] = (T[ix1(nz - 1, n, L1)] - T[ix1(nz, n, L1)]) / dz;
        }
        if (lane == 0) {
            trz[ixn(nzmin, n, nl)] = R(0);
            trz[ixn(nzmax, n, nl)] = R(0);
        }
    }
}

// area-weighted mean of tr_xy over the node's elements wet at level nz
// (fill_up_dn_grad, src/oce_muscl_adv.F90:388-405)
template <typename R>
__device__ __forceinline__ void node_mean_grad(const DTopo &tp, const DGeom<R> &g, const R *trxy, int node, int nz,
                                               R &gx, R &gy) {
    const int L1 = tp.L1;
    R tvol = R(0), tx = R(0), ty = R(0);
    for (int k = tp.nie_ptr[node]; k < tp.nie_ptr[node + 1]; k++) {
        const int el = tp.nie_idx[k];
        if (tp.t_nlev[el] - 1 < nz || nz < tp.t_ulev[el]) continue;
        const R ea = g.elem_area[el];
        tvol = tvol + ea;
        tx = tx + trxy[2 * ix1(nz, el, L1)] * ea;
        ty = ty + trxy[2 * ix1(nz, el, L1) + 1] * ea;
    }
    gx = tx / tvol;
    gy = ty / tvol;
}

template <typename R>
__device__ __forceinline__ R min3r(R a, R b, R c) { return rmin(rmin(a, b), c); }
// Fortran sign(1, b)
template <typename R>
__device__ __forceinline__ R sign1(R b) { return signbit(b) ? R(-1.0) : R(1.0); }

// interface value tv(k) of adv_tra_vert_ppm (src/oce_adv_tra_ver.F90:488-562) on a column:
// Tc, hc 1-based views of the layer values and the new thicknesses
template <typename R>
__device__ R ppm_tv(const R *Tc, const R *hc, int k, int nzmin, int nzmax) {
    if (k == nzmax) return Tc[nzmax - 1];
    if (k == nzmin) return Tc[nzmin];
    if (k == nzmax - 1) return R(0.5) * (Tc[nzmax - 2] + Tc[nzmax - 1]);
    if (k == nzmin + 1) return R(0.5) * (Tc[nzmin] + Tc[nzmin + 1]);
    const int nz = k - 1;
    const R dzjm1 = hc[nz - 1], dzj = hc[nz], dzjp1 = hc[nz + 1], dzjp2 = hc[nz + 2];
    const R tm1 = Tc[nz - 1], t0 = Tc[nz], tp1 = Tc[nz + 1], tp2 = Tc[nz + 2];
    R deltaj = dzj / (dzjm1 + dzj + dzjp1) *
               ((R(2.0) * dzjm1 + dzj) / (dzjp1 + dzj) * (tp1 - t0) + (dzj + R(2.0) * dzjp1) / (dzjm1 + dzj) * (t0 - tm1));
    R deltajp1 = dzjp1 / (dzj + dzjp1 + dzjp2) *
                 ((R(2.0) * dzj + dzjp1) / (dzjp2 + dzjp1) * (tp2 - tp1) +
                  (dzjp1 + R(2.0) * dzjp2) / (dzj + dzjp1) * (tp1 - t0));
    if ((tp1 - t0) * (t0 - tm1) > R(0.0))
        deltaj = min3r(rabs(deltaj), R(2.0) * rabs(tp1 - t0), R(2.0) * rabs(t0 - tm1)) * sign1(deltaj);
    else
        deltaj = R(0.0);
    if ((tp2 - tp1) * (tp1 - t0) > R(0.0))
        deltajp1 = min3r(rabs(deltajp1), R(2.0) * rabs(tp2 - tp1), R(2.0) * rabs(tp1 - t0)) * sign1(deltajp1);
    else
        deltajp1 = R(0.0);
    return t0 + dzj / (dzj + dzjp1) * (tp1 - t0) +
           R(1.0) / (dzjm1 + dzj + dzjp1 + dzjp2) *
               ((R(2.0) * dzjp1 * dzj) / (dzj + dzjp1) *
                    ((dzjm1 + dzj) / (R(2.0) * dzj + dzjp1) - (dzjp2 + dzjp1) / (R(2.0) * dzjp1 + dzj)) * (tp1 - t0) -
                dzj * (dzjm1 + dzj) / (R(2.0) * dzj + dzjp1) * deltajp1 +
                dzjp1 * (dzjp1 + dzjp2) / (dzj + R(2.0) * dzjp1) * deltaj);
}

// the PPM flux of interface nz (:564-620): the monotonised parabola of the upwind layer (nz
// when w(nz) > 0, nz-1 when w(nz) < 0) integrated over the part swept in dt (old thickness);
// the surface takes -tv w area, the bottom 0; minus the input flux
template <typename R>
__device__ R ver_ppm_flux(const R *T, const R *W, const R *area, const R *hn, const R *ho, R dt, int nz, int n,
                          int nzmin, int nzmax, int L1, int nl, R fin) {
    const R *Tc = T + (size_t)n * L1 - 1, *hc = hn + (size_t)n * L1 - 1, *oc = ho + (size_t)n * L1 - 1;
    const R *Wc = W + (size_t)n * nl - 1, *ac = area + (size_t)n * nl - 1;
    if (nz == nzmin) return -(ppm_tv(Tc, hc, nzmin, nzmin, nzmax) * Wc[nzmin] * ac[nzmin]) - fin;
    if (nz == nzmax) return R(0.0) - fin;
    const R w = Wc[nz];
    if (!(w > R(0.0)) && !(w < R(0.0))) return R(0.0) - fin;
    const bool top = w > R(0.0);
    const int j = top ? nz : nz - 1;  // the upwind layer
    R aL = ppm_tv(Tc, hc, j, nzmin, nzmax), aR = ppm_tv(Tc, hc, j + 1, nzmin, nzmax);
    const R t = Tc[j];
    if ((aR - t) * (t - aL) <= R(0.0)) {
        aL = t;
        aR = t;
    }
    if ((aR - aL) * (t - R(0.5) * (aL + aR)) > (aR - aL) * (aR - aL) / R(6.0)) aL = R(3.0) * t - R(2.0) * aR;
    if ((aR - aL) * (t - R(0.5) * (aR + aL)) < -((aR - aL) * (aR - aL) / R(6.0))) aR = R(3.0) * t - R(2.0) * aL;
    const R dzj = oc[j];
    const R aj = R(6.0) * (t - R(0.5) * (aL + aR));
    R v;
    if (top) {
        const R x = rmin(w * dt / dzj, R(1.0));
        v = -aL - R(0.5) * x * (aR - aL + (R(1.0) - R(2.0) / R(3.0) * x) * aj);
    } else {
        const R x = rmin(-(w * dt / dzj), R(1.0));
        v = -aR + R(0.5) * x * (aR - aL - (R(1.0) - R(2.0) / R(3.0) * x) * aj);
    }
    return v * ac[nz] * w - fin;
}

// ===========================================================================
// diff_ver_part_impl_ale (src/oce_ale_tracer.F90:1071-1430): one thread per
// column, arithmetic in A (double for both forms).  Scratch holds Z_n, cp and
// tp level-major ([level][node]) so that a warp's accesses are coalesced.
// ===========================================================================
// ---------------------------------------------------------------------------
// diff_part_hor_redi (oce_ale_tracer.F90:1526-1689): per edge-layer the flux c of the segment
// (A/D: element 1, B/E: element 2, C: both), Kh = (Ki(n1) + Ki(n2)) / 2, F = Kh grad T, with
// Redi F = Kh (grad T + S_xy Tz): Tz = mean over the layer of the vertical gradient at each
// edge node, S_xy Tz = (Tz(n1) S(n1) + Tz(n2) S(n2)) / 2 (:1583-1595)
// ---------------------------------------------------------------------------
// tracer_gradient_z (oce_tracer_mod.F90:192-232) of T at interface nz of node n: 0 at the
// column's top and bottom interfaces
template <typename R>
__device__ __forceinline__ R trz_node(const DTopo &tp, const DGeom<R> &g, const R *T, int n, int nz) {
    const int L1 = tp.L1;
    if (nz <= tp.n_ulev[n] || nz >= tp.n_nlev[n]) return R(0);
    const R dz = R(0.5) * (g.hnode[ix1(nz - 1, n, L1)] + g.hnode[ix1(nz, n, L1)]);
    return (T[ix1(nz - 1, n, L1)] - T[ix1(nz, n, L1)]) / dz;
}

template <typename R>
__device__ __forceinline__ void hdiff_flux(const DTopo &tp, const DGeom<R> &g, const DTracers<R> &tr, const R *T,
                                          int n1, int n2, int nz, R Kh, R Tx, R Ty, R &Fx, R &Fy) {
    if (!tr.slope) {
        Fx = Kh * Tx;
        Fy = Kh * Ty;
        return;
    }
    const int L1 = tp.L1;
    const R tz1 = R(0.5) * (trz_node(tp, g, T, n1, nz) + trz_node(tp, g, T, n1, nz + 1));
    const R tz2 = R(0.5) * (trz_node(tp, g, T, n2, nz) + trz_node(tp, g, T, n2, nz + 1));
    const R *s1 = tr.slope + 3 * ix1(nz, n1, L1), *s2 = tr.slope + 3 * ix1(nz, n2, L1);
    const R sx = (tz1 * s1[0] + tz2 * s2[0]) / R(2.0);
    const R sy = (tz1 * s1[1] + tz2 * s2[1]) / R(2.0);
    Fx = Kh * (Tx + sx);
    Fy = Kh * (Ty + sy);
}

template <typename R>
__global__ void __launch_bounds__(kThreads) k_hdiff(DTopo tp, DGeom<R> g, DTracers<R> tr) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L1 = tp.L1;
    for (int e = blockIdx.x * kWarpsPerBlock + warp; e < tp.E2; e += gridDim.x * kWarpsPerBlock) {
        const int el1 = tp.e_t1[e], el2 = tp.e_t2[e], n1 = tp.e_n1[e], n2 = tp.e_n2[e];
        const int nl1 = tp.t_nlev[el1] - 1, ul1 = tp.t_ulev[el1];
        int nl2 = 0, ul2 = 0;
        const R dX1 = g.ecd[4 * (size_t)e], dY1 = g.ecd[4 * (size_t)e + 1];
        R dX2 = R(0), dY2 = R(0);
        if (el2 >= 0) {
            nl2 = tp.t_nlev[el2] - 1;
            ul2 = tp.t_ulev[el2];
            dX2 = g.ecd[4 * (size_t)e + 2];
            dY2 = g.ecd[4 * (size_t)e + 3];
        }
        const int nl12 = nl1 < nl2 ? nl1 : nl2, ul12 = ul1 > ul2 ? ul1 : ul2;
        for (int nz = tp.e_lo[e] + lane; nz <= tp.e_hi[e]; nz += 32) {
            int seg = 0;
            if (nz >= ul1 && nz <= ul12 - 1) seg = 1;                    // (A)
            else if (ul2 > 0 && nz >= ul2 && nz <= ul12 - 1) seg = 2;    // (B)
            else if (nz >= ul12 && nz <= nl12) seg = 3;                 // (C)
            else if (nz >= nl12 + 1 && nz <= nl1) seg = 1;              // (D)
            else if (nz >= nl12 + 1 && nz <= nl2) seg = 2;              // (E)
            for (int t = 0; t < tr.ntr; t++) {
                const R *Ki = tr.Ki;
                const R *xy = tr.trxy + t * tr.sT;
                const R *T = tr.T + t * tr.sN;
                const R Kh = (Ki[ix1(nz, n1, L1)] + Ki[ix1(nz, n2, L1)]) / R(2.0);
                R c = R(0), Fx, Fy;
                if (seg == 1) {
                    const R dz = g.helem[ix1(nz, el1, L1)];
                    hdiff_flux(tp, g, tr, T, n1, n2, nz, Kh, xy[2 * ix1(nz, el1, L1)], xy[2 * ix1(nz, el1, L1) + 1], Fx,
                               Fy);
                    c = (-dX1 * Fy + dY1 * Fx) * dz;
                } else if (seg == 2) {
                    const R dz = g.helem[ix1(nz, el2, L1)];
                    hdiff_flux(tp, g, tr, T, n1, n2, nz, Kh, xy[2 * ix1(nz, el2, L1)], xy[2 * ix1(nz, el2, L1) + 1], Fx,
                               Fy);
                    c = (dX2 * Fy - dY2 * Fx) * dz;
                } else if (seg == 3) {
                    const R dz = (g.helem[ix1(nz, el1, L1)] + g.helem[ix1(nz, el2, L1)]) / R(2.0);
                    const R Tx = R(0.5) * (xy[2 * ix1(nz, el1, L1)] + xy[2 * ix1(nz, el2, L1)]);
                    const R Ty = R(0.5) * (xy[2 * ix1(nz, el1, L1) + 1] + xy[2 * ix1(nz, el2, L1) + 1]);
                    hdiff_flux(tp, g, tr, T, n1, n2, nz, Kh, Tx, Ty, Fx, Fy);
                    c = ((dX2 - dX1) * Fy - (dY2 - dY1) * Fx) * dz;
                }
                tr.HD[t * tr.sE + ix1(nz, e, L1)] = c;
            }
        }
    }
}

// del(n) += rhs * dt / areasvol(n) for each edge of n in ascending edge order; rhs = 0 + c at
// edges(1,e), 0 - c at edges(2,e) (oce_ale_tracer.F90:1677-1684)
template <typename R>
__device__ __forceinline__ R hdiff_add(const DTopo &tp, const R *HD, R del, int n, int nz, int L1, R dt, R av) {
    for (int k = tp.ne_ptr[n]; k < tp.ne_ptr[n + 1]; k++) {
        const int code = tp.ne_idx[k];
        const int e = code >= 0 ? code : ~code;
        if (nz < tp.e_lo[e] || nz > tp.e_hi[e]) continue;
        const R c = HD[ix1(nz, e, L1)];
        const R rhs = code >= 0 ? R(0) + c : R(0) - c;
        del = del + rhs * dt / av;
    }
    return del;
}

template <typename R>
__global__ void __launch_bounds__(kThreads) k_hdiff_gather(DTopo tp, DGeom<R> g, DTracers<R> tr, R dt, R *del) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L1 = tp.L1, nl = tp.nl;
    for (int n = blockIdx.x * kWarpsPerBlock + warp; n < tp.N2; n += gridDim.x * kWarpsPerBlock) {
        const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
        for (int t = 0; t < tr.ntr; t++)
            for (int nz = nzmin + lane; nz <= nzmax - 1; nz += 32) {
                const size_t i = ix1(nz, n, L1);
                del[t * tr.sN + i] =
                    hdiff_add(tp, tr.HD + t * tr.sE, del[t * tr.sN + i], n, nz, L1, dt, g.areasvol[ixn(nz, n, nl)]);
            }
    }
}

// ---------------------------------------------------------------------------
// diff_ver_part_expl_ale (oce_ale_tracer.F90:841-902): vd(ul) = surface flux (f.bc),
// vd(nz) = Kv (T(nz-1) - T(nz)) / (Z(nz-1) - Z(nz)) area; increment of layer nz
// (vd(nz) - vd(nz+1)) / (zbar(nz) - zbar(nz+1)) dt / areasvol, at the bottom layer
// (vd(nl1) / (zbar(nl1) - zbar(nl1+1))) dt / areasvol
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ R vexpl_vd(const DTopo &tp, const DGeom<R> &g, const R *Kv, const R *T, R fsurf, int n,
                                      int nz, int ul1, int nl1, int L1, int nl) {
    if (nz == ul1) return fsurf;
    if (nz > nl1) return R(0);
    const R zinv1 = R(1.0) / (g.Z3[ix1(nz - 1, n, L1)] - g.Z3[ix1(nz, n, L1)]);
    return Kv[ixn(nz, n, nl)] * (T[ix1(nz - 1, n, L1)] - T[ix1(nz, n, L1)]) * zinv1 * g.area[ixn(nz, n, nl)];
}

template <typename R>
__global__ void __launch_bounds__(kThreads) k_vexpl(DTopo tp, DGeom<R> g, DForcing<R> f, DTracers<R> tr, R dt,
                                                    R *out, int all, int add) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L1 = tp.L1, nl = tp.nl;
    for (int n = blockIdx.x * kWarpsPerBlock + warp; n < tp.N2; n += gridDim.x * kWarpsPerBlock) {
        const int nl1 = tp.n_nlev[n] - 1, ul1 = tp.n_ulev[n];
        for (int t = 0; t < tr.ntr; t++) {
            if (!all && tr.cfg[t].ivd) continue;
            const R *T = tr.T + t * tr.sN;
            const R fs = f.bc ? f.bc[(size_t)t * tp.N2 + n] : R(0);
            for (int nz = ul1 + lane; nz <= nl1; nz += 32) {
                const size_t i = ix1(nz, n, L1);
                const R av = g.areasvol[ixn(nz, n, nl)];
                const R v0 = vexpl_vd(tp, g, f.Kv, T, fs, n, nz, ul1, nl1, L1, nl);
                R inc;
                if (nz <= nl1 - 1) {
                    const R v1 = vexpl_vd(tp, g, f.Kv, T, fs, n, nz + 1, ul1, nl1, L1, nl);
                    inc = (v0 - v1) / (g.zbar3[ixn(nz, n, nl)] - g.zbar3[ixn(nz + 1, n, nl)]) * dt / av;
                } else {
                    inc = (v0 / (g.zbar3[ixn(nz, n, nl)] - g.zbar3[ixn(nz + 1, n, nl)])) * dt / av;
                }
                R *o = out + t * tr.sN;
                o[i] = add ? o[i] + inc : inc;
            }
        }
    }
}

// ===========================================================================
// adv_tra_vert_impl (src/oce_adv_tra_ver.F90:90-240) on the LO values of the FCT tracers:
// implicit upwind advection by w_i, one thread per column, arithmetic in A (double); scratch
// holds cp and tp level-major
// ===========================================================================
template <typename R>
__global__ void __launch_bounds__(128) k_lo_impl(DTopo tp, DGeom<R> g, DForcing<R> f, DTracers<R> tr, double dt,
                                                 double *scratch) {
    typedef double A;
    const int L1 = tp.L1, nl = tp.nl;
    const size_t N2 = tp.N2;
    A *cps = scratch, *tps = scratch + (size_t)(L1 + 1) * N2;
#define CP(k) cps[(size_t)(k) * N2 + n]
#define TP(k) tps[(size_t)(k) * N2 + n]
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < tp.N2; n += gridDim.x * blockDim.x) {
        const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
        const R *hn = g.hnode_new + (size_t)n * L1 - 1;
        const R *ar = g.area + (size_t)n * nl - 1;
        const R *av = g.areasvol + (size_t)n * nl - 1;
        const R *wi = f.wi + (size_t)n * nl - 1;
        for (int t = 0; t < tr.ntr; t++) {
            if (!tr.cfg[t].lim) continue;
            R *Tc = tr.LO + t * tr.sN + (size_t)n * L1 - 1;
            const A zinv = 1.0 * dt;
            int nz = nzmin;
            A v = zinv * (A)ar[nz] / (A)av[nz];
            A b = (A)hn[nz] + (A)wi[nz] * v;
            v = zinv * (A)ar[nz + 1] / (A)av[nz];
            b = b - fmin(0.0, (A)wi[nz + 1]) * v;
            A c = -(fmax(0.0, (A)wi[nz + 1]) * v);
            A T0 = (A)Tc[nz], Tp1 = (A)Tc[nz + 1], Tm;
            A rhs = -((b - (A)hn[nz]) * T0) - c * Tp1;
            A cp = c / b, tpv = rhs / b;
            CP(nz) = cp;
            TP(nz) = tpv;
            for (nz = nzmin + 1; nz <= nzmax - 2; nz++) {
                v = zinv * (A)ar[nz] / (A)av[nz];
                const A a = fmin(0.0, (A)wi[nz]) * v;
                b = (A)hn[nz] + fmax(0.0, (A)wi[nz]) * v;
                v = zinv * (A)ar[nz + 1] / (A)av[nz];
                b = b - fmin(0.0, (A)wi[nz + 1]) * v;
                c = -(fmax(0.0, (A)wi[nz + 1]) * v);
                Tm = T0;
                T0 = Tp1;
                Tp1 = (A)Tc[nz + 1];
                rhs = -(a * Tm) - (b - (A)hn[nz]) * T0 - c * Tp1;
                const A m = b - cp * a;
                cp = c / m;
                tpv = (rhs - tpv * a) / m;
                CP(nz) = cp;
                TP(nz) = tpv;
            }
            nz = nzmax - 1;
            {
                v = zinv * (A)ar[nz] / (A)av[nz];
                const A a = fmin(0.0, (A)wi[nz]) * v;
                b = (A)hn[nz] + fmax(0.0, (A)wi[nz]) * v;
                Tm = T0;
                T0 = Tp1;
                rhs = -(a * Tm) - (b - (A)hn[nz]) * T0;
                const A m = b - cp * a;
                tpv = (rhs - tpv * a) / m;
            }
            A trv = tpv;
            Tc[nzmax - 1] = (R)((A)Tc[nzmax - 1] + trv);
            for (nz = nzmax - 2; nz >= nzmin; nz--) {
                trv = TP(nz) - CP(nz) * trv;
                Tc[nz] = (R)((A)Tc[nz] + trv);
            }
        }
    }
#undef CP
#undef TP
}

template <typename R>
__global__ void __launch_bounds__(128) k_vdiff(DTopo tp, DGeom<R> g, DForcing<R> f, DTracers<R> tr, double dt,
                                               double *scratch) {
    const int L1 = tp.L1, nl = tp.nl;
    const size_t N2 = tp.N2;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < tp.N2; n += gridDim.x * blockDim.x) {
        const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
        const R *hn = g.hnode_new + (size_t)n * L1 - 1;  // hn[nz], 1-based
        const R *ar = g.area + (size_t)n * nl - 1;
        const R *av = g.areasvol + (size_t)n * nl - 1;
        const R *kv = f.Kv + (size_t)n * nl - 1;
        const R *wi = f.wi + (size_t)n * nl - 1;
        const ColScratch cs{scratch + n, scratch + (size_t)(L1 + 1) * N2 + n, scratch + 2 * (size_t)(L1 + 1) * N2 + n,
                            N2};
        vdiff_col_z<R>(cs, nzmin, nzmax, (double)g.zbar_n_bot[n], hn);
        for (int t = 0; t < tr.ntr; t++) {
            if (!tr.cfg[t].ivd) continue;
            // the implicit part of a split vertical velocity joins the solve without a limiter (:961)
            const bool wimpl = f.wsplit && !tr.cfg[t].lim;
            const double bc = f.bc ? (double)f.bc[(size_t)t * N2 + n] : 0.0;
            vdiff_col_solve<R>(cs, nzmin, nzmax, hn, ar, av, kv, wimpl, wi, bc, dt, tr.T + t * tr.sN + (size_t)n * L1 - 1);
        }
    }
}

// ---------------------------------------------------------------------------
// diff_ver_part_redi_expl (oce_ale_tracer.F90:1439-1518), one thread per column, walking the
// column bottom up: node gradients (sum over the node's elements wet at nz of tr_xy
// elem_area) / 3 / areasvol; depths zbar_n, z_n from hnode and zbar_n_bot; interface flux
// vd(nz) = ((z(nz-1) - zbar(nz)) S.g(nz-1) Ki(nz-1) + (zbar(nz) - z(nz)) S.g(nz) Ki(nz))
// / (z(nz-1) - z(nz)) area(nz); increment (vd(nz) - vd(nz+1)) dt / areasvol into RV
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ R redi_proj(const DTopo &tp, const DGeom<R> &g, const R *xy, const R *slope, int n, int nz) {
    const int L1 = tp.L1;
    R tx = R(0), ty = R(0);
    for (int k = tp.nie_ptr[n]; k < tp.nie_ptr[n + 1]; k++) {
        const int el = tp.nie_idx[k];
        if (nz <= tp.t_nlev[el] - 1 && nz >= tp.t_ulev[el]) {
            tx = tx + xy[2 * ix1(nz, el, L1)] * g.elem_area[el];
            ty = ty + xy[2 * ix1(nz, el, L1) + 1] * g.elem_area[el];
        }
    }
    const R av = g.areasvol[ixn(nz, n, tp.nl)];
    const R gx = tx / R(3.0) / av, gy = ty / R(3.0) / av;
    const R *s = slope + 3 * ix1(nz, n, L1);
    return s[0] * gx + s[1] * gy;
}

template <typename R>
__global__ void __launch_bounds__(128) k_redi_v(DTopo tp, DGeom<R> g, DTracers<R> tr, R dt, int add) {
    const int L1 = tp.L1, nl = tp.nl;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < tp.N2; n += gridDim.x * blockDim.x) {
        const int nl1 = tp.n_nlev[n] - 1, ul1 = tp.n_ulev[n];
        const R *Ki = tr.Ki;
        for (int t = 0; t < tr.ntr; t++) {
            const R *xy = tr.trxy + t * tr.sT;
            R *out = tr.RV + t * tr.sN;
            R zb = g.zbar_n_bot[n];                                  // zbar_n(nz + 1)
            R zc = zb + g.hnode[ix1(nl1, n, L1)] / R(2.0);           // z_n(nz)
            R pc = redi_proj(tp, g, xy, tr.slope, n, nl1);           // S . grad at nz
            R below = R(0);                                          // vd(nz + 1)
            for (int nz = nl1; nz >= ul1; nz--) {
                R vd = R(0);
                if (nz >= ul1 + 1) {
                    const R zbn = zb + g.hnode[ix1(nz, n, L1)];                  // zbar_n(nz)
                    const R zu = zbn + g.hnode[ix1(nz - 1, n, L1)] / R(2.0);     // z_n(nz - 1)
                    const R pu = redi_proj(tp, g, xy, tr.slope, n, nz - 1);
                    R v = (zu - zbn) * pu * Ki[ix1(nz - 1, n, L1)];
                    v = v + (zbn - zc) * pc * Ki[ix1(nz, n, L1)];
                    vd = v / (zu - zc) * g.area[ixn(nz, n, nl)];
                    zb = zbn;
                    zc = zu;
                    pc = pu;
                }
                const R inc = (vd - below) * dt / g.areasvol[ixn(nz, n, nl)];
                out[ix1(nz, n, L1)] = add ? out[ix1(nz, n, L1)] + inc : inc;
                below = vd;
            }
        }
    }
}

// K33 = Kv + Ty of diff_ver_part_impl_ale with Redi (oce_ale_tracer.F90:1099-1204) at the
// interfaces nzmin < nz < nzmax, from zbar_n / Z_n of hnode_new bottom up:
// Ty = (zbar(nz) - Z(nz)) / dZ s3(nz-1)^2 Ki(nz-1) + (Z(nz-1) - zbar(nz)) / dZ s3(nz)^2 Ki(nz),
// dZ = Z(nz-1) - Z(nz) (the Ty1 of the layer above is the same number); Kv elsewhere
template <typename R>
__global__ void __launch_bounds__(128) k_k33(DTopo tp, DGeom<R> g, const R *Kv, const R *Ki, const R *slope, R *K33) {
    const int L1 = tp.L1, nl = tp.nl;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < tp.N2; n += gridDim.x * blockDim.x) {
        const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
        for (int nz = 1; nz <= nl; nz++) K33[ixn(nz, n, nl)] = Kv[ixn(nz, n, nl)];
        R zb = g.zbar_n_bot[n];                                         // zbar_n(nz + 1)
        R Zc = zb + g.hnode_new[ix1(nzmax - 1, n, L1)] / R(2.0);        // Z_n(nz)
        for (int nz = nzmax - 1; nz >= nzmin + 1; nz--) {
            const R zbn = zb + g.hnode_new[ix1(nz, n, L1)];             // zbar_n(nz)
            const R Zu = zbn + g.hnode_new[ix1(nz - 1, n, L1)] / R(2.0);  // Z_n(nz - 1)
            const R zinv = R(1.0) / (Zu - Zc);
            const R sa = slope[3 * ix1(nz - 1, n, L1) + 2], sb = slope[3 * ix1(nz, n, L1) + 2];
            const R Ty = (zbn - Zc) * zinv * (sa * sa) * Ki[ix1(nz - 1, n, L1)] +
                         (Zu - zbn) * zinv * (sb * sb) * Ki[ix1(nz, n, L1)];
            K33[ixn(nz, n, nl)] = Kv[ixn(nz, n, nl)] + Ty;
            zb = zbn;
            Zc = Zu;
        }
    }
}

// ===========================================================================
// Global content sum over wet node-layers of T * hnode_new * areasvol (FP64),
// deterministic: fixed per-block partials, then one ordered pass.
// ===========================================================================
template <typename R>
__global__ void __launch_bounds__(256) k_content_partial(DTopo tp, DGeom<R> g, DTracers<R> tr, double *partials) {
    __shared__ double red[256];
    const int L1 = tp.L1, nl = tp.nl;
    for (int t = 0; t < tr.ntr; t++) {
        const R *T = tr.T + t * tr.sN;
        double s = 0.0;
        for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < tp.N2; n += gridDim.x * blockDim.x) {
            for (int nz = tp.n_ulev[n]; nz <= tp.n_nlev[n] - 1; nz++) {
                const size_t i = ix1(nz, n, L1);
                s += (double)T[i] * (double)g.hnode_new[i] * (double)g.areasvol[ixn(nz, n, nl)];
            }
        }
        red[threadIdx.x] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) partials[(size_t)t * gridDim.x + blockIdx.x] = red[0];
        __syncthreads();
    }
}

static __global__ void k_content_final(const double *partials, int nblk, int ntr, double *out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntr) return;
    double s = 0.0;
    for (int b = 0; b < nblk; b++) s += partials[(size_t)t * nblk + b];
    out[t] = s;
}

// ===========================================================================
// launch wrappers
// ===========================================================================
static inline int grid_for(int nent, int per_block) {
    int b = (nent + per_block - 1) / per_block;
    const int cap = 152 * 64;
    if (b > cap) b = cap;
    return b < 1 ? 1 : b;
}

template <typename R>
void Launch<R>::trz(const DTopo &tp, const DGeom<R> &g, const R *T, R *trz, cudaStream_t s) {
    k_trz<R><<<grid_for(tp.N2, kWarpsPerBlock), kThreads, 0, s>>>(tp, g, T, trz);
}
template <typename R>
void Launch<R>::lo_impl(const DTopo &tp, const DGeom<R> &g, const DForcing<R> &f, DTracers<R> &tr, double dt,
                        double *scratch, cudaStream_t s) {
    k_lo_impl<R><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, tr, dt, scratch);
}
template <typename R>
void Launch<R>::content(const DTopo &tp, const DGeom<R> &g, const DTracers<R> &tr, double *partials, int nblk,
                        double *out, cudaStream_t s) {
    k_content_partial<R><<<nblk, 256, 0, s>>>(tp, g, tr, partials);
    k_content_final<<<(tr.ntr + 63) / 64, 64, 0, s>>>(partials, nblk, tr.ntr, out);
}

template <typename R>
void Launch<R>::hdiff(const DTopo &tp, const DGeom<R> &g, DTracers<R> &tr, cudaStream_t s) {
    k_hdiff<R><<<grid_for(tp.E2, kWarpsPerBlock), kThreads, 0, s>>>(tp, g, tr);
}
template <typename R>
void Launch<R>::hdiff_gather(const DTopo &tp, const DGeom<R> &g, DTracers<R> &tr, double dt, R *del, cudaStream_t s) {
    k_hdiff_gather<R><<<grid_for(tp.N2, kWarpsPerBlock), kThreads, 0, s>>>(tp, g, tr, (R)dt, del);
}
template <typename R>
void Launch<R>::vexpl(const DTopo &tp, const DGeom<R> &g, const DForcing<R> &f, DTracers<R> &tr, double dt, R *out,
                      int all, int add, cudaStream_t s) {
    k_vexpl<R><<<grid_for(tp.N2, kWarpsPerBlock), kThreads, 0, s>>>(tp, g, f, tr, (R)dt, out, all, add);
}
template <typename R>
void Launch<R>::redi_v(const DTopo &tp, const DGeom<R> &g, DTracers<R> &tr, double dt, int add, cudaStream_t s) {
    k_redi_v<R><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, tr, (R)dt, add);
}
template <typename R>
void Launch<R>::k33(const DTopo &tp, const DGeom<R> &g, const R *Kv, const R *Ki, const R *slope, R *K33,
                    cudaStream_t s) {
    k_k33<R><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, Kv, Ki, slope, K33);
}

}  // namespace fesom
