// kernels_fp32_batched.cu -- the FP32 batched form of the tracer step.
//
// All tracers of a launch group in one launch per stage, the whole step in one CUDA graph:
//
//   k32_vflux        edge volume fluxes per edge-layer (oce_adv_tra_hor.F90:159-250
//                    segment rule); shared by every tracer
//   k32_vfactors     factorisation of the implicit vertical-diffusion matrix of every
//                    column (oce_ale_tracer.F90:1088-1204, 1406-1414): the pivots
//                    m = b - cp*a, where thin bottom cells cancel most bits, are formed
//                    in FP32 from their excess over |c|, a recurrence of non-negative
//                    terms; stored as FP32 a, c, 1/m, c/m
//   k32_lo_ad        per node: the LO solution (edge gather of upwind fluxes + upwind
//                    vertical flux with w_e) and the vertical antidiffusive flux
//                    (QR4C / UPW1 / CDIFF on the AB values; PPM in k32_vppm)
//   k32_ho           per edge: the horizontal antidiffusive flux, MUSCL / MFCT / UPW1 on
//                    the AB values minus the upwind LO flux (k32_ho_nodemean: the few
//                    edge-layers whose gradients are node means)
//   k32_bounds       per node: FCT bounds (max/min of LO and T over the node's
//                    neighbours and the adjacent layers) and R+/R- (oce_adv_tra_fct.F90)
//   k32_update       per node: limited fluxes, flux divergence, T* update, written to
//                    the buffer of the oldest time level; then, in shallow meshes, the
//                    same block runs its columns' implicit vertical diffusion (k32_vdiff's solve)
//   k32_vdiff        per node: the implicit vertical diffusion as two warp scans of
//                    affine maps over the column (forward and back substitution with
//                    the factors of k32_vfactors); its own launch in deep meshes or as set
//   k32_vppm, k32_lo_impl, k32_vdiff_w, k32_hdiff, k32_diff
//                    the optional parts: PPM vertical fluxes, the split vertical
//                    velocity, horizontal and explicit vertical diffusion
//
// Tracer groups: the tracers sit in groups of G slots (G = 4, or 2) of one scheme, side by
// side in every (level, entity) entry of a field.  A lane's load of one entry is one 16-byte
// (8-byte) vector load that brings all G tracers, so the address, the wet-level predicate
// and the load of every gather are formed once for G tracers, and G independent chains of
// arithmetic follow each load.  Slots a group does not fill hold zeros and compute zeros.
//
// Every tracer carries the same quantities whatever its limiter: the LO solution and the
// antidiffusive fluxes "high order minus low order" of the edges and interfaces.  Without
// FCT the update adds them unlimited, which is the high-order flux divergence; with FCT it
// scales them by R+/R- first.
//
// Conservation: every horizontal flux a node sums is formed from the edge's own data in the
// edge's direction (edges(1,e) -> edges(2,e)) and added at one end and subtracted at the
// other, so both ends use the same bits (the upwind LO flux is recomputed at each end by the
// same expression; the antidiffusive flux is stored once per edge-layer and its limiter
// factor min(R+, R-) is the same seen from either end); a vertical flux is one value, or the same
// expression, at the two layers it joins.  With hnode = hnode_new the LO solution is T plus the flux
// divergence (no rescaling of T that would round every value of the column).
//
// Mapping: tiles (tile.cuh).  The node stages take blocks of consecutive whole columns, a layer per
// thread, the layers above and below through shared memory; the edge stages take blocks of 4 or 8
// edges whose wet levels are dealt to the threads.  Every warp but a tile's last is full, nothing is
// computed twice, and a layer's neighbour offsets and tracer-independent geometry serve every group.
// Tiles are consecutive in the node (edge) order, which is spatially local.
//
// No atomics on values: each edge flux is written once and every node sum is a gather.  The
// Adams-Bashforth shift is a rotation of the time-level buffers (no copy).
#include <cuda_runtime.h>

#include <algorithm>

#include "fesom_internal.h"
#include "tile.cuh"

namespace fesom {

namespace {

// The FCT clamp of the advected value into its bounds: k32_bounds stores the bounds, k32_update
// clamps into them and raises FESOM_STATUS_FCT_BOUND where the clamp moved a value by more than
// round-off.  The reference has no such clamp; the FP32 limiter keeps the values inside their
// bounds to FP32 round-off without it, and the two bound arrays cost a write and a read of 8
// bytes per tracer-DOF (7.8 ms of the 24-tracer benchmark step), so the default build leaves it
// out; -DFESOM_FCT_CLAMP=1 builds it in.
#ifndef FESOM_FCT_CLAMP
#define FESOM_FCT_CLAMP 0
#endif
constexpr bool kFctClamp = FESOM_FCT_CLAMP != 0;
// packed FP32 pairs (two slots per instruction) in the edge kernel's arithmetic
#ifndef FESOM_PACKED_PAIRS
#define FESOM_PACKED_PAIRS 1
#endif
constexpr int kWB = 8;                // warps (= nodes) per block
constexpr int kTB = 32 * kWB;
constexpr unsigned kFull = 0xffffffffu;

// resident blocks per SM each group kernel is built for (registers: 65536 / (threads * blocks)),
// and the edge slots whose gathers bounds (ub) and update (uu) keep in flight at once: the fastest
// of sweeps over 2 to 6 blocks and 1 to 6 slots on the 640k-node seamount channel (G = 2), the
// sphere of 8 subdivisions with 24 tracers and the one of 7 with 7 tracers (G = 4).  ms per step:
//   ho     G=2: 1.62 (5 blocks) 1.00 (8) 0.94 (9) 1.04 (10) 1.20 (12); G=4: 4.00 (5) 4.02 (6) 4.70 (8)
//   lo     G=2: 1.30 (4) 1.34 (5) 1.40 (6); G=4: 4.30 (2) 3.64 (3) 3.60 (4) 4.34 (5)
//   bounds G=2: 1.15 (5 x 2 slots) 1.21 (4 x 3) 1.30 (4 x 6); G=4: 5.54 (4 x 3) 5.84 (3 x 3) 6.26 (4 x 2)
//   hdiff  G=4, Redi: 0.70 (6 to 8, with ho) 0.68 (9); diff 0.65 (2) 0.47 (3) 0.41 (4)
//   update G=2: 1.70 (5 x 1) 1.76 (5 x 2) 1.98 (4 x 6); G=4: 7.16 (3 x 2) 7.55 (4 x 2) 8.17 (3 x 3)
template <int G>
struct MinB {
    static constexpr int lo = 4;
    static constexpr int ho = G == 4 ? 6 : 9;  // blocks of kTileThreads
    static constexpr int bounds = G == 4 ? 4 : 5, ub = G == 4 ? 3 : 2;
    static constexpr int update = G == 4 ? 3 : 5, uu = G == 4 ? 2 : 1;
    static constexpr int hdiff = 9;  // blocks of kTileThreads
    static constexpr int diff = 4;
};

__device__ __forceinline__ size_t i1(int nz, int n, int L1) { return (size_t)n * L1 + (nz - 1); }

// FP32 quotients of the node stages (geometry factors, limiter ratios): the fast division
// (2 ulp) instead of the correctly rounded one; far inside the FP32 form's 1e-5.  A limited value
// may pass its bounds by the last bits of R+/R- (a build with the FCT clamp holds it inside them)
__device__ __forceinline__ float qdiv(float a, float b) { return __fdividef(a, b); }

}  // namespace

// the value of the lane d below / above in the warp
__device__ __forceinline__ float sh_up(float v, int d) { return __shfl_up_sync(kFull, v, d); }
__device__ __forceinline__ float sh_dn(float v, int d) { return __shfl_down_sync(kFull, v, d); }

// ---------------------------------------------------------------------------
// k32_vflux: volume flux of every edge-layer (shared by all tracers)
// ---------------------------------------------------------------------------
// A tile of edges.  Bound by issue (52 %) and the gathers of two elements: 95 -> 63 us on the sphere of
// 7 subdivisions, 48 levels, against a warp per edge.
struct EdgeV {
    int el1, el2, nl1, nu1, nl2, nu2;
    float dX1, dY1, dX2, dY2;
};

// tile ti of `tile` edges
__device__ __forceinline__ void vflux_tile(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, float *VF,
                                           int ti, int tile, Tile &S, EdgeV *Ed) {
    const int L1 = tp.L1, e0 = ti * tile;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, e = e0 + j;
        const bool in = j < tile && e < tp.E2;
        if (in) {
            EdgeV &E = Ed[j];
            const int el1 = tp.e_t1[e], el2 = tp.e_t2[e];
            E.el1 = el1;
            E.el2 = el2;
            E.nl1 = tp.t_nlev[el1] - 1;
            E.nu1 = tp.t_ulev[el1];
            const float4 d = reinterpret_cast<const float4 *>(g.ecd)[e];
            E.dX1 = d.x;
            E.dY1 = d.y;
            E.nl2 = E.nu2 = 0;
            E.dX2 = E.dY2 = 0.f;
            if (el2 >= 0) {
                E.nl2 = tp.t_nlev[el2] - 1;
                E.nu2 = tp.t_ulev[el2];
                E.dX2 = d.z;
                E.dY2 = d.w;
            }
        }
        S.fill(j, in ? tp.e_lo[e] : 1, in ? tp.e_hi[e] - tp.e_lo[e] + 1 : 0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j];
        const EdgeV &E = Ed[j];
        const int fnl12 = min(E.nl1, E.nl2), fnu12 = max(E.nu1, E.nu2);
        int seg = 0;
        if (nz >= E.nu1 && nz <= fnu12 - 1) seg = 1;
        else if (E.nu2 > 0 && nz >= E.nu2 && nz <= fnu12 - 1) seg = 2;
        else if (nz >= fnu12 && nz <= fnl12) seg = 3;
        else if (nz >= fnl12 + 1 && nz <= E.nl1) seg = 1;
        else if (nz >= fnl12 + 1 && nz <= E.nl2) seg = 2;
        float vf = 0.f;
        if (seg & 1) {
            const size_t k = i1(nz, E.el1, L1);
            const float2 q = reinterpret_cast<const float2 *>(f.uv)[k];
            vf = (-(q.y * E.dX1) + q.x * E.dY1) * g.helem[k];
        }
        if (seg & 2) {
            const size_t k = i1(nz, E.el2, L1);
            const float2 q = reinterpret_cast<const float2 *>(f.uv)[k];
            vf += (q.y * E.dX2 - q.x * E.dY2) * g.helem[k];
        }
        VF[i1(nz, e0 + j, L1)] = vf;
    }
}

__global__ void __launch_bounds__(kTileThreads)
k32_vflux(DTopo tp, DGeom<float> g, DForcing<float> f, float *VF, int tile) {
    __shared__ Tile S;
    __shared__ EdgeV Ed[kTileMax];
    vflux_tile(tp, g, f, VF, blockIdx.x, tile, S, Ed);
}

// ---------------------------------------------------------------------------
// k32_vfactors: factorisation of each column's tridiagonal system
// ---------------------------------------------------------------------------
// a(k) = -Kv(k) dt/(Z_n(k-1)-Z_n(k)) area(k)/areasvol(k), c(k) = -Kv(k+1) dt/(Z_n(k)-Z_n(k+1))
// area(k+1)/areasvol(k), b = -a - c + hnode_new (oce_ale_tracer.F90:1099-1204), with
// Z_n(k)-Z_n(k+1) = (hnode_new(k) + hnode_new(k+1))/2 (the mid-depths of :1088-1096);
// Thomas pivots m(k) = b(k) - cp(k-1) a(k), cp(k) = c(k)/m(k) (:1406-1414).
// With a, c <= 0 and b = |a| + |c| + h, the pivot is m(k) = |c(k)| + d(k) with the excess
// d(k) = h(k) + |a(k)| d(k-1) / (d(k-1) + |c(k-1)|) (d = h at the top layer): the textbook form
// subtracts |a| |c(k-1)| / m(k-1) from |a| + |c| + h, which cancels most bits where a thin cell
// (small h) sits under strong diffusion; every term of the excess form is non-negative, so FP32
// keeps the pivots within a few ulps of the exact ones for any cell thickness.
//
// d(k) is a linear-fractional map of d(k-1): (d, 1) -> M_k (d, 1) projectively, with the
// non-negative M_k = [[h + |a|, h |c(k-1)|], [1, |c(k-1)|]] (the top layer: [[0, h], [0, 1]]).
// A warp takes a column, its lanes over 32-level chunks (coalesced loads and stores, each value
// read once): the lanes' maps are combined by an inclusive warp scan of 2x2 products (the later
// level's map on the left; each product rescaled by a power of two, exactly), applied to the
// vector carried from the chunk above.  Products and sums of non-negative numbers do not cancel,
// so the scan keeps the same few-ulp accuracy as the sequential recurrence.
struct M22 {
    float a, b, c, d;  // [[a, b], [c, d]]
};
__device__ __forceinline__ M22 m22_mul(const M22 &x, const M22 &y) {
    return {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}
// 2^-e with 2^e <= x < 2^(e+1) for a normal positive x
__device__ __forceinline__ float pow2_inv(float x) {
    const int e = ((__float_as_int(x) >> 23) & 0xff) - 127;
    return __int_as_float((127 - e) << 23);
}
__device__ __forceinline__ M22 m22_norm(const M22 &m) {
    const float s = pow2_inv(fmaxf(fmaxf(m.a, m.b), fmaxf(m.c, m.d)));
    return {m.a * s, m.b * s, m.c * s, m.d * s};
}

__device__ __forceinline__ void vfactors_col(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f,
                                             float dtf, const VFactors &vf, int n, int lane) {
    const int L1 = tp.L1, nl = tp.nl;
    const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
    float cx = 1.f, cy = 1.f;       // the excess vector at the last level of the chunk above
    float h_up = 0.f, c_up = 0.f;   // h and c of that level
    for (int nz0 = nzmin; nz0 <= nzmax - 1; nz0 += 32) {
        const int nz = nz0 + lane;
        const bool ok = nz <= nzmax - 1;
        const size_t i = (size_t)n * L1 + nz - 1, iv = (size_t)n * nl + nz - 1;
        float h = 0.f, ar = 0.f, av = 1.f, kv = 0.f;
        if (ok) {
            h = g.hnode_new[i];
            ar = g.area[iv];
            av = g.areasvol[iv];
            kv = f.Kv[iv];
        }
        // the level below (c) from the next lane, the chunk's last lane loads it
        float hn = sh_dn(h, 1), arn = sh_dn(ar, 1), kvn = sh_dn(kv, 1);
        if (lane == 31 && nz + 1 <= nzmax - 1) {
            hn = g.hnode_new[i + 1];
            arn = g.area[iv + 1];
            kvn = f.Kv[iv + 1];
        }
        // the level above (a) from the previous lane, the chunk's first lane from the chunk above
        float hu = sh_up(h, 1);
        if (lane == 0) hu = h_up;
        const float ravz = 1.f / av;
        float a = 0.f, c = 0.f;
        if (ok && nz > nzmin) a = -(kv * (2.f / (hu + h)) * dtf * (ar * ravz));
        if (ok && nz < nzmax - 1) c = -(kvn * (2.f / (h + hn)) * dtf * arn * ravz);
        float cu = sh_up(c, 1);
        if (lane == 0) cu = c_up;
        M22 S;
        if (!ok) S = {1.f, 0.f, 0.f, 1.f};
        else if (nz == nzmin) S = {0.f, h, 0.f, 1.f};
        else S = {h - a, h * -cu, 1.f, -cu};
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const M22 P = {sh_up(S.a, off), sh_up(S.b, off), sh_up(S.c, off), sh_up(S.d, off)};
            if (lane >= off) S = m22_norm(m22_mul(S, P));
        }
        const float v0 = S.a * cx + S.b * cy, v1 = S.c * cx + S.d * cy;
        if (ok) {
            const float m = v0 / v1 - c;
            vf.a[i] = a;
            vf.c[i] = c;
            vf.inv[i] = 1.f / m;
            vf.cp[i] = c / m;
        }
        // past the column's end the maps are identities: lane 31 holds the chunk's last level
        const float w0 = __shfl_sync(kFull, v0, 31), w1 = __shfl_sync(kFull, v1, 31);
        const float sc = pow2_inv(fmaxf(w0, w1));
        cx = w0 * sc;
        cy = w1 * sc;
        h_up = __shfl_sync(kFull, h, 31);
        c_up = __shfl_sync(kFull, c, 31);
    }
}

__global__ void __launch_bounds__(kTB) k32_vfactors(DTopo tp, DGeom<float> g, DForcing<float> f, float dt,
                                                    VFactors vf) {
    for (int n = blockIdx.x * kWB + (threadIdx.x >> 5); n < tp.N2; n += gridDim.x * kWB)
        vfactors_col(tp, g, f, dt, vf, n, threadIdx.x & 31);
}

// chunk ch of a column over a warp's lanes, HU halo levels above and HD below the stored levels
template <int HU, int HD>
struct Chunk {
    static constexpr int OUT = 32 - HU - HD;
    int nz;
    bool lvl, out;
    __device__ __forceinline__ Chunk(int nzmin, int nzmax, int ch, int lane) {
        nz = nzmin - HU + OUT * ch + lane;
        lvl = nz >= nzmin && nz <= nzmax - 1;
        out = lvl && lane >= HU && lane < 32 - HD;
    }
    static __device__ __forceinline__ int count(int nzmin, int nzmax) { return (nzmax - nzmin + OUT - 1) / OUT; }
};

// ---------------------------------------------------------------------------
// entries of G floats
// ---------------------------------------------------------------------------
template <int G>
struct Vec {
    float c[G];
};
template <int G>
__device__ __forceinline__ Vec<G> vfill(float x) {
    Vec<G> r;
#pragma unroll
    for (int k = 0; k < G; k++) r.c[k] = x;
    return r;
}
template <int G>
__device__ __forceinline__ Vec<G> vld(const float *__restrict__ p, int i);
template <>
__device__ __forceinline__ Vec<4> vld<4>(const float *__restrict__ p, int i) {
    const float4 q = reinterpret_cast<const float4 *>(p)[i];
    return Vec<4>{{q.x, q.y, q.z, q.w}};
}
template <>
__device__ __forceinline__ Vec<2> vld<2>(const float *__restrict__ p, int i) {
    const float2 q = reinterpret_cast<const float2 *>(p)[i];
    return Vec<2>{{q.x, q.y}};
}
// entry i where ok, zeros elsewhere (no load issued where !ok)
template <int G>
__device__ __forceinline__ Vec<G> vldc(bool ok, const float *__restrict__ p, int i) {
    Vec<G> r = vfill<G>(0.f);
    if (ok) r = vld<G>(p, i);
    return r;
}
// entry i where ok, read at L2 (ld.global.cg): values the same kernel stored before a
// __syncwarp, which a load through the read-only or L1 path is not bound to see
template <int G>
__device__ __forceinline__ Vec<G> vldcg(bool ok, const float *p, int i);
template <>
__device__ __forceinline__ Vec<4> vldcg<4>(bool ok, const float *p, int i) {
    Vec<4> r = vfill<4>(0.f);
    if (ok) {
        const float4 q = __ldcg(reinterpret_cast<const float4 *>(p) + i);
        r = Vec<4>{{q.x, q.y, q.z, q.w}};
    }
    return r;
}
template <>
__device__ __forceinline__ Vec<2> vldcg<2>(bool ok, const float *p, int i) {
    Vec<2> r = vfill<2>(0.f);
    if (ok) {
        const float2 q = __ldcg(reinterpret_cast<const float2 *>(p) + i);
        r = Vec<2>{{q.x, q.y}};
    }
    return r;
}
template <int G>
__device__ __forceinline__ void vst(float *p, int i, const Vec<G> &v);
template <>
__device__ __forceinline__ void vst<4>(float *p, int i, const Vec<4> &v) {
    reinterpret_cast<float4 *>(p)[i] = make_float4(v.c[0], v.c[1], v.c[2], v.c[3]);
}
template <>
__device__ __forceinline__ void vst<2>(float *p, int i, const Vec<2> &v) {
    reinterpret_cast<float2 *>(p)[i] = make_float2(v.c[0], v.c[1]);
}
// group g of a field of `count` entries per group
template <int G>
__device__ __forceinline__ const float *grp(const float *base, int g, size_t count) {
    return base + (size_t)g * count * G;
}
template <int G>
__device__ __forceinline__ float *grp(float *base, int g, size_t count) {
    return base + (size_t)g * count * G;
}

// Adams-Bashforth value minus the current value: AB2 -(0.5+eps) T^{n-1} + (1.5+eps) T^n,
// AB3 (23 T^n - 16 T^{n-1} + 5 T^{n-2}) / 12 (oce_tracer_mod.F90:53, 67-68), eps = 0.1
__device__ __forceinline__ float ab_delta(int ab, float t, float o1, float o2) {
    return ab == 2 ? 0.6f * (t - o1) : (11.f * (t - o1) - 5.f * (o1 - o2)) * (1.f / 12.f);
}

// upwind flux of an edge-layer in the edge's direction, -(T1 v+ + T2 v-)
// (oce_adv_tra_hor.F90:174-177, 0.5 (v +- |v|) = v+ / v-), both products rounded and then
// summed: the rounding k32_lo_ad's node sums use for the same flux
__device__ __forceinline__ float upw_flux(float T1, float T2, float v) {
    return -__fadd_rn(__fmul_rn(T1, fmaxf(v, 0.f)), __fmul_rn(T2, fminf(v, 0.f)));
}

// Packed FP32 pairs: two slots of a group in one instruction (Blackwell's two-wide FP32 add,
// multiply and fused multiply-add).  Each element rounds as the scalar
// operation does; a - b is formed as fma(b, -1, a), which rounds once, like the subtraction.
__device__ __forceinline__ float2 pk(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <int G>
__device__ __forceinline__ float2 pr(const Vec<G> &a, int j) {
    return make_float2(a.c[2 * j], a.c[2 * j + 1]);
}

// The per-group arithmetic of k32_lo_ad for two slots at once, from the values of the column's
// neighbouring layers: the upwind vertical flux with w_e, LO from the edge-flux sum hs, and the
// vertical antidiffusive flux (QR4C / UPW1 / CDIFF, oce_adv_tra_ver.F90:332-434, 635-695; the
// branches are taken per lane and group, so both slots of a pair share them).
// adv_tra_ver_upw1's flux of an interface with velocity w and area ar
__device__ __forceinline__ float2 upw_pair(float2 tn, float2 Tu, float w, float ar, bool top) {
    if (top) return pmul(tn, pk(-(w * ar)));
    const float aw = fabsf(w);
    return pmul(pfma(tn, pk(w + aw), pmul(Tu, pk(w - aw))), pk(-0.5f * ar));
}
struct LoLane {  // tracer-independent data of a node-layer
    int nz, nzmin, nzmax;
    float ar0, we0, w0, ar1, we1, sdt, dhr, idz0, idzp, idzm, g1, g2;
};
template <bool WS>
__device__ __forceinline__ void lo_ad_pair(const DForcing<float> &f, int ver, bool lim, float2 pv, const LoLane &k,
                                           float2 tn, float2 Tu, float2 Td, float2 tab, float2 tabu, float2 tabu2,
                                           float2 tabd, float2 hs, float2 &lo, float2 &ad) {
    const int nz = k.nz;
    const bool top = nz == k.nzmin;
    const float2 fv0 = upw_pair(tn, Tu, k.we0, k.ar0, top);
    const float2 fv1 = nz == k.nzmax - 1 ? pk(0.f) : upw_pair(Td, tn, k.we1, k.ar1, false);
    lo = padd(tn, pfma(tn, pk(k.dhr), pmul(padd(hs, psub(fv0, fv1)), pk(k.sdt))));
    float2 fw0 = fv0;
    if (WS && f.wsplit) fw0 = upw_pair(tn, Tu, k.w0, k.ar0, top);
    const float pw = lim ? k.w0 : k.we0;
    float2 Cf;
    if (top) {
        Cf = pmul(tab, pk(-(pw * k.ar0)));
    } else if (ver != 0 || nz == k.nzmin + 1 || nz == k.nzmax - 1) {
        if (ver != 1) {
            Cf = pmul(padd(tabu, tab), pk(-0.5f * pw * k.ar0));
        } else {
            const float aw = fabsf(pw);
            Cf = pmul(pfma(tab, pk(pw + aw), pmul(tabu, pk(pw - aw))), pk(-0.5f * k.ar0));
        }
    } else {
        const float2 qc = pmul(psub(tabu, tab), pk(k.idz0));
        const float2 qu = pmul(psub(tab, tabd), pk(k.idzp));
        const float2 qd = pmul(psub(tabu2, tabu), pk(k.idzm));
        const float2 Tm1 = pfma(pfma(pk(2.f), qc, qu), pk(k.g1), tab);
        const float2 Tm2 = pfma(pfma(pk(2.f), qc, qd), pk(k.g2), tabu);
        const float aw = fabsf(pw);
        const float2 Tmean = pfma(pk(pw + aw), Tm1, pmul(pk(pw - aw), Tm2));
        // (-(0.5 (1 - pv) Tmean) - pv (0.5 (Tm1 + Tm2)) pw) ar0
        const float2 a1 = pmul(pk(-0.5f), psub(pk(1.f), pv)), a2 = pmul(pk(-0.5f * pw), pv);
        Cf = pmul(pfma(a1, Tmean, pmul(a2, padd(Tm1, Tm2))), pk(k.ar0));
    }
    // flux = C - flux_in; FCT passes the LO flux in, otherwise zero
    float2 F = lim ? psub(Cf, fw0) : Cf;
    // a two-layer column writes its middle interface twice (statements nzmin+1, nzmax-1)
    if (ver == 0 && k.nzmin + 1 == k.nzmax - 1 && nz == k.nzmin + 1) F = psub(Cf, F);
    ad = lim ? F : psub(F, fv0);
}

// ---------------------------------------------------------------------------
// tiles of nodes
// ---------------------------------------------------------------------------
// A block takes a tile of consecutive whole columns with at most 256 wet layers in all (tiles cut
// once per mesh), one layer per thread, and keeps the layer's geometry, neighbour offsets and
// volume fluxes in registers for every tracer group of the launch.  The layers above and below
// sit in the neighbouring threads: they pass through shared memory, double-buffered over the
// groups, so a group costs one barrier.  Nothing is computed twice (a warp per column needs 3 of
// 32 lanes as halo and leaves the rest of a column's last chunk idle: 47 layers filled 73 % of
// two chunks), and a node's edge list is read once per tile into shared memory.
constexpr int kNT = kNodeTileLevels;  // threads
constexpr int kND = 6;                // edge slots of a node that k32_lo_ad holds in registers
constexpr int kSlots = kMaxDeg + 2;   // slots of a node in a tile: the last pass over ub or uu slots may run past kMaxDeg
struct NodeTile {
    int n0, cnt, total, degmax;
    int pre[kNodeTileNodes + 1], top[kNodeTileNodes], deg[kNodeTileNodes];
    // slot u of node j: first entry of the other end's column, of the edge's column, the edge's
    // levels lo | hi << 16, and whether the node is edges(1, e)
    int4 slot[kNodeTileNodes][kSlots];
    __device__ __forceinline__ int find(int i) const {
        int j = i >= pre[16] ? 16 : 0;
        j += i >= pre[j + 8] ? 8 : 0;
        j += i >= pre[j + 4] ? 4 : 0;
        j += i >= pre[j + 2] ? 2 : 0;
        return j + (i >= pre[j + 1] ? 1 : 0);
    }
};

// every thread of the block; the tile's data are visible after it
__device__ __forceinline__ void node_tile_load(const DTopo &tp, int ti, NodeTile &S) {
    const int n0 = tp.nt_ptr[ti], cnt = tp.nt_ptr[ti + 1] - n0;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, n = n0 + j;
        const bool in = j < cnt;
        int s = in ? tp.n_nlev[n] - tp.n_ulev[n] : 0;
        S.top[j] = in ? tp.n_ulev[n] : 1;
        const int deg = in ? min(tp.ne_ptr[n + 1] - tp.ne_ptr[n], kMaxDeg) : 0;
        S.deg[j] = deg;
        const int dm = __reduce_max_sync(kFull, deg);
        if (j == 0) S.degmax = dm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, s, o);
            if (j >= o) s += v;
        }
        S.pre[j + 1] = s;
        if (j == 0) {
            S.pre[0] = 0;
            S.n0 = n0;
            S.cnt = cnt;
        }
        if (j == 31) S.total = s;
    }
    for (int s = threadIdx.x; s < cnt * kMaxDeg; s += kNT) {
        const int j = s / kMaxDeg, u = s % kMaxDeg;
        const int k = tp.ne_ptr[n0 + j] + u;
        if (k >= tp.ne_ptr[n0 + j + 1]) continue;
        const int code = tp.ne_idx[k], e = code >= 0 ? code : ~code;
        const int m = code >= 0 ? tp.e_n2[e] : tp.e_n1[e];
        S.slot[j][u] = make_int4(m * tp.L1, e * tp.L1, tp.e_lo[e] | tp.e_hi[e] << 16, code >= 0);
    }
    __syncthreads();
}

// the thread's layer of a tile
struct TileLane {
    bool on;
    int j, n, nz, nzmin, nzmax, i, iv;
    __device__ __forceinline__ TileLane(const DTopo &tp, const NodeTile &S) {
        on = threadIdx.x < S.total;
        j = S.find(on ? threadIdx.x : 0);
        n = S.n0 + j;
        nzmin = S.top[j];
        nzmax = nzmin + S.pre[j + 1] - S.pre[j];
        nz = nzmin + (on ? (int)threadIdx.x - S.pre[j] : 0);
        i = n * tp.L1 + nz - 1;
        iv = n * tp.nl + nz - 1;
    }
};
__device__ __forceinline__ bool slot_wet(const int4 &q, int nz) { return nz >= (q.z & 0xffff) && nz <= (q.z >> 16); }

// loop of the blocks over the tiles (one launch may hold fewer blocks than tiles)
#define FOR_NODE_TILES(ti, ntiles) for (int ti = blockIdx.x; ti < (ntiles); ti += gridDim.x)

// ---------------------------------------------------------------------------
// k32_lo_ad
// ---------------------------------------------------------------------------
// The node's share of an edge's upwind flux F = -(T1 v+ + T2 v-) (+F at edges(1,e), -F at
// edges(2,e)) is rn(rn(T_n p) + rn(T_m q)) with (p, q) = (-v+, -v-) at edges(1,e) and (v-, v+) at
// edges(2,e): the same two products and the same sum as at the other end, so the two ends add
// exactly opposite values.
//
// Bound by the latency of its gathers (issue 43 %, 32 warps per SM).  A warp per node and chunk, its
// gathers staged by cp.async: 307 us on the sphere of 7 subdivisions, 48 levels, T and S, this form
// 165; with 24 tracers on the sphere of 8, 70 levels, 4.4 -> 3.6 ms.
__device__ __forceinline__ void edge_share(float v, bool own, float &p, float &q) {
    const float vp = fmaxf(v, 0.f), vm = fminf(v, 0.f);
    p = own ? -vp : vm;
    q = own ? -vm : vp;
}
template <int G>
using LoBuf = Vec<G>[2][2][kNT];  // [buffer][T, AB value][thread]

template <int G, bool WS>
__device__ __forceinline__ void lo_ad_tile(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f,
                                           const B32View &B, const float *__restrict__ VF, float dt,
                                           const NodeTile &S, LoBuf<G> &X) {
    const TileLane k(tp, S);
    const int x = threadIdx.x, i = k.i, iv = k.iv, nz = k.nz, deg = S.deg[k.j];
    // dry and missing slots: offset -1, no flux
    int off[kND];
    float pq[kND], qq[kND];
#pragma unroll
    for (int u = 0; u < kND; u++) {
        const int4 q = S.slot[k.j][u];
        const bool ok = k.on && u < deg && slot_wet(q, nz);
        off[u] = ok ? q.x + nz - 1 : -1;
        edge_share(ok ? VF[q.y + nz - 1] : 0.f, q.w != 0, pq[u], qq[u]);
    }
    LoLane L{nz, k.nzmin, k.nzmax, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (k.on) {
        L.ar0 = g.area[iv];
        L.we0 = f.we[iv];
        L.w0 = f.w[iv];
        const float hn = g.hnode_new[i];
        L.sdt = qdiv(dt, g.areasvol[iv] * hn);
        L.dhr = qdiv(g.hnode[i] - hn, hn);
        if (nz < k.nzmax - 1) {
            L.ar1 = g.area[iv + 1];
            L.we1 = f.we[iv + 1];
        }
        // QR4C interior geometry, nzmin+2 <= nz <= nzmax-2 (oce_adv_tra_ver.F90:409-425)
        if (nz >= k.nzmin + 2 && nz <= k.nzmax - 2) {
            const float Z0 = g.Z3[i], Zm1 = g.Z3[i - 1], Zm2 = g.Z3[i - 2], Zp1 = g.Z3[i + 1], zb = g.zbar3[iv];
            L.idz0 = qdiv(1.f, Zm1 - Z0);
            L.idzp = qdiv(1.f, Z0 - Zp1);
            L.idzm = qdiv(1.f, Zm2 - Zm1);
            L.g1 = (zb - Z0) * (1.f / 3.f);
            L.g2 = (zb - Zm1) * (1.f / 3.f);
        }
    }
#pragma unroll 1
    for (int gi = 0; gi < B.ng; gi++) {
        const bool lim = (B.fct >> gi) & 1ull;
        const int ver = B.ver[gi];
        const float *__restrict__ T = grp<G>(B.T, gi, B.sN);
        // every load of the group first
        const Vec<G> Tn = vldc<G>(k.on, T, i);
        const Vec<G> o1 = vldc<G>(k.on, grp<G>(B.O1, gi, B.sN), i);
        const Vec<G> o2 = vldc<G>(k.on && B.ab == 3, B.ab == 3 ? grp<G>(B.O2, gi, B.sN) : T, i);
        Vec<G> tm[kND];
#pragma unroll
        for (int u = 0; u < kND; u++) tm[u] = vldc<G>(off[u] >= 0, T, off[u]);
        Vec<G> ta;
#pragma unroll
        for (int j = 0; j < G / 2; j++) {
            const float2 tn = pr(Tn, j), p1 = pr(o1, j), p2 = pr(o2, j);
            const float2 t = B.ab == 2 ? pfma(pk(0.6f), psub(tn, p1), tn)
                                       : pfma(pfma(pk(11.f), psub(tn, p1), pmul(pk(-5.f), psub(p1, p2))),
                                              pk(1.f / 12.f), tn);
            ta.c[2 * j] = t.x;
            ta.c[2 * j + 1] = t.y;
        }
        Vec<G>(&xt)[kNT] = X[gi & 1][0], (&xa)[kNT] = X[gi & 1][1];
        xt[x] = Tn;
        xa[x] = ta;
        float2 hs[G / 2];
#pragma unroll
        for (int j = 0; j < G / 2; j++) {
            hs[j] = pk(0.f);
#pragma unroll
            for (int u = 0; u < kND; u++)
                hs[j] = padd(hs[j], padd(pmul(pr(Tn, j), pk(pq[u])), pmul(pr(tm[u], j), pk(qq[u]))));
        }
        for (int u = kND; u < deg; u++) {  // nodes of more edges
            const int4 q = S.slot[k.j][u];
            if (!k.on || !slot_wet(q, nz)) continue;
            float p, r;
            edge_share(VF[q.y + nz - 1], q.w != 0, p, r);
            const Vec<G> t = vld<G>(T, q.x + nz - 1);
#pragma unroll
            for (int j = 0; j < G / 2; j++) hs[j] = padd(hs[j], padd(pmul(pr(Tn, j), pk(p)), pmul(pr(t, j), pk(r))));
        }
        __syncthreads();
        if (!k.on) continue;
        // the layers above (up to two) and below; at the column's ends the thread's own entry (unused)
        const int a1 = nz > k.nzmin ? x - 1 : x, a2 = nz > k.nzmin + 1 ? x - 2 : x, d1 = nz < k.nzmax - 1 ? x + 1 : x;
        const Vec<G> Tu = xt[a1], Td = xt[d1], au = xa[a1], au2 = xa[a2], adn = xa[d1];
        Vec<G> lo, ad;
#pragma unroll
        for (int j = 0; j < G / 2; j++) {
            float2 l2, d2;
            lo_ad_pair<WS>(f, ver, lim, make_float2(B.pv[gi * G + 2 * j], B.pv[gi * G + 2 * j + 1]), L, pr(Tn, j),
                           pr(Tu, j), pr(Td, j), pr(ta, j), pr(au, j), pr(au2, j), pr(adn, j), hs[j], l2, d2);
            lo.c[2 * j] = l2.x;
            lo.c[2 * j + 1] = l2.y;
            ad.c[2 * j] = d2.x;
            ad.c[2 * j + 1] = d2.y;
        }
        vst<G>(grp<G>(B.LO, gi, B.sN), i, lo);
        // PPM fluxes come from k32_vppm
        if (ver != 3) vst<G>(grp<G>(B.ADv, gi, B.sNI), iv, ad);
    }
}

template <int G, bool WS>
__global__ void __launch_bounds__(kNT, MinB<G>::lo)
k32_lo_ad(DTopo tp, DGeom<float> g, DForcing<float> f, B32View B, const float *__restrict__ VF, float dt) {
    __shared__ NodeTile S;
    __shared__ LoBuf<G> X;
    FOR_NODE_TILES(ti, tp.n_nt) {
        node_tile_load(tp, ti, S);
        lo_ad_tile<G, WS>(tp, g, f, B, VF, dt, S, X);
        __syncthreads();
    }
}

// grid-stride loop of the warps over the units (one launch may hold fewer blocks than units)
#define FOR_WARP_UNITS(j, count)                                                               \
    for (int j = blockIdx.x * kWB + (threadIdx.x >> 5); j < (count); j += gridDim.x * kWB)

// high-order minus low-order flux of one edge-layer from the two end values, their
// previous time levels and the projected gradients s1 (up) / s2 (down)
__device__ __forceinline__ float ho_minus_lo(int hor, float ph, int ab, float T1, float T2, float o1a, float o1b,
                                             float o2a, float o2b, float s1, float s2, float v, float cl1, float cl2) {
    const float vp = fmaxf(v, 0.f), vm = fminf(v, 0.f);
    const float t1 = T1 + ab_delta(ab, T1, o1a, o2a);
    const float t2 = T2 + ab_delta(ab, T2, o1b, o2b);
    const float flo = upw_flux(T1, T2, v);
    float hf;
    if (hor == 2) {
        hf = upw_flux(t1, t2, v);
    } else {
        // c_lo = 1 up to nboundary_lay (MUSCL), always 1 (MFCT)
        const float clo1 = hor == 0 ? cl1 : 1.f, clo2 = hor == 0 ? cl2 : 1.f;
        const float d2 = 2.f * (t2 - t1);
        const float Tm2 = t2 - (d2 + s2) * (1.f / 6.f) * clo2;
        const float Tm1 = t1 + (d2 + s1) * (1.f / 6.f) * clo1;
        const float cHO = 2.f * (vp * Tm1 + vm * Tm2);
        hf = -(0.5f * (1.f - ph) * cHO) - v * ph * 0.5f * (Tm1 + Tm2);
    }
    return hf - flo;
}

// hor, ab uniform over the pair; q1 = 1 - ph, q2 = v ph / 2 per slot; vp, vm the upwind parts of v
__device__ __forceinline__ float2 ho_minus_lo2(int hor, int ab, float2 q1, float2 q2, float2 T1, float2 T2,
                                               float2 o1a, float2 o1b, float2 o2a, float2 o2b, float2 s1,
                                               float2 s2, float vp, float vm, float cl1, float cl2) {
    float2 t1, t2;
    if (ab == 2) {
        t1 = pfma(pk(0.6f), psub(T1, o1a), T1);
        t2 = pfma(pk(0.6f), psub(T2, o1b), T2);
    } else {
        t1 = pfma(pfma(pk(11.f), psub(T1, o1a), pmul(pk(-5.f), psub(o1a, o2a))), pk(1.f / 12.f), T1);
        t2 = pfma(pfma(pk(11.f), psub(T2, o1b), pmul(pk(-5.f), psub(o1b, o2b))), pk(1.f / 12.f), T2);
    }
    // minus the LO flux: + (T1 v+ + T2 v-), both products rounded, then summed
    const float2 lo = padd(pmul(T1, pk(vp)), pmul(T2, pk(vm)));
    if (hor == 2) return psub(lo, padd(pmul(t1, pk(vp)), pmul(t2, pk(vm))));
    const float clo1 = hor == 0 ? cl1 : 1.f, clo2 = hor == 0 ? cl2 : 1.f;
    const float2 d2 = pmul(pk(2.f), psub(t2, t1));
    const float2 Tm2 = pfma(pmul(padd(d2, s2), pk(1.f / 6.f)), pk(-clo2), t2);
    const float2 Tm1 = pfma(pmul(padd(d2, s1), pk(1.f / 6.f)), pk(clo1), t1);
    // hf = -(1 - ph) (v+ Tm1 + v- Tm2) - (v ph / 2) (Tm1 + Tm2)
    const float2 c = pfma(pk(vp), Tm1, pmul(pk(vm), Tm2));
    return psub(lo, pfma(q1, c, pmul(q2, padd(Tm1, Tm2))));
}

// ---------------------------------------------------------------------------
// k32_ho: high-order minus low-order flux of every edge-layer
// ---------------------------------------------------------------------------
// A tile of edges over their levels [nu12, nl12].  MUSCL / MFCT
// (adv_tra_hor_muscl / _mfct, oce_adv_tra_hor.F90:261-834) on the AB values with the
// gradients of fill_up_dn_grad (oce_muscl_adv.F90:356-525); UPW1 (:64-257).  The LO
// flux is the upwind flux of the current values (oce_adv_tra_driver.F90:131-190).
//
// The up triangle holds edges(1,e) and the down triangle edges(2,e); their gradients,
// projected on the edge, are wu.y (T(un.y) - T1) + wu.z (T(un.z) - T1) and the same
// for the down triangle (the three weights of a triangle sum to zero).  Those apply
// at the levels where every element around both nodes is wet, [gzmin, gzmax); the
// other edge-layers (under one percent of an ocean mesh's) take the node means in
// k32_ho_nodemean.
//
// Bound by the latency of ten gathers per edge-layer and group.  A warp per edge took 237 us on the
// sphere of 7 subdivisions, 48 levels, T and S, this form 132; 4.6 -> 4.0 ms with 24 tracers on the
// sphere of 8, 70 levels.
// the group's high-minus-low fluxes of one edge-layer from its gathered entries
template <int G>
__device__ __forceinline__ Vec<G> ho_group(const B32View &B, int gq, int hor, const Vec<G> &T1, const Vec<G> &T2,
                                           const Vec<G> &o1a, const Vec<G> &o1b, const Vec<G> &o2a, const Vec<G> &o2b,
                                           const Vec<G> &ga, const Vec<G> &gb, const Vec<G> &gc, const Vec<G> &gd,
                                           const float4 &wu, const float4 &wd, float v, float cl1, float cl2) {
    Vec<G> out;
#if FESOM_PACKED_PAIRS
    const float vp = fmaxf(v, 0.f), vm = fminf(v, 0.f);
#pragma unroll
    for (int j = 0; j < G / 2; j++) {
        const float2 ph = make_float2(B.ph[gq * G + 2 * j], B.ph[gq * G + 2 * j + 1]);
        const float2 q1 = psub(pk(1.f), ph), q2 = pmul(pk(0.5f * v), ph);
        const float2 t1 = pr(T1, j), t2 = pr(T2, j);
        const float2 s1 = pfma(pk(wu.y), psub(pr(ga, j), t1), pmul(pk(wu.z), psub(pr(gb, j), t1)));
        const float2 s2 = pfma(pk(wd.y), psub(pr(gc, j), t2), pmul(pk(wd.z), psub(pr(gd, j), t2)));
        const float2 r = ho_minus_lo2(hor, B.ab, q1, q2, t1, t2, pr(o1a, j), pr(o1b, j), pr(o2a, j), pr(o2b, j), s1,
                                      s2, vp, vm, cl1, cl2);
        out.c[2 * j] = r.x;
        out.c[2 * j + 1] = r.y;
    }
#else
#pragma unroll
    for (int c = 0; c < G; c++) {
        const float s1 = wu.y * (ga.c[c] - T1.c[c]) + wu.z * (gb.c[c] - T1.c[c]);
        const float s2 = wd.y * (gc.c[c] - T2.c[c]) + wd.z * (gd.c[c] - T2.c[c]);
        out.c[c] = ho_minus_lo(hor, B.ph[gq * G + c], B.ab, T1.c[c], T2.c[c], o1a.c[c], o1b.c[c], o2a.c[c], o2b.c[c],
                               s1, s2, v, cl1, cl2);
    }
#endif
    return out;
}

struct EdgeH {
    int ia, ib, ua, ub, da, db;  // first entries of the columns of both ends and of the triangles' other nodes
    int gmin, gmax, nbl1, nbl2;
    float uy, uz, dy, dz;
};

// tile ti of `tile` edges
template <int G>
__device__ __forceinline__ void ho_tile(const DTopo &tp, const B32View &B, const MusclW &mw,
                                        const float *__restrict__ VF, int ti, int tile, Tile &S, EdgeH *Ed) {
    const int L1 = tp.L1, e0 = ti * tile;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, e = e0 + j;
        const bool in = j < tile && e < tp.E2;
        if (in) {
            EdgeH &E = Ed[j];
            const int n1 = tp.e_n1[e], n2 = tp.e_n2[e];
            const int4 un = mw.un[e], dn = mw.dn[e];
            const float4 wu = mw.wu[e], wd = mw.wd[e];
            E.ia = n1 * L1;
            E.ib = n2 * L1;
            E.ua = un.y * L1;
            E.ub = un.z * L1;
            E.da = dn.y * L1;
            E.db = dn.z * L1;
            E.gmin = un.w & 0xffff;
            E.gmax = un.w >> 16;
            E.nbl1 = tp.n_nbl[n1];
            E.nbl2 = tp.n_nbl[n2];
            E.uy = wu.y;
            E.uz = wu.z;
            E.dy = wd.y;
            E.dz = wd.z;
        }
        S.fill(j, in ? tp.e_lo[e] : 1, in ? tp.e_hi[e] - tp.e_lo[e] + 1 : 0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j], k = nz - 1;
        const EdgeH &E = Ed[j];
        const bool tri = nz >= E.gmin && nz <= E.gmax - 1;
        const int ie = (e0 + j) * L1 + k, ia = E.ia + k, ib = E.ib + k;
        const int ua = E.ua + k, ub = E.ub + k, da = E.da + k, db = E.db + k;
        const float v = VF[ie];
        const float cl1 = (E.nbl1 - nz) >= 0 ? 1.f : 0.f, cl2 = (E.nbl2 - nz) >= 0 ? 1.f : 0.f;
        const float4 wu = make_float4(0.f, E.uy, E.uz, 0.f), wd = make_float4(0.f, E.dy, E.dz, 0.f);
#pragma unroll 1
        for (int gq = 0; gq < B.ng; gq++) {
            const int hor = B.hor[gq];
            // MUSCL / MFCT levels outside the triangles' range: the node-mean launch
            if (hor != 2 && !tri) continue;
            const bool grad = hor != 2;
            const float *__restrict__ T = grp<G>(B.T, gq, B.sN);
            const float *__restrict__ O1 = grp<G>(B.O1, gq, B.sN);
            const float *__restrict__ O2 = B.ab == 3 ? grp<G>(B.O2, gq, B.sN) : O1;
            const Vec<G> T1 = vld<G>(T, ia), T2 = vld<G>(T, ib);
            const Vec<G> o1a = vld<G>(O1, ia), o1b = vld<G>(O1, ib);
            const Vec<G> o2a = vldc<G>(B.ab == 3, O2, ia), o2b = vldc<G>(B.ab == 3, O2, ib);
            const Vec<G> ga = vldc<G>(grad, T, ua), gb = vldc<G>(grad, T, ub);
            const Vec<G> gc = vldc<G>(grad, T, da), gd = vldc<G>(grad, T, db);
            vst<G>(grp<G>(B.ADh, gq, B.sE), ie,
                   ho_group<G>(B, gq, hor, T1, T2, o1a, o1b, o2a, o2b, ga, gb, gc, gd, wu, wd, v, cl1, cl2));
        }
    }
}

template <int G>
__global__ void __launch_bounds__(kTileThreads, MinB<G>::ho)
k32_ho(DTopo tp, B32View B, MusclW mw, const float *__restrict__ VF, int tile) {
    __shared__ Tile S;
    __shared__ EdgeH Ed[kTileMax];
    ho_tile<G>(tp, B, mw, VF, blockIdx.x, tile, S, Ed);
}

// The edge-layers of the node-mean gradients: one thread per (edge, level) item, every
// group, with the projected mean gradients as precomputed neighbour weights.
template <int G>
__device__ __forceinline__ void nodemean_item(const DTopo &tp, const B32View &B, const MusclW &mw,
                                              const float *__restrict__ VF, int j) {
    const int L1 = tp.L1;
    const int e = mw.it_e[j], nz = mw.it_nz[j];
    const int p0 = mw.it_ptr[j], p1 = p0 + mw.it_n1[j], p2 = mw.it_ptr[j + 1];
    const int n1 = tp.e_n1[e], n2 = tp.e_n2[e];
    const int ie = e * L1 + nz - 1, ia = n1 * L1 + nz - 1, ib = n2 * L1 + nz - 1;
    const float v = VF[ie];
    const float cl1 = (tp.n_nbl[n1] - nz) >= 0 ? 1.f : 0.f, cl2 = (tp.n_nbl[n2] - nz) >= 0 ? 1.f : 0.f;
#pragma unroll 1
    for (int gq = 0; gq < B.ng; gq++) {
        const int hor = B.hor[gq];
        if (hor == 2) continue;  // UPW1 has no gradients: k32_ho wrote it
        const float *__restrict__ T = grp<G>(B.T, gq, B.sN);
        const float *__restrict__ O1 = grp<G>(B.O1, gq, B.sN);
        const Vec<G> T1 = vld<G>(T, ia), T2 = vld<G>(T, ib);
        const Vec<G> o1a = vld<G>(O1, ia), o1b = vld<G>(O1, ib);
        const Vec<G> o2a = vldc<G>(B.ab == 3, grp<G>(B.O2, gq, B.sN), ia);
        const Vec<G> o2b = vldc<G>(B.ab == 3, grp<G>(B.O2, gq, B.sN), ib);
        Vec<G> s1 = vfill<G>(0.f), s2 = vfill<G>(0.f);
        for (int p = p0; p < p1; p++) {
            const int2 q = mw.pairs[p];
            const Vec<G> t = vld<G>(T, q.x * L1 + nz - 1);
#pragma unroll
            for (int c = 0; c < G; c++) s1.c[c] += __int_as_float(q.y) * (t.c[c] - T1.c[c]);
        }
        for (int p = p1; p < p2; p++) {
            const int2 q = mw.pairs[p];
            const Vec<G> t = vld<G>(T, q.x * L1 + nz - 1);
#pragma unroll
            for (int c = 0; c < G; c++) s2.c[c] += __int_as_float(q.y) * (t.c[c] - T2.c[c]);
        }
        Vec<G> out;
#pragma unroll
        for (int c = 0; c < G; c++)
            out.c[c] = ho_minus_lo(hor, B.ph[gq * G + c], B.ab, T1.c[c], T2.c[c], o1a.c[c], o1b.c[c], o2a.c[c],
                                   o2b.c[c], s1.c[c], s2.c[c], v, cl1, cl2);
        vst<G>(grp<G>(B.ADh, gq, B.sE), ie, out);
    }
}

template <int G>
__global__ void __launch_bounds__(256) k32_ho_nodemean(DTopo tp, B32View B, MusclW mw, const float *__restrict__ VF) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < mw.n_items; j += gridDim.x * blockDim.x)
        nodemean_item<G>(tp, B, mw, VF, j);
}

// ---------------------------------------------------------------------------
// k32_bounds: FCT bounds and R+ / R- (FCT groups only)
// ---------------------------------------------------------------------------
// FCT bounds (max / min of LO and T over the node, its neighbours and the adjacent layers) and R+ / R-
// of the FCT groups.  Bound by the latency of its gathers, 320 bytes per layer and group of 4: 7.8 warps
// a scheduler at 64 registers issue in 50 % of the cycles, and of the rest most wait for loads; L2 at
// 36 % of its rate, DRAM at 42 % (12 tracers, 70 layers).  Sphere of 7 subdivisions, T and S: 220 -> 152
// us against a warp per node; 24 tracers on the sphere of 8: 5.1 -> 5.5 ms, where the barrier per group
// costs more than the full lanes give.
template <int G>
using BoundsBuf = Vec<G>[2][2][kNT];  // [buffer][max, min][thread]

template <int G>
__device__ __forceinline__ void bounds_tile(const DTopo &tp, const DGeom<float> &g, const B32View &B, float dt,
                                            const NodeTile &S, BoundsBuf<G> &X) {
    constexpr int kUB = MinB<G>::ub;
    const TileLane k(tp, S);
    const int x = threadIdx.x, i = k.i, iv = k.iv, nz = k.nz, deg = S.deg[k.j];
    const float eps = (float)kFluxEps;
    const float s = k.on ? qdiv(dt, g.areasvol[iv] * g.hnode_new[i]) : 0.f;
    int b = 0;
#pragma unroll 1
    for (int gq = 0; gq < B.ng; gq++) {
        if (!((B.fct >> gq) & 1ull)) continue;
        const float *__restrict__ T = grp<G>(B.T, gq, B.sN);
        const float *__restrict__ LO = grp<G>(B.LO, gq, B.sN);
        const float *__restrict__ ADh = grp<G>(B.ADh, gq, B.sE);
        const Vec<G> Tn = vldc<G>(k.on, T, i);
        const Vec<G> lo = vldc<G>(k.on, LO, i);
        const Vec<G> v0 = vldc<G>(k.on, grp<G>(B.ADv, gq, B.sNI), iv);
        const Vec<G> v1 = vldc<G>(k.on && nz < k.nzmax - 1, grp<G>(B.ADv, gq, B.sNI), iv + 1);
        // bounds over the node, its neighbours and the layers above and below
        // (oce_adv_tra_fct.F90:124-248); P / M: sums of the positive / negative antidiffusive
        // fluxes into the node
        Vec<G> mx, mn, Pp = vfill<G>(0.f), M = vfill<G>(0.f);
#pragma unroll
        for (int c = 0; c < G; c++) {
            mx.c[c] = fmaxf(lo.c[c], Tn.c[c]);
            mn.c[c] = fminf(lo.c[c], Tn.c[c]);
        }
#pragma unroll 1
        for (int u0 = 0; u0 < S.degmax; u0 += kUB) {
            Vec<G> tm[kUB], lm[kUB], xe[kUB];
#pragma unroll
            for (int u = 0; u < kUB; u++) {
                const int4 q = S.slot[k.j][u0 + u];
                const bool ok = k.on && u0 + u < deg && slot_wet(q, nz);
                // a dry or missing slot: the node's own values (neutral for the bounds), no flux
                tm[u] = Tn;
                lm[u] = lo;
                if (ok) tm[u] = vld<G>(T, q.x + nz - 1);
                if (ok) lm[u] = vld<G>(LO, q.x + nz - 1);
                xe[u] = vldc<G>(ok, ADh, q.y + nz - 1);
            }
#pragma unroll
            for (int u = 0; u < kUB; u++) {
                const bool ow = S.slot[k.j][u0 + u].w != 0;
#pragma unroll
                for (int c = 0; c < G; c++) {
                    mx.c[c] = fmaxf(mx.c[c], fmaxf(tm[u].c[c], lm[u].c[c]));
                    mn.c[c] = fminf(mn.c[c], fminf(tm[u].c[c], lm[u].c[c]));
                    const float xv = ow ? xe[u].c[c] : -xe[u].c[c];
                    Pp.c[c] += fmaxf(0.f, xv);
                    M.c[c] += fminf(0.f, xv);
                }
            }
        }
        Vec<G>(&xmx)[kNT] = X[b][0], (&xmn)[kNT] = X[b][1];
        xmx[x] = mx;
        xmn[x] = mn;
        b ^= 1;
        __syncthreads();
        if (!k.on) continue;
        if (nz != k.nzmin && nz != k.nzmax - 1) {
            const Vec<G> mxu = xmx[x - 1], mxd = xmx[x + 1], mnu = xmn[x - 1], mnd = xmn[x + 1];
#pragma unroll
            for (int c = 0; c < G; c++) {
                mx.c[c] = fmaxf(fmaxf(mxu.c[c], mx.c[c]), mxd.c[c]);
                mn.c[c] = fminf(fminf(mnu.c[c], mn.c[c]), mnd.c[c]);
            }
        }
        Vec<G> rp, rm;
#pragma unroll
        for (int c = 0; c < G; c++) {
            const float pp = Pp.c[c] + (fmaxf(0.f, v0.c[c]) + fmaxf(0.f, -v1.c[c]));
            const float mm = M.c[c] + (fminf(0.f, v0.c[c]) + fminf(0.f, -v1.c[c]));
            rp.c[c] = fminf(1.f, qdiv(mx.c[c] - lo.c[c], pp * s + eps));
            rm.c[c] = fminf(1.f, qdiv(mn.c[c] - lo.c[c], mm * s - eps));
        }
        vst<G>(grp<G>(B.Rp, gq, B.sN), i, rp);
        vst<G>(grp<G>(B.Rm, gq, B.sN), i, rm);
        if (kFctClamp) {
            // the bounds themselves: the update clamps the advected value into them
            vst<G>(grp<G>(B.Bp, gq, B.sN), i, mx);
            vst<G>(grp<G>(B.Bm, gq, B.sN), i, mn);
        }
    }
}

template <int G>
__global__ void __launch_bounds__(kNT, MinB<G>::bounds)
k32_bounds(DTopo tp, DGeom<float> g, B32View B, float dt) {
    __shared__ NodeTile S;
    __shared__ BoundsBuf<G> X;
    FOR_NODE_TILES(ti, tp.n_nt) {
        node_tile_load(tp, ti, S);
        bounds_tile<G>(tp, g, B, dt, S, X);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// k32_vdiff: implicit vertical diffusion of the advected columns (in Tnew)
// ---------------------------------------------------------------------------
// Forward substitution tp_k = inv_k rhs_k - a_k inv_k tp_{k-1} and back substitution
// x_k = tp_k - cp_k x_{k+1} (oce_ale_tracer.F90:1406-1422) with the column's k32_vfactors
// factors, as scans of affine maps y -> A y + B.  Each lane holds K consecutive levels of the
// column (K = ceil(layers / 32): one warp covers the whole column): it composes its K maps in
// registers, the warp scans the lane maps (five shuffles), and each lane then runs its K
// levels from the carry it receives.  The multipliers A depend on the column only: the lane
// products and their partial products at each scan step are formed once per node (shared
// memory), so a slot's scan step is one shuffle and one multiply-add, and a column costs a slot
// 14 shuffles whatever its depth.  rhs_k = -a_k (T_{k-1} - T_k) - c_k (T_{k+1} - T_k)
// (+ bc_surface at the top, :1216-1229, 1377-1383); T += x.
// CG: the column was stored by the same kernel (the update with the diffusion as its epilogue):
// its values are read at L2.
constexpr int kWV = 4;                    // warps (nodes) per block of the diffusion kernel
constexpr int kScan = 5;                  // steps of a 32-lane scan

struct VdiffWarp {
    float4 fac[130];                      // (a, c, 1/m, c/m), 1-based levels
    float af[kScan][32];                  // forward: lane-map product of the window at each step (0 below the offset)
    float ab[kScan][32];                  // backward (0 past the offset)
};

// per-lane column data of a node: the factors of the lane's K levels
template <int K>
struct VdiffLane {
    float a[K], c[K], inv[K], A[K], Ad[K];
    bool ok[K];
};

// a group's column values of the lane's K levels and its surface flux
template <int K, int G>
struct VdiffCol {
    Vec<G> a[K];
    Vec<G> bc;
};

template <int K, int G, bool CG>
__device__ __forceinline__ void vdiff_load(const DTopo &tp, const B32View &B, int n, int lane, int nzmin, int gq,
                                           const VdiffLane<K> &V, VdiffCol<K, G> &x) {
    const int L1 = tp.L1;
    const int nz0 = nzmin + lane * K;  // the lane's first level
    const float *Tg = grp<G>(B.Tnew, gq, B.sN);
    x.bc = B.fsurf ? vld<G>(B.fsurf, gq * tp.N2 + n) : vfill<G>(0.f);
#pragma unroll
    for (int t = 0; t < K; t++)
        x.a[t] = CG ? vldcg<G>(V.ok[t], Tg, n * L1 + nz0 + t - 1) : vldc<G>(V.ok[t], Tg, n * L1 + nz0 + t - 1);
}

template <int K, int G>
__device__ __forceinline__ void vdiff_group(const DTopo &tp, const B32View &B, int n, int lane, int nzmin, int nzmax,
                                            int gq, const VdiffLane<K> &V, const VdiffWarp &W,
                                            const VdiffCol<K, G> &x) {
    const int L1 = tp.L1;
    const int nz0 = nzmin + lane * K;  // the lane's first level
    float *__restrict__ Tg = grp<G>(B.Tnew, gq, B.sN);
    const Vec<G>(&a)[K] = x.a;
    const Vec<G> &bc = x.bc;
    Vec<G> y[K];
#pragma unroll
    for (int c = 0; c < G; c++) {
        // the levels next to the lane's ends come from the neighbouring lanes
        const float up = sh_up(a[K - 1].c[c], 1), dn = sh_dn(a[0].c[c], 1);
        float bl = 0.f;  // the lane's composed forward map applied to 0
#pragma unroll
        for (int t = 0; t < K; t++) {
            const int nz = nz0 + t;
            const float tu = t > 0 ? a[t - 1].c[c] : up, td = t < K - 1 ? a[t + 1].c[c] : dn;
            const float tc = a[t].c[c];
            float r = 0.f;
            if (nz > nzmin) r -= V.a[t] * (tu - tc);
            if (nz < nzmax - 1) r -= V.c[t] * (td - tc);
            if (nz == nzmin) r += bc.c[c];
            y[t].c[c] = V.ok[t] ? r * V.inv[t] : 0.f;
            bl = fmaf(V.A[t], bl, y[t].c[c]);
        }
        // inclusive scan of the lane maps: bl = tp at the lane's last level
#pragma unroll
        for (int s = 0, off = 1; s < kScan; s++, off <<= 1) bl = fmaf(W.af[s][lane], __shfl_up_sync(kFull, bl, off), bl);
        float yv = __shfl_up_sync(kFull, bl, 1);
        if (lane == 0) yv = 0.f;
#pragma unroll
        for (int t = 0; t < K; t++) {
            yv = fmaf(V.A[t], yv, y[t].c[c]);
            y[t].c[c] = yv;
        }
        // back substitution: the lane's composed backward map, the suffix scan, the lane's levels
        float xl = 0.f;
#pragma unroll
        for (int t = K - 1; t >= 0; t--) xl = fmaf(V.Ad[t], xl, y[t].c[c]);
#pragma unroll
        for (int s = 0, off = 1; s < kScan; s++, off <<= 1)
            xl = fmaf(W.ab[s][lane], __shfl_down_sync(kFull, xl, off), xl);
        float xv = __shfl_down_sync(kFull, xl, 1);
        if (lane == 31) xv = 0.f;
#pragma unroll
        for (int t = K - 1; t >= 0; t--) {
            xv = fmaf(V.Ad[t], xv, y[t].c[c]);
            y[t].c[c] = a[t].c[c] + xv;
        }
    }
#pragma unroll
    for (int t = 0; t < K; t++) {
        if (!V.ok[t]) continue;
        bool fin = true;
#pragma unroll
        for (int c = 0; c < G; c++) fin = fin && isfinite(y[t].c[c]);
        vst<G>(Tg, n * L1 + nz0 + t - 1, y[t]);
        if (!fin) atomicOr(B.status, 1u);
    }
}

template <int K, int G, bool CG>
__device__ __forceinline__ void vdiff_node(const DTopo &tp, const B32View &B, int n, int lane, int nzmin, int nzmax,
                                           VdiffWarp &W) {
    VdiffLane<K> V;
    float A = 1.f, Ad = 1.f;
#pragma unroll
    for (int t = 0; t < K; t++) {
        const int nz = nzmin + lane * K + t;
        V.ok[t] = nz <= nzmax - 1;
        const float4 fz = V.ok[t] ? W.fac[nz] : make_float4(0.f, 0.f, 0.f, 0.f);
        V.a[t] = fz.x;
        V.c[t] = fz.y;
        V.inv[t] = fz.z;
        // levels past the column's end are identity maps
        V.A[t] = V.ok[t] ? -(fz.x * fz.z) : 1.f;
        V.Ad[t] = V.ok[t] ? -fz.w : 1.f;
        A *= V.A[t];
        Ad *= V.Ad[t];
    }
    // partial products of the lane maps at each scan step
#pragma unroll
    for (int s = 0, off = 1; s < kScan; s++, off <<= 1) {
        W.af[s][lane] = lane >= off ? A : 0.f;
        W.ab[s][lane] = lane + off < 32 ? Ad : 0.f;
        const float Ap = __shfl_up_sync(kFull, A, off), An = __shfl_down_sync(kFull, Ad, off);
        if (lane >= off) A *= Ap;
        if (lane + off < 32) Ad *= An;
    }
    __syncwarp();
    unsigned long long todo = (B.ivd & ~B.wimpl) & (B.ng >= 64 ? ~0ull : ((1ull << B.ng) - 1));
    // (loading the next group's column during the current solve measured slower after the
    // update: the extra registers spill)
    while (todo) {
        const int gq = __ffsll((long long)todo) - 1;
        todo &= todo - 1;
        VdiffCol<K, G> x;
        vdiff_load<K, G, CG>(tp, B, n, lane, nzmin, gq, V, x);
        vdiff_group<K, G>(tp, B, n, lane, nzmin, nzmax, gq, V, W, x);
    }
}

template <int G, bool CG = false>
__device__ __forceinline__ void vdiff_unit(const DTopo &tp, const B32View &B, const VFactors &vf, int n,
                                           VdiffWarp &W) {
    const int lane = threadIdx.x & 31;
    if (n >= tp.N2) return;
    const int L1 = tp.L1;
    const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
    const int K = (nzmax - nzmin + 31) / 32;
    __syncwarp();  // the previous node's reads of W are done
    for (int nz = nzmin + lane; nz <= nzmax - 1; nz += 32) {
        const int i = n * L1 + nz - 1;
        W.fac[nz] = make_float4(vf.a[i], vf.c[i], vf.inv[i], vf.cp[i]);
    }
    __syncwarp();
    switch (K) {
        case 1: vdiff_node<1, G, CG>(tp, B, n, lane, nzmin, nzmax, W); break;
        case 2: vdiff_node<2, G, CG>(tp, B, n, lane, nzmin, nzmax, W); break;
        case 3: vdiff_node<3, G, CG>(tp, B, n, lane, nzmin, nzmax, W); break;
        default: vdiff_node<4, G, CG>(tp, B, n, lane, nzmin, nzmax, W); break;
    }
}

// ---------------------------------------------------------------------------
// k32_update: limited update, T*
// ---------------------------------------------------------------------------
// Bound by the latency of its gathers, 440 bytes per layer and group of 4 (R+ and R- of six neighbours,
// six edge fluxes): issue 38 % with 5.9 warps a scheduler at 80 registers, L2 at 30 % of its rate, DRAM
// at 42 % (12 tracers, 70 layers).  Sphere of 7 subdivisions, T and S, with the diffusion: 331 -> 231 us
// against a warp per node; 24 tracers on the sphere of 8: 7.2 -> 7.2 ms.
template <int G>
using UpdateBuf = Vec<G>[2][kNT];  // [buffer][thread]: limited interface fluxes

template <int G>
__device__ __forceinline__ void update_tile(const DTopo &tp, const DGeom<float> &g, const B32View &B, float dt,
                                            const NodeTile &S, UpdateBuf<G> &X) {
    constexpr int kUU = MinB<G>::uu;
    const TileLane k(tp, S);
    const int x = threadIdx.x, i = k.i, iv = k.iv, nz = k.nz, deg = S.deg[k.j];
    const bool top = nz == k.nzmin;
    const float sdt = k.on ? qdiv(dt, g.areasvol[iv] * g.hnode_new[i]) : 0.f;
#pragma unroll 1
    for (int gq = 0; gq < B.ng; gq++) {
        const bool fct = (B.fct >> gq) & 1ull, dif = (B.diff >> gq) & 1ull;
        const bool lf = k.on && fct;
        const float *__restrict__ Rp = grp<G>(B.Rp, gq, B.sN);
        const float *__restrict__ Rm = grp<G>(B.Rm, gq, B.sN);
        const float *__restrict__ ADh = grp<G>(B.ADh, gq, B.sE);
        float *__restrict__ Tn = grp<G>(B.Tnew, gq, B.sN);
        const Vec<G> lo = vldc<G>(k.on, grp<G>(B.LO, gq, B.sN), i);
        const Vec<G> f0 = vldc<G>(k.on, grp<G>(B.ADv, gq, B.sNI), iv);
        const Vec<G> r0p = lf ? vld<G>(Rp, i) : vfill<G>(1.f);
        const Vec<G> r0m = lf ? vld<G>(Rm, i) : vfill<G>(1.f);
        const Vec<G> rup = lf && !top ? vld<G>(Rp, i - 1) : vfill<G>(1.f);
        const Vec<G> rum = lf && !top ? vld<G>(Rm, i - 1) : vfill<G>(1.f);
        const Vec<G> tbp = vldc<G>(lf && kFctClamp, grp<G>(B.Bp, gq, B.sN), i);
        const Vec<G> tbm = vldc<G>(lf && kFctClamp, grp<G>(B.Bm, gq, B.sN), i);
        // the diffusion increment k32_diff parked in Tnew (the limiter acts on advection only)
        const Vec<G> dd = vldc<G>(k.on && dif, Tn, i);
        Vec<G> hs = vfill<G>(0.f);
        // horizontal limiting (oce_adv_tra_fct.F90:468-500) seen from the node: with G the
        // antidiffusive flux into the node and m the other end, G >= 0 takes
        // min(R+(n), R-(m)), G < 0 takes min(R-(n), R+(m))
#pragma unroll 1
        for (int u0 = 0; u0 < S.degmax; u0 += kUU) {
            Vec<G> xe[kUU], rmp[kUU], rmm[kUU];
#pragma unroll
            for (int u = 0; u < kUU; u++) {
                const int4 q = S.slot[k.j][u0 + u];
                const bool ok = k.on && u0 + u < deg && slot_wet(q, nz);
                xe[u] = vldc<G>(ok, ADh, q.y + nz - 1);
                rmp[u] = vldc<G>(ok && fct, Rp, q.x + nz - 1);
                rmm[u] = vldc<G>(ok && fct, Rm, q.x + nz - 1);
            }
#pragma unroll
            for (int u = 0; u < kUU; u++) {
                const bool ow = S.slot[k.j][u0 + u].w != 0;
#pragma unroll
                for (int c = 0; c < G; c++) {
                    float Gf = ow ? xe[u].c[c] : -xe[u].c[c];
                    if (fct) Gf *= Gf >= 0.f ? fminf(r0p.c[c], rmm[u].c[c]) : fminf(r0m.c[c], rmp[u].c[c]);
                    hs.c[c] += Gf;
                }
            }
        }
        // vertical limiting (oce_adv_tra_fct.F90:425-456): interface nz by R of layers nz-1 and nz;
        // the next interface is the next thread's
        Vec<G> fz = f0;
        if (fct) {
#pragma unroll
            for (int c = 0; c < G; c++) {
                if (top) fz.c[c] *= fz.c[c] >= 0.f ? r0p.c[c] : r0m.c[c];
                else fz.c[c] *= fz.c[c] >= 0.f ? fminf(rum.c[c], r0p.c[c]) : fminf(rup.c[c], r0m.c[c]);
            }
        }
        Vec<G>(&xf)[kNT] = X[gq & 1];
        xf[x] = fz;
        __syncthreads();
        if (!k.on) continue;
        const Vec<G> f1 = nz == k.nzmax - 1 ? vfill<G>(0.f) : xf[x + 1];
        Vec<G> out;
        bool fin = true;
#pragma unroll
        for (int c = 0; c < G; c++) {
            // del_ttf = (LO hnode_new - T hnode) + limited flux divergence dt / areasvol;
            // T* = T + (del_ttf + T (hnode - hnode_new)) / hnode_new = LO + fluxes dt / areasvol / hnode_new
            // (oce_adv_tra_driver.F90:535-620, oce_ale_tracer.F90:319-321, 743-754)
            float val = lo.c[c] + ((fz.c[c] - f1.c[c]) + hs.c[c]) * sdt;
            if (kFctClamp && fct) {
                const float vc = fminf(fmaxf(val, tbm.c[c]), tbp.c[c]);
                // a clamp beyond round-off means the limiter itself failed
                if (fabsf(vc - val) > 1e-5f * (tbp.c[c] - tbm.c[c]) + 1e-6f * fabsf(vc)) atomicOr(B.status, 2u);
                val = vc;
            }
            if (dif) val += dd.c[c];
            out.c[c] = val;
            fin = fin && isfinite(val);
        }
        vst<G>(Tn, i, out);
        if (!fin) atomicOr(B.status, 1u);
    }
}

// the implicit vertical diffusion of the tile's columns, a warp per column (T* of the whole tile
// is written before the block's barrier)
template <int G>
__device__ __forceinline__ void update_tile_vdiff(const DTopo &tp, const B32View &B, const VFactors &vf,
                                                  const NodeTile &S, VdiffWarp *W) {
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    for (int j = warp; j < S.cnt; j += kNT / 32) vdiff_unit<G, true>(tp, B, vf, S.n0 + j, W[warp]);
}

// VD: with the implicit vertical diffusion of the groups in ivd & ~wimpl as the epilogue of each
// tile (factors vf)
template <int G, bool VD>
__global__ void __launch_bounds__(kNT, MinB<G>::update)
k32_update(DTopo tp, DGeom<float> g, B32View B, float dt, VFactors vf) {
    __shared__ NodeTile S;
    __shared__ union {
        UpdateBuf<G> X;
        VdiffWarp W[VD ? kNT / 32 : 1];
    } U;
    FOR_NODE_TILES(ti, tp.n_nt) {
        node_tile_load(tp, ti, S);
        update_tile<G>(tp, g, B, dt, S, U.X);
        if (VD) update_tile_vdiff<G>(tp, B, vf, S, U.W);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// k32_vppm: adv_tra_vert_ppm (oce_adv_tra_ver.F90:438-631) on the AB values of the groups
// in the ppm mask, minus the LO flux, into ADv.  A warp per node over chunks of 27 interfaces
// with 3 levels of halo above and 2 below: the interface value tv(k) needs the layers
// k-2..k+1, the flux of interface nz the parabola of layer nz or nz-1.
// ---------------------------------------------------------------------------
template <int G>
__device__ __forceinline__ void vppm_node(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f,
                                          const B32View &B, float dt, int n, int lane) {
    using C = Chunk<3, 2>;
    const int L1 = tp.L1, nl = tp.nl;
    const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
    const int nch = C::count(nzmin, nzmax);
    for (int ch = 0; ch < nch; ch++) {
        const C k(nzmin, nzmax, ch, lane);
        const int nz = k.nz;
        const int i = n * L1 + nz - 1, iv = n * nl + nz - 1;
        float hn0 = 0.f, ho0 = 0.f, ar0 = 0.f, w0 = 0.f, we0 = 0.f;
        if (k.lvl) {
            hn0 = g.hnode_new[i];
            ho0 = g.hnode[i];
            ar0 = g.area[iv];
            w0 = f.w[iv];
            we0 = f.we[iv];
        }
        const float hm1 = sh_up(hn0, 1), hm2 = sh_up(hn0, 2), hp1 = sh_dn(hn0, 1);
        const float hom1 = sh_up(ho0, 1);
        unsigned long long todo = B.ppm & (B.ng >= 64 ? ~0ull : ((1ull << B.ng) - 1));
        while (todo) {
            const int gq = __ffsll((long long)todo) - 1;
            todo &= todo - 1;
            const bool lim = (B.fct >> gq) & 1ull;
            const Vec<G> Tv = vldc<G>(k.lvl, grp<G>(B.T, gq, B.sN), i);
            const Vec<G> o1 = vldc<G>(k.lvl, grp<G>(B.O1, gq, B.sN), i);
            const Vec<G> o2 = vldc<G>(k.lvl && B.ab == 3, grp<G>(B.O2, gq, B.sN), i);
            Vec<G> out;
#pragma unroll
            for (int c = 0; c < G; c++) {
                const float Tn = Tv.c[c];
                const float tab = Tn + (k.lvl ? ab_delta(B.ab, Tn, o1.c[c], o2.c[c]) : 0.f);
                const float tm1 = sh_up(tab, 1), tm2 = sh_up(tab, 2), tp1 = sh_dn(tab, 1);
                const float Tu = sh_up(Tn, 1);
                // tv(nz) (:488-562): centred next to the ends, the non-uniform PPM value between
                float tv;
                if (nz == nzmax) {
                    tv = tm1;
                } else if (nz == nzmin) {
                    tv = tab;
                } else if (nz == nzmax - 1 || nz == nzmin + 1) {
                    tv = 0.5f * (tm1 + tab);
                } else {
                    // layer j = nz-1: dzjm1 = h(nz-2), dzj = h(nz-1), dzjp1 = h(nz), dzjp2 = h(nz+1)
                    const float a0 = hm2, a1 = hm1, a2 = hn0, a3 = hp1;
                    const float d10 = tab - tm1, d0m = tm1 - tm2, d21 = tp1 - tab;
                    float dj = a1 / (a0 + a1 + a2) *
                               ((2.f * a0 + a1) / (a2 + a1) * d10 + (a1 + 2.f * a2) / (a0 + a1) * d0m);
                    float dj1 = a2 / (a1 + a2 + a3) *
                                ((2.f * a1 + a2) / (a3 + a2) * d21 + (a2 + 2.f * a3) / (a1 + a2) * d10);
                    dj = d10 * d0m > 0.f ? copysignf(fminf(fminf(fabsf(dj), 2.f * fabsf(d10)), 2.f * fabsf(d0m)), dj)
                                         : 0.f;
                    dj1 = d21 * d10 > 0.f
                              ? copysignf(fminf(fminf(fabsf(dj1), 2.f * fabsf(d21)), 2.f * fabsf(d10)), dj1)
                              : 0.f;
                    tv = tm1 + a1 / (a1 + a2) * d10 +
                         1.f / (a0 + a1 + a2 + a3) *
                             ((2.f * a2 * a1) / (a1 + a2) * ((a0 + a1) / (2.f * a1 + a2) - (a3 + a2) / (2.f * a2 + a1)) *
                                  d10 -
                              a1 * (a0 + a1) / (2.f * a1 + a2) * dj1 + a2 * (a2 + a3) / (a1 + 2.f * a2) * dj);
                }
                const float tvu = sh_up(tv, 1), tvd = sh_dn(tv, 1);
                const float pw = lim ? w0 : we0;
                float Cf = 0.f;
                if (nz == nzmin) {
                    Cf = -(tv * pw * ar0);
                } else if (pw > 0.f || pw < 0.f) {
                    // the parabola of the upwind layer (:564-620)
                    const bool top = pw > 0.f;
                    float aL = top ? tv : tvu, aR = top ? tvd : tv;
                    const float tt = top ? tab : tm1, dz = top ? ho0 : hom1;
                    if ((aR - tt) * (tt - aL) <= 0.f) aL = aR = tt;
                    if ((aR - aL) * (tt - 0.5f * (aL + aR)) > (aR - aL) * (aR - aL) * (1.f / 6.f)) aL = 3.f * tt - 2.f * aR;
                    if ((aR - aL) * (tt - 0.5f * (aR + aL)) < -((aR - aL) * (aR - aL) * (1.f / 6.f)))
                        aR = 3.f * tt - 2.f * aL;
                    const float aj = 6.f * (tt - 0.5f * (aL + aR));
                    const float x = fminf(fabsf(pw) * dt / dz, 1.f);
                    const float v = top ? -aL - 0.5f * x * (aR - aL + (1.f - (2.f / 3.f) * x) * aj)
                                        : -aR + 0.5f * x * (aR - aL - (1.f - (2.f / 3.f) * x) * aj);
                    Cf = v * ar0 * pw;
                }
                // minus the upwind LO flux: of w_e, or of the full w for FCT with the split velocity
                const float wl = (lim && f.wsplit) ? w0 : we0;
                float fl;
                if (nz == nzmin) {
                    fl = -(wl * Tn * ar0);
                } else {
                    const float aw = fabsf(wl);
                    fl = -(0.5f * (Tn * (wl + aw) + Tu * (wl - aw)) * ar0);
                }
                out.c[c] = Cf - fl;
            }
            if (k.out) vst<G>(grp<G>(B.ADv, gq, B.sNI), iv, out);
        }
    }
}

template <int G>
__global__ void __launch_bounds__(kTB) k32_vppm(DTopo tp, DGeom<float> g, DForcing<float> f, B32View B, float dt) {
    FOR_WARP_UNITS(n, tp.N2) vppm_node<G>(tp, g, f, B, dt, n, threadIdx.x & 31);
}

// ---------------------------------------------------------------------------
// split vertical velocity, FP32 form: adv_tra_vert_impl by w_i on the LO values of the FCT
// groups (oce_adv_tra_ver.F90:90-240), and the implicit vertical diffusion with the w_i
// terms for the groups without the limiter (oce_ale_tracer.F90:907-1435, do_wimpl).  One
// thread per column, FP64 arithmetic; scratch holds Z_n, cp and tp level-major.
// ---------------------------------------------------------------------------
// one slot's column of a group field (1-based levels)
struct SlotCol {
    float *p;
    int G;
    __device__ __forceinline__ float &operator[](int nz) const { return p[(size_t)(nz - 1) * G]; }
};

__device__ __forceinline__ void lo_impl_slot(const float *hn, const float *ar, const float *av, const float *wi,
                                             double dt, double *cps, double *tps, size_t N2, int n, int nzmin,
                                             int nzmax, SlotCol Tc) {
#define CP(k) cps[(size_t)(k) * N2 + n]
#define TP(k) tps[(size_t)(k) * N2 + n]
    int nz = nzmin;
    double v = dt * ar[nz] / av[nz];
    double b = (double)hn[nz] + (double)wi[nz] * v;
    v = dt * ar[nz + 1] / av[nz];
    b = b - fmin(0.0, (double)wi[nz + 1]) * v;
    double c = -(fmax(0.0, (double)wi[nz + 1]) * v);
    double T0 = Tc[nz], Tp1 = Tc[nz + 1], Tm;
    double rhs = -((b - hn[nz]) * T0) - c * Tp1;
    double cp = c / b, tpv = rhs / b;
    CP(nz) = cp;
    TP(nz) = tpv;
    for (nz = nzmin + 1; nz <= nzmax - 1; nz++) {
        v = dt * ar[nz] / av[nz];
        const double a = fmin(0.0, (double)wi[nz]) * v;
        b = (double)hn[nz] + fmax(0.0, (double)wi[nz]) * v;
        c = 0.0;
        if (nz <= nzmax - 2) {
            v = dt * ar[nz + 1] / av[nz];
            b = b - fmin(0.0, (double)wi[nz + 1]) * v;
            c = -(fmax(0.0, (double)wi[nz + 1]) * v);
        }
        Tm = T0;
        T0 = Tp1;
        Tp1 = nz <= nzmax - 2 ? (double)Tc[nz + 1] : 0.0;
        rhs = -(a * Tm) - (b - hn[nz]) * T0 - c * Tp1;
        const double m = b - cp * a;
        cp = c / m;
        tpv = (rhs - tpv * a) / m;
        CP(nz) = cp;
        TP(nz) = tpv;
    }
    double x = tpv;
    Tc[nzmax - 1] = (float)(Tc[nzmax - 1] + x);
    for (nz = nzmax - 2; nz >= nzmin; nz--) {
        x = TP(nz) - CP(nz) * x;
        Tc[nz] = (float)(Tc[nz] + x);
    }
#undef CP
#undef TP
}

template <int G>
__device__ __forceinline__ void lo_impl_column(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f,
                                               const B32View &B, double dt, double *scratch, int n) {
    const int L1 = tp.L1, nl = tp.nl;
    const size_t N2 = tp.N2;
    double *cps = scratch, *tps = scratch + (size_t)(L1 + 1) * N2;
    const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
    const float *hn = g.hnode_new + (size_t)n * L1 - 1;
    const float *ar = g.area + (size_t)n * nl - 1, *av = g.areasvol + (size_t)n * nl - 1;
    const float *wi = f.wi + (size_t)n * nl - 1;
    unsigned long long todo = B.fct & (B.ng >= 64 ? ~0ull : ((1ull << B.ng) - 1));
    while (todo) {
        const int gq = __ffsll((long long)todo) - 1;
        todo &= todo - 1;
        float *base = grp<G>(B.LO, gq, B.sN) + (size_t)n * L1 * G;
        for (int c = 0; c < G; c++)
            lo_impl_slot(hn, ar, av, wi, dt, cps, tps, N2, n, nzmin, nzmax, SlotCol{base + c, G});
    }
}

template <int G>
__device__ __forceinline__ void vdiff_w_column(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f,
                                               const B32View &B, double dt, double *scratch, int n) {
    const int L1 = tp.L1, nl = tp.nl;
    const size_t N2 = tp.N2;
    double *Zs = scratch, *cps = scratch + (size_t)(L1 + 1) * N2, *tps = cps + (size_t)(L1 + 1) * N2;
#define ZN(k) Zs[(size_t)(k) * N2 + n]
#define CP(k) cps[(size_t)(k) * N2 + n]
#define TP(k) tps[(size_t)(k) * N2 + n]
    const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
    const float *hn = g.hnode_new + (size_t)n * L1 - 1;
    const float *ar = g.area + (size_t)n * nl - 1, *av = g.areasvol + (size_t)n * nl - 1;
    const float *kv = f.Kv + (size_t)n * nl - 1, *wi = f.wi + (size_t)n * nl - 1;
    double zb = g.zbar_n_bot[n];
    ZN(nzmax - 1) = zb + (double)hn[nzmax - 1] / 2.0;
    for (int nz = nzmax - 1; nz >= nzmin + 1; nz--) {
        zb = zb + (double)hn[nz];
        ZN(nz - 1) = zb + (double)hn[nz - 1] / 2.0;
    }
    unsigned long long todo = B.wimpl & (B.ng >= 64 ? ~0ull : ((1ull << B.ng) - 1));
    while (todo) {
        const int gq = __ffsll((long long)todo) - 1;
        todo &= todo - 1;
        float *base = grp<G>(B.Tnew, gq, B.sN) + (size_t)n * L1 * G;
        for (int cs = 0; cs < G; cs++) {
            const SlotCol Tc{base + cs, G};
            const double bc = B.fsurf ? (double)B.fsurf[((size_t)gq * N2 + n) * G + cs] : 0.0;
            int nz = nzmin;
            double zinv2 = 1.0 / (ZN(nz) - ZN(nz + 1)), zinv1;
            double c = -((double)kv[nz + 1] * zinv2 * dt * ar[nz + 1] / av[nz]);
            double b = -c + hn[nz];
            double v = dt * ((double)ar[nz] / av[nz]);
            b = b + (double)wi[nz] * v;
            v = dt * ar[nz + 1] / av[nz];
            b = b - fmin(0.0, (double)wi[nz + 1]) * v;
            c = c - fmax(0.0, (double)wi[nz + 1]) * v;
            double T0 = Tc[nz], Tp1 = Tc[nz + 1], Tm;
            double rhs = -((b - hn[nz]) * T0) - c * Tp1 + bc;
            double cp = c / b, tpv = rhs / b;
            CP(nz) = cp;
            TP(nz) = tpv;
            zinv1 = zinv2;
            for (nz = nzmin + 1; nz <= nzmax - 1; nz++) {
                const bool bot = nz == nzmax - 1;
                double a = -((double)kv[nz] * zinv1 * dt * ((double)ar[nz] / av[nz]));
                c = 0.0;
                if (!bot) {
                    zinv2 = 1.0 / (ZN(nz) - ZN(nz + 1));
                    c = -((double)kv[nz + 1] * zinv2 * dt * ar[nz + 1] / av[nz]);
                }
                b = -a - c + hn[nz];
                zinv1 = zinv2;
                v = dt * ((double)ar[nz] / av[nz]);
                a = a + fmin(0.0, (double)wi[nz]) * v;
                b = b + fmax(0.0, (double)wi[nz]) * v;
                if (!bot) {
                    v = dt * ar[nz + 1] / av[nz];
                    b = b - fmin(0.0, (double)wi[nz + 1]) * v;
                    c = c - fmax(0.0, (double)wi[nz + 1]) * v;
                }
                Tm = T0;
                T0 = Tp1;
                Tp1 = bot ? 0.0 : (double)Tc[nz + 1];
                rhs = -(a * Tm) - (b - hn[nz]) * T0 - c * Tp1;
                const double m = b - cp * a;
                cp = c / m;
                tpv = (rhs - tpv * a) / m;
                CP(nz) = cp;
                TP(nz) = tpv;
            }
            double x = tpv;
            Tc[nzmax - 1] = (float)(Tc[nzmax - 1] + x);
            for (nz = nzmax - 2; nz >= nzmin; nz--) {
                x = TP(nz) - CP(nz) * x;
                Tc[nz] = (float)(Tc[nz] + x);
            }
        }
    }
#undef ZN
#undef CP
#undef TP
}

template <int G>
__global__ void __launch_bounds__(128) k32_lo_impl(DTopo tp, DGeom<float> g, DForcing<float> f, B32View B, double dt,
                                                   double *scratch) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < tp.N2) lo_impl_column<G>(tp, g, f, B, dt, scratch, n);
}
template <int G>
__global__ void __launch_bounds__(128) k32_vdiff_w(DTopo tp, DGeom<float> g, DForcing<float> f, B32View B, double dt,
                                                   double *scratch) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < tp.N2) vdiff_w_column<G>(tp, g, f, B, dt, scratch, n);
}

// ---------------------------------------------------------------------------
// diffusion of diff_tracers_ale (oce_ale_tracer.F90:560-772) in the FP32 form
// ---------------------------------------------------------------------------
// k32_hdiff: diff_part_hor_redi (:1526-1689) flux c of every edge-layer from the element
// gradients of the current values: segments A/D (element 1), B/E (element 2), C (both); with
// Redi the gradient gains S_xy Tz: Tz at each edge node the layer mean of the vertical gradient
// (tracer_gradient_z, 0 at the column's top and bottom interfaces), S_xy Tz = (Tz(n1) S(n1)
// + Tz(n2) S(n2)) / 2 (:1583-1595)
//
// A tile of edges, as k32_ho.  The element gradients, projected on the edge's cross vectors, are
// weights of the differences to T(edges(1,e)) formed once per edge: 4 + 4 gathers (the elements'
// nodes, the layers next to both ends) per edge-layer and group where gradients of two elements and
// vertical differences took 12, and a third of the arithmetic.  Latency of the gathers bounds it: 1.10
// -> 0.39 ms on the sphere of 7 subdivisions, 47 layers, 7 tracers with Redi.
//
// That holds where an edge's elements contain both its ends and an element's weights add up to zero.  OWN:
// meshes whose edge_tri names some other element or whose weights do not (not diff_by_edges): each
// element's gradient from its own three nodes, 6 + 6 gathers.
struct EdgeD {
    int ia, ib, xa, xb, l1, l2;          // first entries of the columns of both ends, the elements' third nodes, the elements
    int nl1, ul1, nl2, ul2;              // levels of the elements
    int top1, bot1, top2, bot2;          // ulevels / nlevels of the end nodes
    float dX1, dY1, dX2, dY2;
    float w1b, w1x, w2b, w2x, w3b, w3x, w3y;  // projected gradients as weights of T(node) - T(edges(1,e))
};

// gradient_sca of element el at node n: d/dx and d/dy weights
__device__ __forceinline__ float2 gs_at(const DTopo &tp, const DGeom<float> &g, int el, int n) {
    const int k = tp.t_n[3 * el] == n ? 0 : tp.t_n[3 * el + 1] == n ? 1 : 2;
    const float *gs = g.gs + 6 * (size_t)el;
    return make_float2(gs[k], gs[3 + k]);
}

// tile ti of `tile` edges
template <int G, bool OWN>
__device__ __forceinline__ void hdiff_tile(const DTopo &tp, const DGeom<float> &g, const B32View &B, int ti, int tile,
                                           Tile &S, EdgeD *Ed) {
    const int L1 = tp.L1, e0 = ti * tile;
    if (!B.Ki) return;
    if (threadIdx.x < 32) {
        const int j = threadIdx.x, e = e0 + j;
        const bool in = j < tile && e < tp.E2;
        if (in) {
            EdgeD &E = Ed[j];
            const int n1 = tp.e_n1[e], n2 = tp.e_n2[e], el1 = tp.e_t1[e], el2 = tp.e_t2[e];
            const float4 d = reinterpret_cast<const float4 *>(g.ecd)[e];
            E.ia = n1 * L1;
            E.ib = n2 * L1;
            E.l1 = el1 * L1;
            E.nl1 = tp.t_nlev[el1] - 1;
            E.ul1 = tp.t_ulev[el1];
            E.dX1 = d.x;
            E.dY1 = d.y;
            E.l2 = 0;
            E.nl2 = E.ul2 = 0;
            E.dX2 = E.dY2 = 0.f;
            if (el2 >= 0) {
                E.l2 = el2 * L1;
                E.nl2 = tp.t_nlev[el2] - 1;
                E.ul2 = tp.t_ulev[el2];
                E.dX2 = d.z;
                E.dY2 = d.w;
            }
            if (!OWN) {
                auto third = [&](int el) { return tp.t_n[3 * el] + tp.t_n[3 * el + 1] + tp.t_n[3 * el + 2] - n1 - n2; };
                const int x1 = third(el1);
                const float2 b1 = gs_at(tp, g, el1, n2), c1 = gs_at(tp, g, el1, x1);
                E.xa = x1 * L1;
                E.w1b = d.y * b1.x - d.x * b1.y;
                E.w1x = d.y * c1.x - d.x * c1.y;
                E.xb = 0;
                E.w2b = E.w2x = E.w3b = E.w3x = E.w3y = 0.f;
                if (el2 >= 0) {
                    const int x2 = third(el2);
                    const float2 b2 = gs_at(tp, g, el2, n2), c2 = gs_at(tp, g, el2, x2);
                    const float X = d.z - d.x, Y = d.w - d.y;
                    E.xb = x2 * L1;
                    E.w2b = d.z * b2.y - d.w * b2.x;
                    E.w2x = d.z * c2.y - d.w * c2.x;
                    E.w3b = 0.5f * (X * (b1.y + b2.y) - Y * (b1.x + b2.x));
                    E.w3x = 0.5f * (X * c1.y - Y * c1.x);
                    E.w3y = 0.5f * (X * c2.y - Y * c2.x);
                }
            }
            E.top1 = tp.n_ulev[n1];
            E.bot1 = tp.n_nlev[n1];
            E.top2 = tp.n_ulev[n2];
            E.bot2 = tp.n_nlev[n2];
        }
        S.fill(j, in ? tp.e_lo[e] : 1, in ? tp.e_hi[e] - tp.e_lo[e] + 1 : 0);
    }
    __syncthreads();
    const bool redi = B.slope != nullptr;
    for (int i = threadIdx.x; i < S.total; i += kTileThreads) {
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j], k = nz - 1;
        const EdgeD &E = Ed[j];
        const int i1 = E.ia + k, i2 = E.ib + k;
        const int nl12 = min(E.nl1, E.nl2), ul12 = max(E.ul1, E.ul2);
        int seg = 0;
        if (nz >= E.ul1 && nz <= ul12 - 1) seg = 1;
        else if (E.ul2 > 0 && nz >= E.ul2 && nz <= ul12 - 1) seg = 2;
        else if (nz >= ul12 && nz <= nl12) seg = 3;
        else if (nz >= nl12 + 1 && nz <= E.nl1) seg = 1;
        else if (nz >= nl12 + 1 && nz <= E.nl2) seg = 2;
        const bool u1 = seg & 1, u2 = seg & 2;
        // the flux is Kh h (weights . (T - T1) + dY S_x Tz - dX S_y Tz)
        const float h = !seg ? 0.f : 0.5f * (B.Ki[i1] + B.Ki[i2]) *
                        (seg == 3 ? 0.5f * (g.helem[E.l1 + k] + g.helem[E.l2 + k]) : g.helem[(u2 ? E.l2 : E.l1) + k]);
        const float wb = OWN ? 0.f : h * (seg == 3 ? E.w3b : u1 ? E.w1b : u2 ? E.w2b : 0.f);
        const float wx = u1 && !OWN ? h * (seg == 3 ? E.w3x : E.w1x) : 0.f,
                    wy = u2 && !OWN ? h * (seg == 3 ? E.w3y : E.w2x) : 0.f;
        // Redi: weights of the differences to the layers above and below at both ends (0 at the
        // columns' ends)
        float a1 = 0.f, b1 = 0.f, a2 = 0.f, b2 = 0.f;
        if (redi && seg) {
            const float dX = (u1 ? E.dX1 : 0.f) - (u2 ? E.dX2 : 0.f), dY = (u1 ? E.dY1 : 0.f) - (u2 ? E.dY2 : 0.f);
            const float *s1 = B.slope + 3 * (size_t)i1, *s2 = B.slope + 3 * (size_t)i2;
            const float q1 = 0.5f * h * (dY * s1[0] - dX * s1[1]), q2 = 0.5f * h * (dY * s2[0] - dX * s2[1]);
            const float h1 = g.hnode[i1], h2 = g.hnode[i2];
            if (nz > E.top1) a1 = q1 / (g.hnode[i1 - 1] + h1);
            if (nz + 1 < E.bot1) b1 = q1 / (h1 + g.hnode[i1 + 1]);
            if (nz > E.top2) a2 = q2 / (g.hnode[i2 - 1] + h2);
            if (nz + 1 < E.bot2) b2 = q2 / (h2 + g.hnode[i2 + 1]);
        }
        const bool t1 = redi && nz > E.top1, d1 = redi && nz + 1 < E.bot1, t2 = redi && nz > E.top2,
                   d2 = redi && nz + 1 < E.bot2;
#pragma unroll 1
        for (int gq = 0; gq < B.ng; gq++) {
            const float *__restrict__ T = grp<G>(B.T, gq, B.sN);
            const Vec<G> T1 = vld<G>(T, i1), T2 = vld<G>(T, i2);
            const Vec<G> Tx = vldc<G>(u1 && !OWN, T, E.xa + k), Ty = vldc<G>(u2 && !OWN, T, E.xb + k);
            const Vec<G> m1 = vldc<G>(t1, T, i1 - 1), p1 = vldc<G>(d1, T, i1 + 1);
            const Vec<G> m2 = vldc<G>(t2, T, i2 - 1), p2 = vldc<G>(d2, T, i2 + 1);
            Vec<G> out;
            if (OWN) {
                out = vfill<G>(0.f);
#pragma unroll 1
                for (int q = 0; q < 6; q++) {
                    if (!(q < 3 ? u1 : u2)) continue;
                    const int el = (q < 3 ? E.l1 : E.l2) / L1, v = q < 3 ? q : q - 3;
                    // weights of the element's d/dx and d/dy: the cross vectors of its segment, the mean of
                    // both elements' gradients in segment C
                    const float cx = seg == 3 ? 0.5f * (E.dY1 - E.dY2) : q < 3 ? E.dY1 : -E.dY2;
                    const float cy = seg == 3 ? 0.5f * (E.dX2 - E.dX1) : q < 3 ? -E.dX1 : E.dX2;
                    const float w = h * (cx * g.gs[6 * (size_t)el + v] + cy * g.gs[6 * (size_t)el + 3 + v]);
                    const Vec<G> t = vld<G>(T, tp.t_n[3 * el + v] * L1 + k);
#pragma unroll
                    for (int c = 0; c < G; c++) out.c[c] += w * (tp.grad_zero ? t.c[c] - T1.c[c] : t.c[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < G; c++) {
                const float x1 = T1.c[c], x2 = T2.c[c];
                float f = OWN ? out.c[c] : wb * (x2 - x1);
                if (!OWN && u1) f += wx * (Tx.c[c] - x1);
                if (!OWN && u2) f += wy * (Ty.c[c] - x1);
                if (redi) {
                    f += a1 * (m1.c[c] - x1) + b1 * (x1 - p1.c[c]);
                    f += a2 * (m2.c[c] - x2) + b2 * (x2 - p2.c[c]);
                }
                out.c[c] = f;
            }
            vst<G>(grp<G>(B.HD, gq, B.sE), (e0 + j) * L1 + k, out);
        }
    }
}

template <int G, bool OWN>
__global__ void __launch_bounds__(kTileThreads, MinB<G>::hdiff) k32_hdiff(DTopo tp, DGeom<float> g, B32View B, int tile) {
    __shared__ Tile S;
    __shared__ EdgeD Ed[kTileMax];
    hdiff_tile<G, OWN>(tp, g, B, blockIdx.x, tile, S, Ed);
}

// k32_diff: the diffusion increment to T* of every group in the diff mask, parked in Tnew:
// (sum of the node's edge fluxes +- c) dt / (areasvol hnode_new) and, without implicit vertical
// diffusion, diff_ver_part_expl_ale (:841-902): vd(ul) = surface flux, vd(nz) = Kv (T(nz-1)
// - T(nz)) / (Z(nz-1) - Z(nz)) area, increment (vd(nz) - vd(nz+1)) / (zbar(nz) - zbar(nz+1))
// dt / (areasvol hnode_new).  With Redi, diff_ver_part_redi_expl (:1439-1518): the node
// gradient g(nz) = sum over the node's elements wet at nz of grad T elem_area / 3 / areasvol,
// p = S_xy . g, interface flux vd(nz) = (h(nz-1) p(nz-1) Ki(nz-1) + h(nz) p(nz) Ki(nz)) /
// (h(nz-1) + h(nz)) area(nz) with h = hnode (the reference's depth differences z(nz-1) -
// zbar(nz) = h(nz-1)/2 etc. in exact arithmetic), increment (vd(nz) - vd(nz+1)) dt / (areasvol
// hnode_new)
//
// A tile of nodes, as k32_lo_ad; the vertical neighbours of S_xy . g pass through shared memory.
// With the weights below, 6 gathers of T per group instead of 18: 0.68 -> 0.41 ms on the sphere of 7
// subdivisions, 47 layers, 7 tracers with Redi.
//
// Redi: the node gradient's weights per edge slot (diff_by_edges; else the elements themselves).  The
// gradients of the node's elements sum over
// the neighbours: with weights of a triangle that add up to zero, sum_el ea grad T = sum_m w_m
// (T_m - T_n), where w_m joins the node's two elements at edge (n, m), each where it is wet.
struct DiffSlots {
    float4 w[kNodeTileNodes][kSlots];  // elem_area * gradient_sca at m of the edge's two elements (x, y; x, y)
    int2 r[kNodeTileNodes][kSlots];    // their levels lo | hi << 16 (0: no element)
};
__device__ __forceinline__ void diff_slots_load(const DTopo &tp, const DGeom<float> &g, const NodeTile &S,
                                                DiffSlots &D) {
    for (int s = threadIdx.x; s < S.cnt * kMaxDeg; s += kNT) {
        const int j = s / kMaxDeg, u = s % kMaxDeg;
        if (u >= S.deg[j]) continue;
        const int4 q = S.slot[j][u];
        const int e = q.y / tp.L1, m = q.x / tp.L1;
        float2 w[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        int r[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int el = k ? tp.e_t2[e] : tp.e_t1[e];
            if (el < 0) continue;
            const float2 v = gs_at(tp, g, el, m);
            const float ea = g.elem_area[el];
            w[k] = make_float2(ea * v.x, ea * v.y);
            r[k] = tp.t_ulev[el] | (tp.t_nlev[el] - 1) << 16;
        }
        D.w[j][u] = make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
        D.r[j][u] = make_int2(r[0], r[1]);
    }
    __syncthreads();
}
template <int G>
using DiffBuf = Vec<G>[2][kNT];  // [buffer][thread]: S_xy . node gradient

template <int G>
__device__ __forceinline__ void diff_tile(const DTopo &tp, const DGeom<float> &g, const B32View &B, float dt,
                                          const NodeTile &S, const DiffSlots &D, DiffBuf<G> &X) {
    const TileLane k(tp, S);
    const int x = threadIdx.x, i = k.i, iv = k.iv, nz = k.nz, deg = S.deg[k.j], nl = tp.nl;
    const bool top = nz == k.nzmin, bot = nz == k.nzmax - 1;
    float sdt = 0.f, q = 0.f, kz = 0.f, kzd = 0.f;
    // Redi: weights of p above and at the interfaces nz and nz + 1, the slopes / (3 areasvol)
    float cu = 0.f, cd = 0.f, cu1 = 0.f, cd1 = 0.f, sx = 0.f, sy = 0.f;
    if (k.on) {
        sdt = dt / (g.areasvol[iv] * g.hnode_new[i]);
        if (!top) kz = B.Kv[iv] / (g.Z3[i - 1] - g.Z3[i]) * g.area[iv];
        if (!bot) kzd = B.Kv[iv + 1] / (g.Z3[i] - g.Z3[i + 1]) * g.area[iv + 1];
        q = sdt / (g.zbar3[iv] - g.zbar3[iv + 1]);
        if (B.slope) {
            const float r3 = 1.f / (3.f * g.areasvol[iv]), h = g.hnode[i], kh = h * B.Ki[i];
            sx = B.slope[3 * (size_t)i] * r3;
            sy = B.slope[3 * (size_t)i + 1] * r3;
            if (!top) {
                const float hu = g.hnode[i - 1], w = g.area[iv] / (hu + h);
                cu = hu * B.Ki[i - 1] * w;
                cd = kh * w;
            }
            if (!bot) {
                const float hd = g.hnode[i + 1], w = g.area[iv + 1] / (h + hd);
                cu1 = kh * w;
                cd1 = hd * B.Ki[i + 1] * w;
            }
        }
    }
    (void)nl;
    int b = 0;
#pragma unroll 1
    for (int gq = 0; gq < B.ng; gq++) {
        if (!((B.diff >> gq) & 1ull)) continue;
        const float *__restrict__ T = grp<G>(B.T, gq, B.sN);
        const float *__restrict__ HD = grp<G>(B.HD, gq, B.sE);
        const Vec<G> Tn = vldc<G>(k.on, T, i);
        Vec<G> d = vfill<G>(0.f), p = vfill<G>(0.f);
        if (B.Ki) {
#pragma unroll 1
            for (int u0 = 0; u0 < S.degmax; u0 += 3) {
                Vec<G> xe[3], tm[3];
                float w[3];
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    const int4 s = S.slot[k.j][u0 + u];
                    const bool ok = k.on && u0 + u < deg && slot_wet(s, nz);
                    xe[u] = vldc<G>(ok, HD, s.y + nz - 1);
                    w[u] = 0.f;
                    tm[u] = Tn;
                    if (B.slope && ok) {
                        tm[u] = vld<G>(T, s.x + nz - 1);
                        const float4 v = D.w[k.j][u0 + u];
                        const int2 r = D.r[k.j][u0 + u];
                        if (nz >= (r.x & 0xffff) && nz <= (r.x >> 16)) w[u] += sx * v.x + sy * v.y;
                        if (nz >= (r.y & 0xffff) && nz <= (r.y >> 16)) w[u] += sx * v.z + sy * v.w;
                    }
                }
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    const bool ow = S.slot[k.j][u0 + u].w != 0;
#pragma unroll
                    for (int c = 0; c < G; c++) {
                        d.c[c] += ow ? xe[u].c[c] : -xe[u].c[c];
                        p.c[c] += w[u] * (tm[u].c[c] - Tn.c[c]);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < G; c++) d.c[c] *= sdt;
        }
        if (!((B.ivd >> gq) & 1ull) && k.on) {
            const Vec<G> Tu = vldc<G>(!top, T, i - 1), Td = vldc<G>(!bot, T, i + 1);
            const Vec<G> fs = B.fsurf ? vld<G>(B.fsurf, gq * tp.N2 + k.n) : vfill<G>(0.f);
#pragma unroll
            for (int c = 0; c < G; c++) {
                const float vd0 = top ? fs.c[c] : kz * (Tu.c[c] - Tn.c[c]);
                const float vd1 = bot ? 0.f : kzd * (Tn.c[c] - Td.c[c]);
                d.c[c] += (vd0 - vd1) * q;
            }
        }
        if (B.slope) {
            if (!tp.diff_by_edges() && k.on) {  // the elements themselves
                p = vfill<G>(0.f);
                for (int kk = tp.nie_ptr[k.n]; kk < tp.nie_ptr[k.n + 1]; kk++) {
                    const int el = tp.nie_idx[kk];
                    if (nz < tp.t_ulev[el] || nz > tp.t_nlev[el] - 1) continue;
                    const float ea = g.elem_area[el];
                    for (int m = 0; m < 3; m++) {
                        const Vec<G> t = vld<G>(T, tp.t_n[3 * el + m] * tp.L1 + nz - 1);
                        const float w = (sx * g.gs[6 * (size_t)el + m] + sy * g.gs[6 * (size_t)el + 3 + m]) * ea;
#pragma unroll
                        for (int c = 0; c < G; c++) p.c[c] += w * (tp.grad_zero ? t.c[c] - Tn.c[c] : t.c[c]);
                    }
                }
            }
            Vec<G>(&xp)[kNT] = X[b];
            b ^= 1;
            xp[x] = p;
            __syncthreads();
            if (k.on) {
                const Vec<G> pu = xp[top ? x : x - 1], pd = xp[bot ? x : x + 1];
#pragma unroll
                for (int c = 0; c < G; c++) {
                    const float vd = cu * pu.c[c] + cd * p.c[c], vdn = cu1 * p.c[c] + cd1 * pd.c[c];
                    d.c[c] += (vd - vdn) * sdt;
                }
            }
        }
        if (k.on) vst<G>(grp<G>(B.Tnew, gq, B.sN), i, d);
    }
}

template <int G>
__global__ void __launch_bounds__(kNT, MinB<G>::diff) k32_diff(DTopo tp, DGeom<float> g, B32View B, float dt) {
    __shared__ NodeTile S;
    __shared__ DiffSlots D;
    __shared__ DiffBuf<G> X;
    node_tile_load(tp, blockIdx.x, S);
    if (B.slope && tp.diff_by_edges()) diff_slots_load(tp, g, S, D);
    diff_tile<G>(tp, g, B, dt, S, D, X);
}

template <int G>
__global__ void __launch_bounds__(32 * kWV) k32_vdiff(DTopo tp, B32View B, VFactors vf) {
    __shared__ VdiffWarp Wsm[kWV];
    const int warp = threadIdx.x >> 5;
    for (int n = blockIdx.x * kWV + warp; n < tp.N2; n += gridDim.x * kWV) vdiff_unit<G, false>(tp, B, vf, n, Wsm[warp]);
}

// ---------------------------------------------------------------------------
// content sums and layout conversions
// ---------------------------------------------------------------------------
// FP64 content of every slot of ng groups: block b sums its nodes [b*per, (b+1)*per) in a
// fixed order (threads over nodes, then a tree over the block), out = ordered sum of blocks
template <int G>
__global__ void __launch_bounds__(256) k32_content_partial(DTopo tp, DGeom<float> g, const float *T, int ng,
                                                           double *partials) {
    __shared__ double red[256];
    const int L1 = tp.L1, nl = tp.nl;
    const int per = (tp.N2 + gridDim.x - 1) / gridDim.x;
    const int n0 = blockIdx.x * per, n1 = min(tp.N2, n0 + per);
    for (int gq = 0; gq < ng; gq++) {
        double acc[G];
#pragma unroll
        for (int c = 0; c < G; c++) acc[c] = 0.0;
        const float *Tg = grp<G>(T, gq, (size_t)tp.N2 * L1);
        for (int n = n0 + threadIdx.x; n < n1; n += blockDim.x) {
            const int nzmin = tp.n_ulev[n], nzmax = tp.n_nlev[n];
            for (int nz = nzmin; nz <= nzmax - 1; nz++) {
                const Vec<G> t = vld<G>(Tg, n * L1 + nz - 1);
                const double w = (double)g.hnode_new[n * L1 + nz - 1] * (double)g.areasvol[n * nl + nz - 1];
#pragma unroll
                for (int c = 0; c < G; c++) acc[c] += (double)t.c[c] * w;
            }
        }
#pragma unroll
        for (int c = 0; c < G; c++) {
            red[threadIdx.x] = acc[c];
            __syncthreads();
            for (int s = 128; s > 0; s >>= 1) {
                if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
                __syncthreads();
            }
            if (threadIdx.x == 0) partials[((size_t)blockIdx.x * ng + gq) * G + c] = red[0];
            __syncthreads();
        }
    }
}
__global__ void k32_content_final(const double *partials, int nblk, int nslots, double *out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    double a = 0.0;
    for (int b = 0; b < nblk; b++) a += partials[(size_t)b * nslots + s];
    out[s] = a;
}

template <typename S>
__global__ void k32_put_slot(const S *src, float *grpf, int G, int c, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        grpf[i * G + c] = (float)src[i];
}
template <typename S>
__global__ void k32_get_slot(const float *grpf, int G, int c, size_t count, S *dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (S)grpf[i * G + c];
}
template <typename S>
__global__ void k32_put_slot_pair(const S *src, float *g1, float *g2, int G, int c, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        g1[i * G + c] = (float)src[2 * i];
        g2[i * G + c] = (float)src[2 * i + 1];
    }
}
template <typename S>
__global__ void k32_get_slot_pair(const float *g1, const float *g2, int G, int c, size_t count, S *dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        dst[2 * i] = (S)g1[i * G + c];
        dst[2 * i + 1] = (S)g2[i * G + c];
    }
}
// blockIdx.y: the array (5 + g: the surface fluxes of group g).  16-byte accesses where both ends allow them.  A
// launch instead of 4 copies, a fill and one kernel per tracer: on a small mesh each costs its 2 us
// (a loop of one step on 2.9k nodes: 97 -> 54 us with the direct reads).
__global__ void __launch_bounds__(256) k32_forcing(ForcingCopy f) {
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, st = (size_t)gridDim.x * blockDim.x;
    const int k = blockIdx.y;
    if (k >= 5) {
        const int g = k - 5;
        for (size_t n = t; n < (size_t)f.N2; n += st) {
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int tr = c < f.G ? f.slot_tr[g * f.G + c] : -1;
                v[c] = (f.bc && tr >= 0) ? f.bc[(size_t)tr * f.N2 + n] : 0.f;
            }
            const size_t e = (size_t)g * f.N2 + n;
            if (f.G == 4) reinterpret_cast<float4 *>(f.bc_dst)[e] = make_float4(v[0], v[1], v[2], v[3]);
            else reinterpret_cast<float2 *>(f.bc_dst)[e] = make_float2(v[0], v[1]);
        }
        return;
    }
    const float *__restrict__ src = f.src[k];
    if (!src) return;
    float *__restrict__ dst = f.dst[k];
    float *__restrict__ dst2 = k == 1 ? f.dst1b : nullptr;
    const size_t n = f.n[k], nv = ((uintptr_t)src % 16) ? 0 : n / 4;
    for (size_t i = t; i < nv; i += st) {
        const float4 v = reinterpret_cast<const float4 *>(src)[i];
        reinterpret_cast<float4 *>(dst)[i] = v;
        if (dst2) reinterpret_cast<float4 *>(dst2)[i] = v;
    }
    for (size_t i = 4 * nv + t; i < n; i += st) {
        dst[i] = src[i];
        if (dst2) dst2[i] = src[i];
    }
}
// element i of slot c's source is src.p[c][i * stride + off] (stride 2: one level of AB3's
// interleaved valuesold); a null source fills its slot with zeros
template <int G, typename S>
__global__ void k32_pack_group(SlotSrc<S> src, float *grpf, size_t count, int stride, int off) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        Vec<G> v;
#pragma unroll
        for (int c = 0; c < G; c++) v.c[c] = src.p[c] ? (float)src.p[c][i * stride + off] : 0.f;
        vst<G>(grpf, (int)i, v);
    }
}
template <int G, typename S>
__global__ void k32_unpack_group(const float *grpf, size_t count, SlotDst<S> dst, int stride, int off) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const Vec<G> v = vld<G>(grpf, (int)i);
#pragma unroll
        for (int c = 0; c < G; c++)
            if (dst.p[c]) dst.p[c][i * stride + off] = (S)v.c[c];
    }
}

// ---------------------------------------------------------------------------
// multi-instance launches: every stage over all instances of a batch at once
// ---------------------------------------------------------------------------
// Units (edges, column blocks, nodes, items) of all instances are numbered one after
// another; ix.start[i] is instance i's first unit.  A warp (or thread, or block) finds
// its instance by binary search over those offsets (kernel parameters, warp-uniform)
// and runs the single-instance body with that instance's descriptor and its group width.
__device__ __forceinline__ int find_inst(const MultiIdx &ix, int u) {
    int lo = 0, hi = ix.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ix.start[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// units: tiles of kTileMax edges, one block each
__global__ void __launch_bounds__(kTileThreads) k32m_vflux(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ Tile S;
    __shared__ EdgeV Ed[kTileMax];
    const int i = find_inst(ix, blockIdx.x);
    vflux_tile(I[i].tp, I[i].g, I[i].f, I[i].VF, blockIdx.x - ix.start[i], kTileMax, S, Ed);
}
__global__ void __launch_bounds__(kTB) k32m_vfactors(const Inst32 *__restrict__ I, MultiIdx ix) {
    FOR_WARP_UNITS(u, ix.start[ix.n]) {
        const int i = find_inst(ix, u);
        vfactors_col(I[i].tp, I[i].g, I[i].f, I[i].dt, I[i].vf, u - ix.start[i], threadIdx.x & 31);
    }
}
// units: node tiles, one block each.  WS: some instance has the split vertical velocity (each
// instance checks its own switch)
template <bool WS>
__global__ void __launch_bounds__(kNT, MinB<4>::lo) k32m_lo_ad(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ NodeTile S;
    __shared__ union {
        LoBuf<4> X4;
        LoBuf<2> X2;
    } U;
    const int i = find_inst(ix, blockIdx.x);
    const Inst32 &d = I[i];
    node_tile_load(d.tp, blockIdx.x - ix.start[i], S);
    if (d.B.G == 4) lo_ad_tile<4, WS>(d.tp, d.g, d.f, d.B, d.VF, d.dt, S, U.X4);
    else lo_ad_tile<2, WS>(d.tp, d.g, d.f, d.B, d.VF, d.dt, S, U.X2);
}
__global__ void __launch_bounds__(kTileThreads, MinB<4>::ho) k32m_ho(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ Tile S;
    __shared__ EdgeH Ed[kTileMax];
    const int i = find_inst(ix, blockIdx.x), ti = blockIdx.x - ix.start[i];
    if (I[i].B.G == 4) ho_tile<4>(I[i].tp, I[i].B, I[i].mw, I[i].VF, ti, kTileMax, S, Ed);
    else ho_tile<2>(I[i].tp, I[i].B, I[i].mw, I[i].VF, ti, kTileMax, S, Ed);
}
__global__ void __launch_bounds__(256) k32m_ho_nodemean(const Inst32 *__restrict__ I, MultiIdx ix) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= ix.start[ix.n]) return;
    const int i = find_inst(ix, u);
    if (I[i].B.G == 4) nodemean_item<4>(I[i].tp, I[i].B, I[i].mw, I[i].VF, u - ix.start[i]);
    else nodemean_item<2>(I[i].tp, I[i].B, I[i].mw, I[i].VF, u - ix.start[i]);
}
__global__ void __launch_bounds__(kNT, MinB<4>::bounds) k32m_bounds(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ NodeTile S;
    __shared__ union {
        BoundsBuf<4> X4;
        BoundsBuf<2> X2;
    } U;
    const int i = find_inst(ix, blockIdx.x);
    const Inst32 &d = I[i];
    node_tile_load(d.tp, blockIdx.x - ix.start[i], S);
    if (d.B.G == 4) bounds_tile<4>(d.tp, d.g, d.B, d.dt, S, U.X4);
    else bounds_tile<2>(d.tp, d.g, d.B, d.dt, S, U.X2);
}
// a tile's columns are then diffused where its instance has groups in ivd & ~wimpl (as k32_update
// with the diffusion epilogue)
__global__ void __launch_bounds__(kNT, MinB<4>::update) k32m_update(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ NodeTile S;
    __shared__ union {
        UpdateBuf<4> X4;
        UpdateBuf<2> X2;
        VdiffWarp W[kNT / 32];
    } U;
    const int i = find_inst(ix, blockIdx.x);
    const Inst32 &d = I[i];
    node_tile_load(d.tp, blockIdx.x - ix.start[i], S);
    const bool vd = (d.B.ivd & ~d.B.wimpl) != 0;
    if (d.B.G == 4) {
        update_tile<4>(d.tp, d.g, d.B, d.dt, S, U.X4);
        if (vd) update_tile_vdiff<4>(d.tp, d.B, d.vf, S, U.W);
    } else {
        update_tile<2>(d.tp, d.g, d.B, d.dt, S, U.X2);
        if (vd) update_tile_vdiff<2>(d.tp, d.B, d.vf, S, U.W);
    }
}
__global__ void __launch_bounds__(kTB) k32m_vppm(const Inst32 *__restrict__ I, MultiIdx ix) {
    FOR_WARP_UNITS(u, ix.start[ix.n]) {
        const int i = find_inst(ix, u);
        if (I[i].B.ppm && I[i].B.G == 4) vppm_node<4>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dt, u - ix.start[i], threadIdx.x & 31);
        else if (I[i].B.ppm) vppm_node<2>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dt, u - ix.start[i], threadIdx.x & 31);
    }
}
__global__ void __launch_bounds__(128) k32m_lo_impl(const Inst32 *__restrict__ I, MultiIdx ix) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= ix.start[ix.n]) return;
    const int i = find_inst(ix, u);
    if (!I[i].f.wsplit) return;
    if (I[i].B.G == 4) lo_impl_column<4>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dtd, I[i].scratch, u - ix.start[i]);
    else lo_impl_column<2>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dtd, I[i].scratch, u - ix.start[i]);
}
__global__ void __launch_bounds__(128) k32m_vdiff_w(const Inst32 *__restrict__ I, MultiIdx ix) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= ix.start[ix.n]) return;
    const int i = find_inst(ix, u);
    if (!I[i].B.wimpl) return;
    if (I[i].B.G == 4) vdiff_w_column<4>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dtd, I[i].scratch, u - ix.start[i]);
    else vdiff_w_column<2>(I[i].tp, I[i].g, I[i].f, I[i].B, I[i].dtd, I[i].scratch, u - ix.start[i]);
}

// the instances that take their elements' own nodes (OWN), or those that do not
template <bool OWN>
__global__ void __launch_bounds__(kTileThreads, MinB<4>::hdiff) k32m_hdiff(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ Tile S;
    __shared__ EdgeD Ed[kTileMax];
    const int i = find_inst(ix, blockIdx.x), ti = blockIdx.x - ix.start[i];
    if (I[i].tp.diff_by_edges() == OWN) return;
    if (I[i].B.G == 4) hdiff_tile<4, OWN>(I[i].tp, I[i].g, I[i].B, ti, kTileMax, S, Ed);
    else hdiff_tile<2, OWN>(I[i].tp, I[i].g, I[i].B, ti, kTileMax, S, Ed);
}
__global__ void __launch_bounds__(kNT, MinB<4>::diff) k32m_diff(const Inst32 *__restrict__ I, MultiIdx ix) {
    __shared__ NodeTile S;
    __shared__ DiffSlots D;
    __shared__ union {
        DiffBuf<4> X4;
        DiffBuf<2> X2;
    } U;
    const int i = find_inst(ix, blockIdx.x);
    const Inst32 &d = I[i];
    if (!d.B.diff) return;
    node_tile_load(d.tp, blockIdx.x - ix.start[i], S);
    if (d.B.slope && d.tp.diff_by_edges()) diff_slots_load(d.tp, d.g, S, D);
    if (d.B.G == 4) diff_tile<4>(d.tp, d.g, d.B, d.dt, S, D, U.X4);
    else diff_tile<2>(d.tp, d.g, d.B, d.dt, S, D, U.X2);
}

// ---------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------
// node-tile kernels: one block per tile, or at most blocks_per_sm blocks per SM looping
static int grid_tiles(int tiles, const LaunchShape &sh) {
    return sh.blocks_per_sm > 0 ? std::min(tiles, 152 * sh.blocks_per_sm) : tiles;
}
static int grid_nodes(int n) { return (n + kWB - 1) / kWB; }
static int grid_flat(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 152 * 32); }

void b32_vflux(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, float *VF, cudaStream_t s) {
    const int t = tile_size(tp.E2, 0);
    k32_vflux<<<(tp.E2 + t - 1) / t, kTileThreads, 0, s>>>(tp, g, f, VF, t);
}
void b32_vfactors(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, double dt, const VFactors &v,
                  cudaStream_t s) {
    k32_vfactors<<<grid_nodes(tp.N2), kTB, 0, s>>>(tp, g, f, (float)dt, v);
}

bool b32_fct_clamp() { return kFctClamp; }

void b32_lo_ad(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, const B32View &B, const float *VF,
               double dt, const LaunchShape &sh, cudaStream_t s) {
    const int nb = grid_tiles(tp.n_nt, sh);
    if (B.G == 4) {
        if (f.wsplit) k32_lo_ad<4, true><<<nb, kNT, 0, s>>>(tp, g, f, B, VF, (float)dt);
        else k32_lo_ad<4, false><<<nb, kNT, 0, s>>>(tp, g, f, B, VF, (float)dt);
    } else {
        if (f.wsplit) k32_lo_ad<2, true><<<nb, kNT, 0, s>>>(tp, g, f, B, VF, (float)dt);
        else k32_lo_ad<2, false><<<nb, kNT, 0, s>>>(tp, g, f, B, VF, (float)dt);
    }
}
template <int G>
static void ho_g(const DTopo &tp, const B32View &B, const MusclW &mw, const float *VF, cudaStream_t s) {
    const int t = tile_size(tp.E2, 0);
    k32_ho<G><<<(tp.E2 + t - 1) / t, kTileThreads, 0, s>>>(tp, B, mw, VF, t);
}
void b32_ho(const DTopo &tp, const DGeom<float> &, const B32View &B, const MusclW &mw, const float *VF,
            cudaStream_t s) {
    if (B.G == 4) ho_g<4>(tp, B, mw, VF, s);
    else ho_g<2>(tp, B, mw, VF, s);
}
void b32_ho_nodemean(const DTopo &tp, const B32View &B, const MusclW &mw, const float *VF, cudaStream_t s) {
    if (!mw.n_items) return;
    const int blocks = std::min((mw.n_items + 255) / 256, 152 * 8);
    if (B.G == 4) k32_ho_nodemean<4><<<blocks, 256, 0, s>>>(tp, B, mw, VF);
    else k32_ho_nodemean<2><<<blocks, 256, 0, s>>>(tp, B, mw, VF);
}
void b32_bounds(const DTopo &tp, const DGeom<float> &g, const B32View &B, double dt, const LaunchShape &sh,
                cudaStream_t s) {
    const int nb = grid_tiles(tp.n_nt, sh);
    if (B.G == 4) k32_bounds<4><<<nb, kNT, 0, s>>>(tp, g, B, (float)dt);
    else k32_bounds<2><<<nb, kNT, 0, s>>>(tp, g, B, (float)dt);
}
template <int G>
static void update_g(const DTopo &tp, const DGeom<float> &g, const B32View &B, double dt, int nb, const VFactors *vf,
                     cudaStream_t s) {
    if (vf) k32_update<G, true><<<nb, kNT, 0, s>>>(tp, g, B, (float)dt, *vf);
    else k32_update<G, false><<<nb, kNT, 0, s>>>(tp, g, B, (float)dt, VFactors{});
}
void b32_update(const DTopo &tp, const DGeom<float> &g, const B32View &B, double dt, const LaunchShape &sh,
                const VFactors *vf, cudaStream_t s) {
    const int nb = grid_tiles(tp.n_nt, sh);
    if (B.G == 4) update_g<4>(tp, g, B, dt, nb, vf, s);
    else update_g<2>(tp, g, B, dt, nb, vf, s);
}
void b32_vdiff(const DTopo &tp, const DForcing<float> &, const B32View &B, const VFactors &v, cudaStream_t s) {
    if (B.G == 4) k32_vdiff<4><<<(tp.N2 + kWV - 1) / kWV, 32 * kWV, 0, s>>>(tp, B, v);
    else k32_vdiff<2><<<(tp.N2 + kWV - 1) / kWV, 32 * kWV, 0, s>>>(tp, B, v);
}
void b32_vppm(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, const B32View &B, double dt,
              cudaStream_t s) {
    if (B.G == 4) k32_vppm<4><<<grid_nodes(tp.N2), kTB, 0, s>>>(tp, g, f, B, (float)dt);
    else k32_vppm<2><<<grid_nodes(tp.N2), kTB, 0, s>>>(tp, g, f, B, (float)dt);
}
void b32_lo_impl(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, const B32View &B, double dt,
                 double *scratch, cudaStream_t s) {
    if (B.G == 4) k32_lo_impl<4><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, B, dt, scratch);
    else k32_lo_impl<2><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, B, dt, scratch);
}
void b32_vdiff_w(const DTopo &tp, const DGeom<float> &g, const DForcing<float> &f, const B32View &B, double dt,
                 double *scratch, cudaStream_t s) {
    if (B.G == 4) k32_vdiff_w<4><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, B, dt, scratch);
    else k32_vdiff_w<2><<<(tp.N2 + 127) / 128, 128, 0, s>>>(tp, g, f, B, dt, scratch);
}
// Redi K33 = Kv + Ty (oce_ale_tracer.F90:1099-1204) of every interface nzmin < nz < nzmax: Ty =
// (zbar(nz) - Z(nz)) / dZ s3(nz-1)^2 Ki(nz-1) + (Z(nz-1) - zbar(nz)) / dZ s3(nz)^2 Ki(nz) with dZ = Z(nz-1)
// - Z(nz): the depth differences are half thicknesses, so Ty = (h(nz) s3(nz-1)^2 Ki(nz-1) + h(nz-1) s3(nz)^2
// Ki(nz)) / (h(nz-1) + h(nz)) with h = hnode_new; Kv outside the column's inner interfaces.
//
// A warp per column; the products, the sums and the quotient as unevaluated sums of two FP32 numbers
// (errors of products and sums by fma and two-sum, T. J. Dekker, Numer. Math. 18, 1971), rounded once:
// within 2^-24 of the exact value plus 2^-44.  FP64 arithmetic along the column, which subtracts
// accumulated depths, took 18 FP64 instructions per interface and strided reads: 293 -> 60 us on the sphere of 7
// subdivisions.  Over 292k interfaces of 20, 47 and 80 layers, thin bottom cells included, both give the FP32
// number nearest to the exact value every time (error 5.9e-8 at most, 2.5e-8 rms).
struct F2 {
    float h, l;
};
__device__ __forceinline__ F2 two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ F2 two_sum(float a, float b) {
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ F2 f2_mul(F2 a, float b) {
    const F2 p = two_prod(a.h, b);
    return {p.h, __fmaf_rn(a.l, b, p.l)};
}
__global__ void __launch_bounds__(kTB) k32_k33(DTopo tp, DGeom<float> g, const float *__restrict__ Kv,
                                               const float *__restrict__ Ki, const float *__restrict__ slope,
                                               float *__restrict__ K33) {
    const int L1 = tp.L1, nl = tp.nl, lane = threadIdx.x & 31;
    const int n = blockIdx.x * kWB + (threadIdx.x >> 5);
    if (n >= tp.N2) return;
    const int nzmax = tp.n_nlev[n], nzmin = tp.n_ulev[n];
    for (int nz = 1 + lane; nz <= nl; nz += 32) {
        const size_t b = (size_t)n * nl + nz - 1, c = (size_t)n * L1 + nz - 1;
        float out = Kv[b];
        if (nz > nzmin && nz < nzmax) {
            const float hu = g.hnode_new[c - 1], hc = g.hnode_new[c];
            const float sa = slope[3 * (c - 1) + 2], sb = slope[3 * c + 2];
            const F2 x = f2_mul(f2_mul(two_prod(sa, sa), Ki[c - 1]), hc);
            const F2 y = f2_mul(f2_mul(two_prod(sb, sb), Ki[c]), hu);
            const F2 m = two_sum(x.h, y.h), d = two_sum(hu, hc);
            const float ml = m.l + (x.l + y.l);
            const float q = __fdiv_rn(m.h, d.h);
            const float r = __fdiv_rn(__fmaf_rn(-q, d.l, __fadd_rn(__fmaf_rn(-q, d.h, m.h), ml)), d.h);
            const F2 t = two_sum(out, q);
            out = __fadd_rn(t.h, __fadd_rn(t.l, r));
        }
        K33[b] = out;
    }
}

void b32_k33(const DTopo &tp, const DGeom<float> &g, const float *Kv, const float *Ki, const float *slope, float *K33,
             cudaStream_t s) {
    k32_k33<<<grid_nodes(tp.N2), kTB, 0, s>>>(tp, g, Kv, Ki, slope, K33);
}

void b32_hdiff(const DTopo &tp, const DGeom<float> &g, const B32View &B, cudaStream_t s) {
    const int t = tile_size(tp.E2, 0), nb = (tp.E2 + t - 1) / t;
    if (B.G == 4) {
        if (tp.diff_by_edges()) k32_hdiff<4, false><<<nb, kTileThreads, 0, s>>>(tp, g, B, t);
        else k32_hdiff<4, true><<<nb, kTileThreads, 0, s>>>(tp, g, B, t);
    } else {
        if (tp.diff_by_edges()) k32_hdiff<2, false><<<nb, kTileThreads, 0, s>>>(tp, g, B, t);
        else k32_hdiff<2, true><<<nb, kTileThreads, 0, s>>>(tp, g, B, t);
    }
}
void b32_diff(const DTopo &tp, const DGeom<float> &g, const B32View &B, double dt, cudaStream_t s) {
    if (B.G == 4) k32_diff<4><<<tp.n_nt, kNT, 0, s>>>(tp, g, B, (float)dt);
    else k32_diff<2><<<tp.n_nt, kNT, 0, s>>>(tp, g, B, (float)dt);
}

void b32_content(const DTopo &tp, const DGeom<float> &g, const float *T, int ng, int G, double *partials, int nblk,
                 double *out, cudaStream_t s) {
    if (G == 4) k32_content_partial<4><<<nblk, 256, 0, s>>>(tp, g, T, ng, partials);
    else k32_content_partial<2><<<nblk, 256, 0, s>>>(tp, g, T, ng, partials);
    const int nslots = ng * G;
    k32_content_final<<<(nslots + 63) / 64, 64, 0, s>>>(partials, nblk, nslots, out);
}
void b32_put_slot(const double *src, float *grpf, int G, int c, size_t count, cudaStream_t s) {
    k32_put_slot<double><<<grid_flat(count), 256, 0, s>>>(src, grpf, G, c, count);
}
void b32_put_slot_f(const float *src, float *grpf, int G, int c, size_t count, cudaStream_t s) {
    k32_put_slot<float><<<grid_flat(count), 256, 0, s>>>(src, grpf, G, c, count);
}
void b32_get_slot(const float *grpf, int G, int c, size_t count, double *dst, cudaStream_t s) {
    k32_get_slot<double><<<grid_flat(count), 256, 0, s>>>(grpf, G, c, count, dst);
}
void b32_get_slot_f(const float *grpf, int G, int c, size_t count, float *dst, cudaStream_t s) {
    k32_get_slot<float><<<grid_flat(count), 256, 0, s>>>(grpf, G, c, count, dst);
}
void b32_put_slot_pair(const double *src, float *g1, float *g2, int G, int c, size_t count, cudaStream_t s) {
    k32_put_slot_pair<double><<<grid_flat(count), 256, 0, s>>>(src, g1, g2, G, c, count);
}
void b32_put_slot_pair_f(const float *src, float *g1, float *g2, int G, int c, size_t count, cudaStream_t s) {
    k32_put_slot_pair<float><<<grid_flat(count), 256, 0, s>>>(src, g1, g2, G, c, count);
}
void b32_get_slot_pair(const float *g1, const float *g2, int G, int c, size_t count, double *dst, cudaStream_t s) {
    k32_get_slot_pair<double><<<grid_flat(count), 256, 0, s>>>(g1, g2, G, c, count, dst);
}
void b32_get_slot_pair_f(const float *g1, const float *g2, int G, int c, size_t count, float *dst, cudaStream_t s) {
    k32_get_slot_pair<float><<<grid_flat(count), 256, 0, s>>>(g1, g2, G, c, count, dst);
}
void b32_forcing(const ForcingCopy &f, cudaStream_t s) {
    size_t n = 0;
    for (size_t m : f.n) n = std::max(n, m);
    const int nb = (int)std::min<size_t>((n / 4 + 255) / 256 + 1, 152 * 8);
    k32_forcing<<<dim3(nb, 5 + f.ngr), 256, 0, s>>>(f);
}
template <typename S>
void b32_pack_group(const SlotSrc<S> &src, float *grpf, int G, size_t count, int stride, int off, cudaStream_t s) {
    if (G == 4) k32_pack_group<4, S><<<grid_flat(count), 256, 0, s>>>(src, grpf, count, stride, off);
    else k32_pack_group<2, S><<<grid_flat(count), 256, 0, s>>>(src, grpf, count, stride, off);
}
template <typename S>
void b32_unpack_group(const float *grpf, int G, size_t count, const SlotDst<S> &dst, int stride, int off,
                      cudaStream_t s) {
    if (G == 4) k32_unpack_group<4, S><<<grid_flat(count), 256, 0, s>>>(grpf, count, dst, stride, off);
    else k32_unpack_group<2, S><<<grid_flat(count), 256, 0, s>>>(grpf, count, dst, stride, off);
}
template void b32_pack_group<float>(const SlotSrc<float> &, float *, int, size_t, int, int, cudaStream_t);
template void b32_pack_group<double>(const SlotSrc<double> &, float *, int, size_t, int, int, cudaStream_t);
template void b32_unpack_group<float>(const float *, int, size_t, const SlotDst<float> &, int, int, cudaStream_t);
template void b32_unpack_group<double>(const float *, int, size_t, const SlotDst<double> &, int, int, cudaStream_t);

// multi-instance launch wrappers: ix_* hold the per-instance unit offsets of each stage
void bm32_vflux(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_vflux<<<u, kTileThreads, 0, s>>>(I, ix);
}
void bm32_vfactors(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_vfactors<<<grid_nodes(u), kTB, 0, s>>>(I, ix);
}
void bm32_lo_ad(const Inst32 *I, const MultiIdx &ix, bool ws, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (!u) return;
    if (ws) k32m_lo_ad<true><<<u, kNT, 0, s>>>(I, ix);
    else k32m_lo_ad<false><<<u, kNT, 0, s>>>(I, ix);
}
void bm32_vppm(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_vppm<<<grid_nodes(u), kTB, 0, s>>>(I, ix);
}
void bm32_lo_impl(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_lo_impl<<<(u + 127) / 128, 128, 0, s>>>(I, ix);
}
void bm32_vdiff_w(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_vdiff_w<<<(u + 127) / 128, 128, 0, s>>>(I, ix);
}
void bm32_ho(const Inst32 *I, const MultiIdx &ix_e, const MultiIdx &ix_items, cudaStream_t s) {
    if (ix_e.start[ix_e.n]) k32m_ho<<<ix_e.start[ix_e.n], kTileThreads, 0, s>>>(I, ix_e);
    const int u = ix_items.start[ix_items.n];
    if (u) k32m_ho_nodemean<<<(u + 255) / 256, 256, 0, s>>>(I, ix_items);
}
void bm32_bounds(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_bounds<<<u, kNT, 0, s>>>(I, ix);
}
void bm32_update(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_update<<<u, kNT, 0, s>>>(I, ix);
}
void bm32_hdiff(const Inst32 *I, const MultiIdx &ix, bool own, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (!u) return;
    k32m_hdiff<false><<<u, kTileThreads, 0, s>>>(I, ix);
    if (own) k32m_hdiff<true><<<u, kTileThreads, 0, s>>>(I, ix);
}
void bm32_diff(const Inst32 *I, const MultiIdx &ix, cudaStream_t s) {
    const int u = ix.start[ix.n];
    if (u) k32m_diff<<<u, kNT, 0, s>>>(I, ix);
}

}  // namespace fesom
