// vdiff_column.cuh -- the column solve of diff_ver_part_impl_ale (FP64), shared by the
// context kernel k_vdiff (tracer_kernels.cuh) and the allocation-free entry point
// (vdiff_noalloc.cu).  Both translation units build with --fmad=false, so the two give
// the same bits.
//
// Two mappings with the same bits: a tile of columns in shared memory (vdiff_tile), and one thread
// per column over a scratch in device memory for columns too deep for it.  Scratch entry k of a column (Z_n, the Thomas factors cp and tp)
// sits at p[k * st]: level-major over the columns of a launch, so the threads of a warp
// touch consecutive addresses at every level.
#pragma once
#include <cuda_runtime.h>

namespace fesom {

struct ColScratch {
    double *z, *cp, *tp;  // already offset to the thread's column
    size_t st;            // distance between consecutive levels of one column
};

// Z_n of the column from the bottom up (src/oce_ale_tracer.F90:1088-1096); hn is 1-based
template <typename R>
__device__ __forceinline__ void vdiff_col_z(const ColScratch &s, int nzmin, int nzmax, double zbot, const R *hn) {
    typedef double A;
    A zb = zbot;
    s.z[(size_t)(nzmax - 1) * s.st] = zb + (A)hn[nzmax - 1] / 2.0;
    for (int nz = nzmax - 1; nz >= nzmin + 1; nz--) {
        zb = zb + (A)hn[nz];
        s.z[(size_t)(nz - 1) * s.st] = zb + (A)hn[nz - 1] / 2.0;
    }
}

// The tridiagonal system of one tracer's column (coefficients built on the fly,
// src/oce_ale_tracer.F90:1099-1229, bc_surface at the top :1377-1383), forward elimination
// (:1406-1414) and back substitution (:1417-1430), T += the solution.  wimpl: the implicit
// part of a split vertical velocity joins the solve (:961, 1134-1216).  Arrays are 1-based
// column pointers; the column holds nzmin .. nzmax-1 with at least two layers.
template <typename R>
__device__ __forceinline__ void vdiff_col_solve(const ColScratch &s, int nzmin, int nzmax, const R *hn, const R *ar,
                                                const R *av, const R *kv, bool wimpl, const R *wi, double bc,
                                                double dt, R *Tc) {
    typedef double A;
#define ZN(k) s.z[(size_t)(k) * s.st]
#define CP(k) s.cp[(size_t)(k) * s.st]
#define TP(k) s.tp[(size_t)(k) * s.st]
    int nz = nzmin;
    A zinv2 = 1.0 / (ZN(nz) - ZN(nz + 1));
    const A zinv = 1.0 * dt;
    A c = -((A)kv[nz + 1] * zinv2 * zinv * (A)ar[nz + 1] / (A)av[nz]);
    A b = -c + (A)hn[nz];
    if (wimpl) {  // :1134-1147
        A v = zinv * ((A)ar[nz] / (A)av[nz]);
        b = b + (A)wi[nz] * v;
        v = zinv * (A)ar[nz + 1] / (A)av[nz];
        b = b - fmin(0.0, (A)wi[nz + 1]) * v;
        c = c - fmax(0.0, (A)wi[nz + 1]) * v;
    }
    A Tm = (A)Tc[nz], T0 = Tm, Tp1 = (A)Tc[nz + 1];
    A dz = (A)hn[nz];
    A rhs = -((b - dz) * T0) - c * Tp1;
    rhs = rhs + bc;
    A cp = c / b, tpv = rhs / b;
    CP(nz) = cp;
    TP(nz) = tpv;
    A zinv1 = zinv2;
    for (nz = nzmin + 1; nz <= nzmax - 2; nz++) {
        zinv2 = 1.0 / (ZN(nz) - ZN(nz + 1));
        A a = -((A)kv[nz] * zinv1 * zinv * ((A)ar[nz] / (A)av[nz]));
        c = -((A)kv[nz + 1] * zinv2 * zinv * (A)ar[nz + 1] / (A)av[nz]);
        b = -a - c + (A)hn[nz];
        zinv1 = zinv2;
        if (wimpl) {  // :1176-1189
            A v = zinv * ((A)ar[nz] / (A)av[nz]);
            a = a + fmin(0.0, (A)wi[nz]) * v;
            b = b + fmax(0.0, (A)wi[nz]) * v;
            v = zinv * (A)ar[nz + 1] / (A)av[nz];
            b = b - fmin(0.0, (A)wi[nz + 1]) * v;
            c = c - fmax(0.0, (A)wi[nz + 1]) * v;
        }
        Tm = T0;
        T0 = Tp1;
        Tp1 = (A)Tc[nz + 1];
        dz = (A)hn[nz];
        rhs = -(a * Tm) - (b - dz) * T0 - c * Tp1;
        const A m = b - cp * a;
        cp = c / m;
        tpv = (rhs - tpv * a) / m;
        CP(nz) = cp;
        TP(nz) = tpv;
    }
    nz = nzmax - 1;
    {
        A a = -((A)kv[nz] * zinv1 * zinv * ((A)ar[nz] / (A)av[nz]));
        b = -a + (A)hn[nz];
        if (wimpl) {  // :1207-1216
            const A v = zinv * ((A)ar[nz] / (A)av[nz]);
            a = a + fmin(0.0, (A)wi[nz]) * v;
            b = b + fmax(0.0, (A)wi[nz]) * v;
        }
        Tm = T0;
        T0 = Tp1;
        dz = (A)hn[nz];
        rhs = -(a * Tm) - (b - dz) * T0;
        const A m = b - cp * a;
        tpv = (rhs - tpv * a) / m;
    }
    A trv = tpv;
    Tc[nzmax - 1] = (R)((A)Tc[nzmax - 1] + trv);
    for (nz = nzmax - 2; nz >= nzmin; nz--) {
        trv = TP(nz) - CP(nz) * trv;
        Tc[nz] = (R)((A)Tc[nz] + trv);
    }
#undef ZN
#undef CP
#undef TP
}

// ---------------------------------------------------------------------------
// the same solve for a tile of 32 columns in shared memory
// ---------------------------------------------------------------------------
// A thread per column (above) reads every array with the stride of a column (32 lines per warp
// load) and runs one chain of five divisions per level, four warps to an SM on a mesh of 20k
// nodes.  Here only the recurrences themselves (mid-depths, pivots, substitutions) run a lane per
// column; coefficients and right-hand sides are formed by all 128 threads, the wet levels of the
// tile dealt out one after another (coalesced, full warps).  Up to 4 tracers share the
// coefficients and the pivots.  Entry (level, column) of a shared array sits at level * 33 +
// column: both a lane per column and a lane per level touch 32 different bank pairs.
// Deeper columns than the shared memory holds (217 layers) take the thread per column.
constexpr int kVCols = 32, kVThreads = 128, kVPad = kVCols + 1;
constexpr size_t kVSmemMax = 224 * 1024;
__host__ __device__ constexpr size_t vtile_smem(int L1, int nt) { return (size_t)(3 + nt) * L1 * kVPad * sizeof(double); }

struct VArgs {
    int N2, nl;
    const int *nlev, *ulev;
    const double *zbot, *hn, *ar, *av, *kv, *wi;
    double dt;
};
struct VTracer {
    double *T;
    const double *bc;  // surface flux per node, null: none
};

struct VTile {
    int total;
    int pre[kVCols + 1], top[kVCols];
    __device__ __forceinline__ void fill(int lane, int first_level, int levels) {
        int s = levels;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        pre[lane + 1] = s;
        top[lane] = first_level;
        if (lane == 0) pre[0] = 0;
        if (lane == 31) total = s;
    }
    __device__ __forceinline__ int find(int i) const {
        int j = i >= pre[16] ? 16 : 0;
        j += i >= pre[j + 8] ? 8 : 0;
        j += i >= pre[j + 4] ? 4 : 0;
        j += i >= pre[j + 2] ? 2 : 0;
        return j + (i >= pre[j + 1] ? 1 : 0);
    }
};

// nt <= NT tracers of one wimpl; every thread of the block, S filled and the block synchronised
template <int NT>
__device__ __forceinline__ void vdiff_tile(const VArgs &P, const VTile &S, int n0, double *sm, const VTracer *tr, int nt,
                                           bool wimpl) {
    const int L1 = P.nl - 1, nl = P.nl;
    const size_t sz = (size_t)L1 * kVPad;
    double *HB = sm, *ZR = sm + sz, *A = sm + 2 * sz, *C = sm + 3 * sz;  // h then b, Z then the first rhs, a, c
    auto R = [&](int t) { return t == 0 ? ZR : sm + (3 + t) * sz; };
#define FOR_ITEMS                                                                                      \
    for (int i = threadIdx.x; i < S.total; i += kVThreads) {                                           \
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j], x = (nz - 1) * kVPad + j;               \
        const bool top = i == S.pre[j], bot = i + 1 == S.pre[j + 1];                                   \
        const size_t k = (size_t)(n0 + j) * L1 + nz - 1, kv = (size_t)(n0 + j) * nl + nz - 1;          \
        (void)top; (void)bot; (void)k; (void)kv; (void)x;
    FOR_ITEMS
        HB[x] = P.hn[k];
    }
    __syncthreads();
    const int lane = threadIdx.x;
    int lo = 0, hi = -1;  // shared-memory rows of the lane's column
    if (lane < kVCols) {
        lo = (S.top[lane] - 1) * kVPad + lane;
        hi = lo + (S.pre[lane + 1] - S.pre[lane] - 1) * kVPad;
        if (hi >= lo) {  // Z_n from the bottom up (src/oce_ale_tracer.F90:1088-1096)
            double zb = P.zbot[n0 + lane];
            for (int x = hi; x >= lo; x -= kVPad) {
                const double h = HB[x];
                ZR[x] = zb + h / 2.0;
                zb = zb + h;
            }
        }
    }
    __syncthreads();
    // the interface above layer nz: a(nz) and c(nz - 1)
    FOR_ITEMS
        if (top) {
            A[x] = 0.0;
            C[((S.top[j] - 1) + (S.pre[j + 1] - S.pre[j] - 1)) * kVPad + j] = 0.0;
        } else {
            const double q = P.kv[kv] * (1.0 / (ZR[x - kVPad] - ZR[x])) * P.dt, ar = P.ar[kv];
            A[x] = -(q * (ar / P.av[kv]));
            C[x - kVPad] = -(q * ar / P.av[kv - 1]);
        }
    }
    __syncthreads();
    FOR_ITEMS
        double a = A[x], c = C[x];
        const double h = HB[x];
        double b = -a - c + h;
        if (wimpl) {  // :1134-1216
            double v = P.dt * (P.ar[kv] / P.av[kv]);
            if (top) {
                b = b + P.wi[kv] * v;
            } else {
                a = a + fmin(0.0, P.wi[kv]) * v;
                b = b + fmax(0.0, P.wi[kv]) * v;
            }
            if (!bot) {
                v = P.dt * P.ar[kv + 1] / P.av[kv];
                b = b - fmin(0.0, P.wi[kv + 1]) * v;
                c = c - fmax(0.0, P.wi[kv + 1]) * v;
            }
            A[x] = a;
            C[x] = c;
        }
        HB[x] = b;
        const double bd = b - h;
#pragma unroll
        for (int t = 0; t < NT; t++) {
            if (t >= nt) break;
            const double *T = tr[t].T;
            double r = -(a * (top ? 0.0 : T[k - 1])) - bd * T[k] - c * (bot ? 0.0 : T[k + 1]);
            if (top) r = r + (tr[t].bc ? tr[t].bc[n0 + j] : 0.0);
            R(t)[x] = r;
        }
    }
    __syncthreads();
    if (lane < kVCols && hi >= lo) {
        // forward elimination (:1406-1414), the next level's entries loaded a level ahead
        double cp = 0.0, tp[NT], an = A[lo], bn = HB[lo], cn = C[lo], rn[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) {
            tp[t] = 0.0;
            rn[t] = t < nt ? R(t)[lo] : 0.0;
        }
        for (int x = lo; x <= hi; x += kVPad) {
            const double a = an, b = bn, c = cn;
            double r[NT];
#pragma unroll
            for (int t = 0; t < NT; t++) r[t] = rn[t];
            if (x < hi) {
                an = A[x + kVPad];
                bn = HB[x + kVPad];
                cn = C[x + kVPad];
#pragma unroll
                for (int t = 0; t < NT; t++)
                    if (t < nt) rn[t] = R(t)[x + kVPad];
            }
            const double m = b - cp * a;
            cp = c / m;
            C[x] = cp;
#pragma unroll
            for (int t = 0; t < NT; t++)
                if (t < nt) {
                    tp[t] = (r[t] - tp[t] * a) / m;
                    R(t)[x] = tp[t];
                }
        }
        // back substitution (:1417-1430); C is 0 at the bottom layer
#pragma unroll
        for (int t = 0; t < NT; t++) tp[t] = 0.0;
        for (int x = hi; x >= lo; x -= kVPad) {
            const double c = C[x];
#pragma unroll
            for (int t = 0; t < NT; t++)
                if (t < nt) {
                    tp[t] = R(t)[x] - c * tp[t];
                    R(t)[x] = tp[t];
                }
        }
    }
    __syncthreads();
    FOR_ITEMS
#pragma unroll
        for (int t = 0; t < NT; t++)
            if (t < nt) tr[t].T[k] = tr[t].T[k] + R(t)[x];
    }
#undef FOR_ITEMS
}

}  // namespace fesom
