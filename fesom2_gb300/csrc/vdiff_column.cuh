// vdiff_column.cuh -- the column solve of diff_ver_part_impl_ale (FP64), shared by the
// context kernel k_vdiff (tracer_kernels.cuh) and the allocation-free entry point
// (vdiff_noalloc.cu).  Both translation units build with --fmad=false, so the two give
// the same bits.
//
// Two mappings with the same bits: a tile of columns in shared memory (vdiff_tile), and one thread
// per column over a scratch in device memory for columns too deep for it and for many deep ones
// (vdiff_by_column).  Scratch entry k of a column (Z_n, the Thomas factors cp and tp)
// sits at p[k * st]: level-major over the columns of a launch, so the threads of a warp
// touch consecutive addresses at every level.
#pragma once
#include <cuda_runtime.h>

#include "fp64_arith.cuh"

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
// load) and runs one chain of five divisions per level.  Here only the recurrences run a lane per
// column; coefficients and right-hand sides are formed by all 256 threads, the wet levels of the
// tile dealt out one after another (coalesced, full warps), and up to 4 tracers share the
// coefficients and the pivots.
//
// What bounds it is the FP64 unit: a warp issues a dependent or independent FP64 instruction every
// 64 cycles whatever its active lanes, and an SM one every 19 (measured; a division is 9 of them).
// A recurrence is one warp's work, so the pivots (11 instructions a level) and each tracer's
// elimination (11) run on different warps, the tracers a chunk of 8 levels behind the pivots.
//
// Entry (level, column) of a shared array sits at level * pad + column with an odd pad: both a lane
// per column and a lane per level touch different banks.  Deeper columns than the shared memory
// holds (217 layers), and many deep ones (vdiff_by_column), take the thread per column.
constexpr int kVCols = 32, kVThreads = 256, kVChunk = 8;
constexpr size_t kVSmemMax = 224 * 1024;
constexpr size_t kVSmemHalf = 115200;  // two blocks of it, their VTile and 1 KB reserved for each fill an SM's 228 KB
__host__ __device__ constexpr size_t vtile_smem(int L1, int cols, int nt) {
    return (size_t)(3 + nt) * L1 * (cols | 1) * sizeof(double);
}
// columns per tile: the recurrences cost an SM 12 + 13 nt FP64 instructions per level and tile, the
// rest 29 + 9 nt per 32 columns and level; the widest tile unless a narrower one shares the tiles
// out better over the 152 SMs (2.9k columns: 20, one tile on each of 146 SMs).  A tile that leaves no room for
// a second one on its SM (32 columns from 110 layers on) has nobody to run while its recurrences do: 1.65
// times the time per tile, where an SM gets several (78k columns of 120 layers: 2192 us with 32 columns, 1319
// with 29)
inline int vtile_cols(int n, int nt, int L1) {
    int best = kVCols;
    double cost = 0.0;
    for (int c = kVCols; c >= 8; c--) {
        const int waves = ((n + c - 1) / c + 151) / 152;
        const bool alone = waves > 1 && vtile_smem(L1, c, nt) > kVSmemHalf;
        const double x = waves * (12.0 + 13.0 * nt + (29.0 + 9.0 * nt) * c / 32.0) * (alone ? 1.65 : 1.0);
        if (c == kVCols || x < 0.98 * cost) {
            best = c;
            cost = x;
        }
    }
    return best;
}

// whether a thread per column is the faster mapping for columns that a tile would hold: deep tiles are narrow
// (17 columns at 200 layers), so their recurrences, a lane per column, cost more of the FP64 unit, and with
// enough columns a thread per column keeps it as busy where every column starts on a 32-byte sector.  Tile /
// thread per column, us: 78k columns of 144 layers 1748 / 1781, 148: 1881 / 1824, 200: 2951 / 2467; 29k
// of 156: 807 / 807, 160: 811 / 827, 172: 975 / 889; 22k of 216: 973 / 1117; off the sector, 78k of 201:
// 2970 / 3510
inline bool vdiff_by_column(int n, int L1) {
    return L1 % 4 == 0 && n >= 26000 && L1 >= (n >= 60000 ? 148 : 160);
}

struct VArgs {
    int N2, nl, cols;
    const int *nlev, *ulev;
    const double *zbot, *hn, *ar, *av, *kv, *wi;
    const double2 *rav;  // reciprocals of av (recip64), null: none at hand
    double dt;
};
struct VTracer {
    double *T;
    const double *bc;  // surface flux per node, null: none
};

struct VTile {
    int total, lo, hi;  // items; first and last level of any column
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
        const int l0 = __reduce_min_sync(0xffffffffu, levels ? first_level : 1 << 20);
        const int l1 = __reduce_max_sync(0xffffffffu, levels ? first_level + levels - 1 : 0);
        if (lane == 31) {
            total = s;
            lo = l0;
            hi = l1;
        }
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
    const int L1 = P.nl - 1, nl = P.nl, pad = P.cols | 1;
    const size_t sz = (size_t)L1 * pad;
    double *HB = sm, *ZR = sm + sz, *A = sm + 2 * sz, *C = sm + 3 * sz;  // h then b, Z then the first rhs, a, c
    auto R = [&](int t) { return t == 0 ? ZR : sm + (3 + t) * sz; };
#define FOR_ITEMS                                                                                      \
    _Pragma("unroll 2") for (int i = threadIdx.x; i < S.total; i += kVThreads) {                                           \
        const int j = S.find(i), nz = S.top[j] + i - S.pre[j], x = (nz - 1) * pad + j;               \
        const bool top = i == S.pre[j], bot = i + 1 == S.pre[j + 1];                                   \
        const size_t k = (size_t)(n0 + j) * L1 + nz - 1, kv = (size_t)(n0 + j) * nl + nz - 1;          \
        (void)top; (void)bot; (void)k; (void)kv; (void)x;
    FOR_ITEMS
        HB[x] = P.hn[k];
    }
    __syncthreads();
    // warp 0: depths and pivots; warp 1 + t: tracer t
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    const int r0 = S.top[lane] - 1, r1 = r0 + S.pre[lane + 1] - S.pre[lane] - 1;  // rows of the lane's column
    if (role == 0) {  // bottom depth of every layer (src/oce_ale_tracer.F90:1088-1096)
        double zb = r1 >= r0 ? P.zbot[n0 + lane] : 0.0;
        for (int r = r1; r >= r0; r--) {
            ZR[r * pad + lane] = zb;
            zb = zb + HB[r * pad + lane];
        }
    }
    __syncthreads();
    FOR_ITEMS
        ZR[x] = ZR[x] + HB[x] / 2.0;  // Z_n
    }
    __syncthreads();
    // the interface above layer nz: a(nz) and c(nz - 1)
    auto by_av = [&](double num, size_t i) {
        return P.rav ? sdiv64(num, P.av[i], P.rav[i]) : num / P.av[i];
    };
    FOR_ITEMS
        if (top) {
            A[x] = 0.0;
            C[((S.top[j] - 1) + (S.pre[j + 1] - S.pre[j] - 1)) * pad + j] = 0.0;
        } else {
            const double q = P.kv[kv] * (1.0 / (ZR[x - pad] - ZR[x])) * P.dt, ar = P.ar[kv];
            A[x] = -(q * by_av(ar, kv));
            C[x - pad] = -by_av(q * ar, kv - 1);
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
    // forward elimination (:1406-1414): the pivots m (into HB) and cp (into C), and the tracers a
    // chunk of levels behind; at the top layer a = 0 and cp = tp = 0
    {
        double cp = 0.0, y = 0.0;
        for (int c0 = S.lo - 1; c0 <= S.hi - 1 + kVChunk; c0 += kVChunk) {
            if (role == 0) {
                const int e = min(c0 + kVChunk - 1, r1);
                for (int r = max(c0, r0); r <= e; r++) {
                    const int x = r * pad + lane;
                    const double m = HB[x] - cp * A[x];
                    cp = C[x] / m;
                    C[x] = cp;
                    HB[x] = m;
                }
            }
#pragma unroll
            for (int t = 0; t < NT; t++) {
                if (t >= nt || role != 1 + t) continue;
                double *Rt = R(t);
                const int e = min(c0 - 1, r1);
                for (int r = max(c0 - kVChunk, r0); r <= e; r++) {
                    const int x = r * pad + lane;
                    y = (Rt[x] - y * A[x]) / HB[x];
                    Rt[x] = y;
                }
            }
            __syncthreads();
        }
    }
    // back substitution (:1417-1430); C is 0 at the bottom layer
#pragma unroll
    for (int t = 0; t < NT; t++) {
        if (t >= nt || role != 1 + t) continue;
        double *Rt = R(t), y = 0.0;
        for (int r = r1; r >= r0; r--) {
            const int x = r * pad + lane;
            y = Rt[x] - C[x] * y;
            Rt[x] = y;
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
