// fp64_arith.cuh -- FP64 helpers of the plain form: the reference's results with fewer
// instructions on the FP64 pipe.
//
// sm_103a issues one FP64 warp instruction per SM every 19 cycles (measured over
// the stages of the form; one warp alone, every 64), so a compare, a maximum or a select done
// in integer instructions costs next to nothing beside one FP64 add, and a division (the time of 9
// FP64 instructions) is the most expensive operation of the form.  Everything here returns the bits of
// the plain expression it replaces (zeros may differ in sign; quotients below 2^-600 take the
// plain division).
#pragma once
#include <cuda_runtime.h>

namespace fesom {

__device__ __forceinline__ bool neg64(double x) { return __double2hiint(x) < 0; }
__device__ __forceinline__ bool nonfinite64(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool nan64(double x) {
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ bool zero64(double x) { return ((unsigned long long)__double_as_longlong(x) << 1) == 0ull; }

// order-preserving integer image of a number (not a NaN): x < y as FP64 is key(x) < key(y), up to
// the sign of zero; the map is its own inverse
__device__ __forceinline__ long long key64(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
__device__ __forceinline__ double unkey64(long long k) {
    return __longlong_as_double(k ^ (long long)((unsigned long long)(k >> 63) >> 1));
}
// a < b ? a : b on integers; either a NaN: b, as the FP64 comparison
__device__ __forceinline__ double min64(double a, double b) {
    return (!nan64(a) && !nan64(b) && key64(a) < key64(b)) ? a : b;
}

// 1/y as an unevaluated sum h + l: h = RN(1/y), l = (1 - y h) h.  Divisors outside 2^+-250 give
// NaNs, which send sdiv to the plain division.
__device__ __forceinline__ double2 recip64(double y) {
    const int e = (__double2hiint(y) >> 20) & 0x7ff;
    if (e < 1023 - 250 || e > 1023 + 250) {
        const double q = __longlong_as_double(0x7ff8000000000000ll);
        return make_double2(q, q);
    }
    const double h = 1.0 / y;
    return make_double2(h, __fma_rn(-y, h, 1.0) * h);
}
// 2^-600 <= |q| < 2^600
__device__ __forceinline__ bool mid_range64(double q) {
    return (unsigned)((__double2hiint(q) & 0x7fffffff) - 0x1a700000) < 0x4b000000u;
}
// a quotient outside the middle range: a zero numerator, or the plain division
__device__ __forceinline__ double div_edge64(double x, double y, bool y_mid) {
    if (y_mid && zero64(x))
        return __longlong_as_double((__double_as_longlong(x) ^ __double_as_longlong(y)) & (1ll << 63));
    return x / y;
}
// RN(x / y) with r = recip64(y): x (h + l) is within a rounding of x/y (a faithful quotient), the
// remainder x - y q is then exact and q + (x - y q) h rounds correctly (P. Markstein, Computation
// of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).
// 4 FP64 instructions instead of 9.
__device__ __forceinline__ double sdiv64(double x, double y, double2 r) {
    double q = __fma_rn(x, r.x, __dmul_rn(x, r.y));
    q = __fma_rn(__fma_rn(-y, q, x), r.x, q);
    if (!mid_range64(q)) q = div_edge64(x, y, !nan64(r.x));
    return q;
}
// RN(x / y) for y = 3 2^k: RN(1/y) is a third of an ulp below 1/y, so RN(x RN(1/y)) is already
// within one ulp of x/y and one remainder step rounds correctly.  3 FP64 instructions.
template <int Y>
__device__ __forceinline__ double div_3x2k(double x) {
    static_assert(Y == 3 || Y == 6 || Y == 12, "a power of two times three");
    constexpr double y = (double)Y, h = 1.0 / y;
    double q = __dmul_rn(x, h);
    q = __fma_rn(__fma_rn(-y, q, x), h, q);
    if (!mid_range64(q)) q = div_edge64(x, y, true);
    return q;
}

}  // namespace fesom
