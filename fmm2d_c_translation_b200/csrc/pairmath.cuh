// pairmath.cuh -- reciprocal and logarithm of the FP64 near-field pairs.
//
// A pair of the Laplace / Cauchy near field needs 1 / r^2 and (with charges)
// ln r^2 of a positive normal number.  The general division and log() check
// for every special operand; here
//   * rcp_pos: PTX's rcp.approx.ftz.f64 and two Newton steps
//     y += y (1 - x y);
//   * half_ln_pos: x = 2^e m, m in [0.75, 1.5), one of 64 intervals of m by
//     its leading bits, each with a constant c near 1/m and -ln(c) / 2 in a
//     table, and ln(m c) by its Taylor series in u = m c - 1, |u| < 1/64,
//     up to u^8 (u^9 / 9 < 7e-18); c = 1 next to m = 1, so the result keeps
//     its relative accuracy there (P. T. P. Tang's table-driven scheme, ACM
//     TOMS 16, 1990).
#pragma once

#include <cuda_runtime.h>

namespace fmm2d {

constexpr int kLnEntries = 64;

constexpr double const_ln(double x) {  // 2 atanh((x - 1) / (x + 1))
    const double t = (x - 1.0) / (x + 1.0), t2 = t * t;
    double s = 0.0, w = t;
    for (int k = 1; k < 60; k += 2) {
        s += w / k;
        w *= t2;
    }
    return 2.0 * s;
}

// (aligned for the 16-byte load of an entry)
struct alignas(sizeof(double2)) LnTable {
    double v[2 * kLnEntries];  // c, -ln(c) / 2
    constexpr LnTable() : v() {
        for (int i = 0; i < kLnEntries; i++) {
            // interval i: 32 of width 1/128 in [0.75, 1), 32 of 1/64 in [1, 1.5)
            const double mid = i < 32 ? 0.75 + (i + 0.5) / 128.0 : 1.0 + (i - 32 + 0.5) / 64.0;
            const double c = (i == 31 || i == 32) ? 1.0 : 1.0 / mid;
            v[2 * i] = c;
            v[2 * i + 1] = -0.5 * const_ln(c);
        }
    }
};
static __device__ LnTable g_ln_table = LnTable();
static_assert(alignof(decltype(g_ln_table)) >= alignof(double2), "entries are read as double2");

__device__ __forceinline__ double rcp_pos(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

__device__ __forceinline__ double half_ln_pos(double x) {
    const int hi = __double2hiint(x), t = hi - 0x3fe80000;
    const int e = t >> 20, i = (t >> 14) & (kLnEntries - 1);
    const double m = x * __hiloint2double((1023 - e) << 20, 0);  // (a NaN stays one)
    const double2 c = __ldg(reinterpret_cast<const double2 *>(g_ln_table.v) + i);
    const double u = fma(m, c.x, -1.0);
    // ln(1 + u) / 2
    double q = -1.0 / 16.0;
    q = fma(q, u, 1.0 / 14.0);
    q = fma(q, u, -1.0 / 12.0);
    q = fma(q, u, 1.0 / 10.0);
    q = fma(q, u, -1.0 / 8.0);
    q = fma(q, u, 1.0 / 6.0);
    q = fma(q, u, -1.0 / 4.0);
    q = fma(q, u, 0.5);
    return fma(q, u, fma((double)e, 0.34657359027997265471, c.y));
}

// The same for any number, outside the inner loops.
__device__ __forceinline__ bool is_normal_pos(double x) { return x >= 2.3e-308 && x <= 1e307; }
__device__ __forceinline__ double rcp_any(double x) {
    return is_normal_pos(x) ? rcp_pos(x) : 1.0 / x;
}
__device__ __forceinline__ double half_ln_any(double x) {
    return is_normal_pos(x) ? half_ln_pos(x) : 0.5 * log(x);
}

}  // namespace fmm2d
