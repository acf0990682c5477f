// helm_bessel.cuh -- H0 and H1 of a positive real argument from one table of
// polynomials in its square.
//
// With s = x^2 the functions of the Helmholtz near field are, up to the
// logarithm and the pole, entire in s (Abramowitz & Stegun 9.1.10-9.1.13):
//     J0 = A(s)            Y0 = C(s) + ln(s) A(s) / pi
//     J1 / x = B(s)        Y1 / x = D(s) + ln(s) B(s) / pi - 2 / (pi s)
// so one table of the four Taylor polynomials of degree 8 about the centers
// of the intervals of width 2 serves every pair with s < 256 (x < 16): 32
// FMAs, one logarithm and one reciprocal, no square root and no branch.
// The first term left out of A is below (1/4)^9 / 9!^2 = 3e-17 everywhere
// (d^m A / ds^m = (-1/2)^m J_m(x) / x^m, largest at s = 0), and C, D, B are
// as close.  The coefficients come from the power series, re-expanded about
// every center in double-double arithmetic on the host (the series cancels
// up to e^16 at s = 256).
//
// Before, the pair evaluated CUDA's j0, j1, y0 and y1 below x = 8 (four
// separate calls, two of them with their own logarithm, each branching on
// the argument) and the continued fraction above: 4.72 ms of near field at
// 2e6 points, zk 200 (1.4e8 pairs), about 640 FP64 instructions per pair;
// with the table 2.12 ms and, with its first row in constant memory, 1.76 ms
// (FP64 pipe and latency: 16 warps per SM at 122-128 registers).
#pragma once

#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "pairmath.cuh"

namespace fmm2d {
namespace hb {

constexpr int kDeg = 8;         // polynomial degree
constexpr int kIntervals = 128; // of width 2 in s
constexpr double kSMax = 256.0;
// double2 per interval: (A, B) and (C, D) of every power, and one of padding
// (an odd number of 16-byte words, so lanes of different intervals spread
// over the banks)
constexpr int kRow = 2 * (kDeg + 1) + 1;

__device__ double2 g_tab[kIntervals * kRow];

// The first interval's row once more, as constant operands of the FMAs.
__constant__ double2 c_tab0[kRow];

// h0 = H0(x), g = H1(x) / x for x = sqrt(s), 0 < s < 256; si = 1 / s.
//
// NEAR: lanes that are all below s = 2 -- the near field of leaves smaller than
// about a tenth of a wavelength, which is most near fields -- take the row from
// constant memory, since the 18 table loads of a pair kept the load unit busier
// (73 %) than the FP64 pipe (39 %), and ln s comes from pairmath.cuh: 2.13 ->
// 1.76 ms at 2e6 points, zk 200; 0.22 -> 0.19 ms at 1e5 clustered points.  (The
// expansions' evaluation, bound by its recurrences, took 0.47 -> 0.51 ms with
// the same.)
template <bool NEAR>
__device__ __forceinline__ void hankel01_sq(double s, double si, double2 &h0, double2 &g) {
    const int iv = (int)(s * 0.5);
    const double t = s - (double)(2 * iv + 1);
    double2 ab, cd;
    if (NEAR && __all_sync(__activemask(), iv == 0)) {
        ab = c_tab0[0];
        cd = c_tab0[1];
#pragma unroll
        for (int m = 1; m <= kDeg; m++) {
            ab.x = fma(ab.x, t, c_tab0[2 * m].x);
            ab.y = fma(ab.y, t, c_tab0[2 * m].y);
            cd.x = fma(cd.x, t, c_tab0[2 * m + 1].x);
            cd.y = fma(cd.y, t, c_tab0[2 * m + 1].y);
        }
    } else {
        const double2 *__restrict__ r = g_tab + iv * kRow;
        ab = __ldg(r);
        cd = __ldg(r + 1);
#pragma unroll
        for (int m = 1; m <= kDeg; m++) {
            const double2 u = __ldg(r + 2 * m), v = __ldg(r + 2 * m + 1);
            ab.x = fma(ab.x, t, u.x);
            ab.y = fma(ab.y, t, u.y);
            cd.x = fma(cd.x, t, v.x);
            cd.y = fma(cd.y, t, v.y);
        }
    }
    const double lg = NEAR ? half_ln_any(s) * 0.63661977236758134308
                           : log(s) * 0.31830988618379067154;
    h0 = make_double2(ab.x, fma(lg, ab.x, cd.x));
    g = make_double2(ab.y, fma(si, -0.63661977236758134308, fma(lg, ab.y, cd.y)));
}

// ---------------------------------------------------------------------------
// Host: the table.
// ---------------------------------------------------------------------------
struct DD {
    double h, l;
};
inline DD dd_norm(double a, double b) {
    const double s = a + b;
    return {s, b - (s - a)};
}
inline DD dd_add(DD a, DD b) {
    const double s = a.h + b.h, v = s - a.h;
    const double e = (a.h - (s - v)) + (b.h - v);
    return dd_norm(s, e + a.l + b.l);
}
inline DD dd_mul(DD a, DD b) {
    const double p = a.h * b.h, e = std::fma(a.h, b.h, -p);
    return dd_norm(p, e + a.h * b.l + a.l * b.h);
}
inline DD dd_div(DD a, double b) {
    const double q = a.h / b;
    const double r = std::fma(-q, b, a.h) + a.l;
    return dd_norm(q, r / b);
}

inline std::vector<double2> make_table() {
    constexpr int K = 96;  // power-series terms: (s/4)^k / k!^2 < 1e-60 at s = 256
    const double gl = 0.57721566490153286061 - 0.69314718055994530942;  // gamma - ln 2
    const double two_pi = 0.63661977236758134308;                      // 2 / pi
    // f[0..3][k]: A, B and the parts of C, D with harmonic numbers
    std::vector<DD> f[4];
    for (auto &v : f) v.resize(K);
    DD a{1.0, 0.0}, hk{0.0, 0.0};
    for (int k = 0; k < K; k++) {
        if (k > 0) {
            a = dd_div(dd_div(a, -4.0 * k), (double)k);
            hk = dd_add(hk, dd_div({1.0, 0.0}, (double)k));
        }
        const DD b = dd_div(a, 2.0 * (k + 1));  // (1/2) (-1/4)^k / (k! (k+1)!)
        const DD h2 = dd_add(hk, dd_div({0.5, 0.0}, (double)(k + 1)));  // (H_k + H_k+1) / 2
        f[0][k] = a;
        f[1][k] = b;
        f[2][k] = dd_mul(a, hk);
        f[3][k] = dd_mul(b, h2);
    }
    std::vector<double2> tab((size_t)kIntervals * kRow, make_double2(0.0, 0.0));
    for (int iv = 0; iv < kIntervals; iv++) {
        const DD c{2.0 * iv + 1.0, 0.0};
        double co[4][kDeg + 1];
        for (int q = 0; q < 4; q++) {
            // Taylor coefficients about c by repeated synthetic division
            std::vector<DD> w = f[q];
            for (int m = 0; m <= kDeg; m++) {
                for (int k = K - 2; k >= m; k--) w[k] = dd_add(w[k], dd_mul(w[k + 1], c));
                co[q][m] = w[m].h;
            }
        }
        for (int m = 0; m <= kDeg; m++) {
            double2 *o = &tab[(size_t)iv * kRow + 2 * (kDeg - m)];
            o[0] = make_double2(co[0][m], co[1][m]);
            o[1] = make_double2(two_pi * (gl * co[0][m] - co[2][m]),
                                two_pi * (gl * co[1][m] - co[3][m]));
        }
    }
    return tab;
}

// Puts the table on the current device, once per device and process.  On the
// call's own stream and waited for: the library's streams do not order with
// the legacy one, and a pageable copy there may return before it has landed.
inline void ensure_table(cudaStream_t s) {
    static std::mutex mu;
    static std::vector<char> done;
    static std::vector<double2> tab;
    int dev = 0;
    FMM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    if (done[dev]) return;
    if (tab.empty()) tab = make_table();
    FMM_CUDA(cudaMemcpyToSymbolAsync(g_tab, tab.data(), tab.size() * sizeof(double2), 0,
                                     cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaMemcpyToSymbolAsync(c_tab0, tab.data(), sizeof(c_tab0), 0,
                                     cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaStreamSynchronize(s));
    done[dev] = 1;
}

}  // namespace hb
}  // namespace fmm2d
