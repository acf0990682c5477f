// helm_shift.cuh -- M2M and L2L with the four children folded by quarter
// turns (included by helmholtz.cu).
//
// The children of a box lie at quarter turns of one another around its
// center, and a turn by pi / 2 multiplies the translation table by
// T_s(q) = i^(-s q) T_0(q) (q = i - j, i the imaginary unit).  So
//   M2M:  out_i = sum_j T_0(i - j) D_((i - j) mod 4),j ,
//         D_m,j = sum_s i^(-s m) M^s_j
//   L2L:  out^s_i = i^(-s i) sum_c i^(s c) P_c,i ,
//         P_c,i = sum_(j mod 4 = c) L_j T_0(i - j) :
// one pass over the table instead of four, with the children's four-point
// transforms on either side.  The powers of the scale that weight the terms
// (|j| + |i-j| - |i| and |i-j| + |i| - |j|) are folded into the input, the
// table and the output where they stay inside the FP64 range; other levels
// keep the general kernels.
//
// A block takes the boxes with children among a range of its level, kShU
// (box, density) units at a time: the units' transforms are staged in shared
// memory, and a thread sums one output of kShR units, so a table entry
// (four shared-memory wavefronts per warp) serves kShR products.  Before,
// a thread per output read the table and the weights per child from L1/L2:
// 0.85 ms (M2M) and 0.73 ms (L2L) at 2e6 points, zk 200.
#pragma once

constexpr int kShThreads = 128;
constexpr int kShR = 4;

// Child (reference numbering) at s quarter turns from child 0.
__device__ __forceinline__ int turn_child(int s) { return s == 2 ? 3 : (s == 3 ? 2 : s); }

// i^k z
__device__ __forceinline__ double2 imul(double2 z, int k) {
    k &= 3;
    if (k == 1) return make_double2(-z.y, z.x);
    if (k == 2) return make_double2(-z.x, -z.y);
    if (k == 3) return make_double2(z.y, -z.x);
    return z;
}

// Units of a block's pass: (box, density) pairs whose outputs fill the block.
__host__ __device__ __forceinline__ int shift_units(int w2) {
    const int g = w2 < kShThreads ? kShThreads / w2 : 1;
    return g * kShR;
}

// The boxes of [lo, hi) that shift_list keeps, in order, in shared memory.
template <class Keep>
__device__ __forceinline__ int shift_list(int lo, int hi, Keep keep, int *list) {
    __shared__ int s_n[kShThreads / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int n = 0;
    for (int b0 = lo; b0 < hi; b0 += kShThreads) {
        const int b = b0 + (int)threadIdx.x;
        const bool k = b < hi && keep(b);
        const unsigned m = __ballot_sync(0xffffffffu, k);
        __syncthreads();
        if (lane == 0) s_n[warp] = __popc(m);
        __syncthreads();
        int at = n + __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < kShThreads / 32; w++) {
            if (w < warp) at += s_n[w];
            n += s_n[w];
        }
        if (k) list[at] = b;
    }
    __syncthreads();
    return n;
}

constexpr int kShRange = 256;  // most boxes of a block's range

// M2M for the parents [lo, hi) of level l; T: scaled table of child 0
// (entry 0 at T + N), in / out: factors of the input and output orders.
__global__ void __launch_bounds__(kShThreads) helm_m2m_fold_kernel(
    int lo, int hi, int range, int nd, const int *__restrict__ nchild,
    const int *__restrict__ child, const int2 *__restrict__ sse, const HLevel *__restrict__ lv,
    int l, const double2 *__restrict__ T, const double *__restrict__ fin,
    const double *__restrict__ fout, double2 *__restrict__ mp) {
    extern __shared__ __align__(16) double2 sh_sm[];
    __shared__ int list[kShRange];
    const HLevel Lp = lv[l], Lc = lv[l + 1];
    const int n2 = Lp.p, n1 = Lc.p, N = n1 + n2, w1 = 2 * n1 + 1, w2 = 2 * n2 + 1;
    const int U = shift_units(w2);
    double2 *sT = sh_sm, *sD = sT + 2 * N + 1;  // sD[(unit w1 + j) 4 + m]
    for (int e = threadIdx.x; e < 2 * N + 1; e += kShThreads) sT[e] = T[e];
    const int r0 = lo + blockIdx.x * range;
    const int n = shift_list(r0, min(hi, r0 + range), [&](int b) { return nchild[b] != 0; }, list);
    const int units = n * nd;
    for (int u0 = 0; u0 < units; u0 += U) {
        const int nu = min(U, units - u0);
        __syncthreads();
        for (int e = threadIdx.x; e < U * w1; e += kShThreads) {
            const int u = e / w1, j = e - u * w1 - n1;
            double2 M[4];
#pragma unroll
            for (int s = 0; s < 4; s++) M[s] = make_double2(0.0, 0.0);
            if (u < nu) {
                const int b = list[(u0 + u) / nd], c = (u0 + u) % nd;
                const double f = fin[abs(j)];
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    const int cb = child[4 * b + turn_child(s)];
                    const int2 r = sse[cb];
                    if (r.y > r.x) M[s] = cscal(coef0(mp, Lc, cb, nd)[(long long)j * nd + c], f);
                }
            }
            const double2 a0 = cadd(M[0], M[2]), a1 = csub(M[0], M[2]);
            const double2 b0 = cadd(M[1], M[3]), b1 = csub(M[1], M[3]);
            double2 *D = sD + (size_t)e * 4;
            D[0] = cadd(a0, b0);
            D[1] = make_double2(a1.x + b1.y, a1.y - b1.x);
            D[2] = csub(a0, b0);
            D[3] = make_double2(a1.x - b1.y, a1.y + b1.x);
        }
        __syncthreads();
        for (int it = threadIdx.x; it < w2 * (U / kShR); it += kShThreads) {
            const int g = it / w2, i = it - g * w2 - n2;
            if (g * kShR >= nu) continue;
            double2 acc[kShR];
#pragma unroll
            for (int r = 0; r < kShR; r++) acc[r] = make_double2(0.0, 0.0);
            const double2 *D = sD + (size_t)g * kShR * w1 * 4;
            for (int j = 0; j < w1; j++) {  // order j - n1
                const int q = i - (j - n1);
                const double2 t = sT[N + q];
                const double2 *d = D + j * 4 + (q & 3);
#pragma unroll
                for (int r = 0; r < kShR; r++) cfma(acc[r], d[(size_t)r * w1 * 4], t);
            }
            const double f = fout[abs(i)];
#pragma unroll
            for (int r = 0; r < kShR; r++) {
                const int u = g * kShR + r;
                if (u >= nu) break;
                coef0(mp, Lp, list[(u0 + u) / nd], nd)[(long long)i * nd + (u0 + u) % nd] =
                    cscal(acc[r], f);
            }
        }
    }
}

// L2L from the boxes [lo, hi) of level l to their children.
__global__ void __launch_bounds__(kShThreads) helm_l2l_fold_kernel(
    int lo, int hi, int range, int nd, const int *__restrict__ nchild,
    const int *__restrict__ child, const HLevel *__restrict__ lv, int l,
    const double2 *__restrict__ T, const double *__restrict__ fin,
    const double *__restrict__ fout, double2 *__restrict__ loc) {
    extern __shared__ __align__(16) double2 sh_sm[];
    __shared__ int list[kShRange];
    const HLevel Lp = lv[l], Lc = lv[l + 1];
    const int n1 = Lp.p, n2 = Lc.p, N = n1 + n2, w1 = 2 * n1 + 1, w2 = 2 * n2 + 1;
    const int U = shift_units(w2);
    double2 *sT = sh_sm, *sL = sT + 2 * N + 1;  // sL[unit w1 + j]
    for (int e = threadIdx.x; e < 2 * N + 1; e += kShThreads) sT[e] = T[e];
    const int r0 = lo + blockIdx.x * range;
    const int n = shift_list(r0, min(hi, r0 + range), [&](int b) { return nchild[b] != 0; }, list);
    const int units = n * nd;
    for (int u0 = 0; u0 < units; u0 += U) {
        const int nu = min(U, units - u0);
        __syncthreads();
        for (int e = threadIdx.x; e < U * w1; e += kShThreads) {
            const int u = e / w1, j = e - u * w1 - n1;
            double2 v = make_double2(0.0, 0.0);
            if (u < nu)
                v = cscal(coef0(loc, Lp, list[(u0 + u) / nd], nd)[(long long)j * nd + (u0 + u) % nd],
                          fin[abs(j)]);
            sL[e] = v;
        }
        __syncthreads();
        for (int it = threadIdx.x; it < w2 * (U / kShR); it += kShThreads) {
            const int g = it / w2, i = it - g * w2 - n2;
            if (g * kShR >= nu) continue;
            // P[r][c]: the terms of order j with (j + n1) mod 4 = c
            double2 P[kShR][4];
#pragma unroll
            for (int r = 0; r < kShR; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) P[r][c] = make_double2(0.0, 0.0);
            const double2 *Lu = sL + (size_t)g * kShR * w1;
            for (int j0 = 0; j0 < w1; j0 += 4) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int j = j0 + c;
                    if (j >= w1) break;
                    const double2 t = sT[N + i - (j - n1)];
#pragma unroll
                    for (int r = 0; r < kShR; r++) cfma(P[r][c], Lu[r * w1 + j], t);
                }
            }
            const double f = fout[abs(i)];
#pragma unroll
            for (int r = 0; r < kShR; r++) {
                const int u = g * kShR + r;
                if (u >= nu) break;
                const int b = list[(u0 + u) / nd], ch = (u0 + u) % nd;
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    // i^(-s i) sum_c i^(s (c - n1)) P_c
                    double2 v = P[r][0];
#pragma unroll
                    for (int c = 1; c < 4; c++) v = cadd(v, imul(P[r][c], s * c));
                    v = cscal(imul(v, -s * (n1 + i)), f);
                    double2 *o = coef0(loc, Lc, child[4 * b + turn_child(s)], nd) +
                                 (long long)i * nd + ch;
                    *o = cadd(*o, v);
                }
            }
        }
    }
}
