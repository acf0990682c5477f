// helm_real.cuh -- P2M, P2L and the evaluation at the points for a positive
// real wavenumber (included by helmholtz.cu).
//
// With k real the Bessel recurrences are real (two FMAs per order where the
// general kernels spend complex products on them), the angle enters only
// through dx/r and dy/r (no atan2, no sincos), and the downward sequence of
// J needs no normalisation: it starts from two values of its ascending
// series at a high order,
//     J_n(x) = (x/2)^n / n! sum_m (-x^2/4)^m / (m! (n+1)...(n+m)),
// so one pass replaces the upward search for the top order, the pass that
// sums the normalisation and the rescaling events.  From order x^2/8 up the
// series' terms are at most e^2 times its sum.
//
// The derivatives of an expansion (mk_mpoleg, mk_mpoleh, helmrouts2d.c:
// 187-292) are sums of the same basis functions with the coefficients
// shifted by one and two orders, so the evaluation accumulates the sums
//   P = C_n E_n, U = a_n C_n+1 E_n, V = b_n C_n-1 E_n,
//   U2 = a_n a_n+1 C_n+2 E_n, V2 = b_n b_n-1 C_n-2 E_n
// (a_n, b_n real) and combines them per point: d/dx = U - V,
// d/dy = i (U + V), dxx = U2 + V2 - k^2 P / 2, dxy = i (U2 - V2),
// dyy = -(U2 + V2 + k^2 P / 2).
#pragma once

constexpr int kRcp = 320;
struct RcpTable {
    double v[kRcp];
    constexpr RcpTable() : v() {
        for (int i = 1; i < kRcp; i++) v[i] = 1.0 / i;
    }
};
__constant__ RcpTable c_rcp = RcpTable();

// Largest k r of a point in its box that jtop takes: the top order x^2/8 + 1
// and its series stay inside the reciprocal table and (x/2)^n / n! above
// 1e-200 at that order.  Larger boxes (levels of more than 9.9 wavelengths)
// keep the general kernels.
constexpr double kRealXMax = 44.0;
constexpr int kRealOrderMax = kRcp - 60;

// Start of the downward sequence j_n = J_n(x) / rs^n, n <= nmax: returns the
// order n (at least nmax, except near x = 0 where the orders above n are
// below 1e-200) and j_n, j_{n+1}.  h = x / (2 rs), u = -x^2 / 4.
__device__ __forceinline__ int jtop(int nmax, double h, double u, double rs, double &jn,
                                    double &jn1) {
    int n = max(nmax, (int)(-0.5 * u) + 1);
    double t = 1.0;
    for (int i = 1; i <= n; i++) {
        const double tn = t * (h * c_rcp.v[i]);
        if (tn < 1e-200) {
            n = i - 1;
            break;
        }
        t = tn;
    }
    double s0 = 1.0, s1 = 1.0, a0 = 1.0, a1 = 1.0;
    for (int m = 1; m < 40; m++) {
        const double um = u * c_rcp.v[m];
        a0 *= um * c_rcp.v[n + m];
        a1 *= um * c_rcp.v[n + 1 + m];
        s0 += a0;
        s1 += a1;
        if (fabs(a0) < 1e-18) break;
    }
    jn = t * s0;
    jn1 = t * (h * c_rcp.v[n + 1]) * s1;
    return n;
}

__device__ __forceinline__ double2 cpow_int(double2 z, int n) {
    double2 r = make_double2(1.0, 0.0);
    while (n > 0) {
        if (n & 1) r = cmul(r, z);
        z = cmul(z, z);
        n >>= 1;
    }
    return r;
}

// Sums v[0..15] over 16 lanes (o < 16 bits of the lane) by halving: at each
// step a lane keeps half of its values and hands the other half over, so 15
// exchanges replace 64; lane i ends with the sum of v[i] in the returned
// value.  W = 32: the two halves of the warp are added too.
template <int W>
__device__ __forceinline__ double halving_sum16(double (&v)[16], int lane, unsigned mask) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (i >= o) break;
            const double keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(mask, send, o);
        }
    }
    if (W == 32) v[0] += __shfl_xor_sync(mask, v[0], 16);
    return v[0];
}

// Adds one lane's sum (lane l < 16: order n(l / 4), component l % 4 of cp.x,
// cp.y, cm.x, cm.y) to the coefficients +n and -n.
__device__ __forceinline__ void put16(double2 *E, int n, int nlo, int nhi, int nd, int c, int l,
                                      double v) {
    if (n < nlo || n > nhi) return;
    const int comp = l & 3;
    if (comp >= 2 && n == 0) return;
    double2 *o = E + (long long)(comp >= 2 ? -n : n) * nd + c;
    double *d = reinterpret_cast<double *>(o) + (comp & 1);
    *d += v;
}

// cp / cm of one source: +n gets pw (q b_n + E1 b_{n-1} - E2 b_{n+1}), -n
// (-1)^n conj(pw) (q b_n + E2 b_{n-1} - E1 b_{n+1}), pw = e^{-i n theta},
// the scales of b_{n-1}, b_{n+1} already in bm, bp (b real or complex).
__device__ __forceinline__ void lin3(double bn, double bm, double bp, double2 q, double2 e1,
                                     double2 e2, double2 &a, double2 &b) {
    const double2 qb = cscal(q, bn);
    a = make_double2(fma(e1.x, bm, fma(-e2.x, bp, qb.x)), fma(e1.y, bm, fma(-e2.y, bp, qb.y)));
    b = make_double2(fma(e2.x, bm, fma(-e1.x, bp, qb.x)), fma(e2.y, bm, fma(-e1.y, bp, qb.y)));
}
__device__ __forceinline__ void lin3(double2 bn, double2 bm, double2 bp, double2 q, double2 e1,
                                     double2 e2, double2 &a, double2 &b) {
    a = cmul(q, bn);
    b = a;
    cfma(a, e1, bm);
    cfma(a, make_double2(-e2.x, -e2.y), bp);
    cfma(b, e2, bm);
    cfma(b, make_double2(-e1.x, -e1.y), bp);
}

// Strengths of one source: q and E1 = (k/2) d conj(V) e^{i theta},
// E2 = (k/2) d V e^{-i theta}, V = v1 + i v2.
__device__ __forceinline__ void src_strengths(int ifc, int ifd, double k, long long kc,
                                              const double2 *charge, const double2 *dipstr,
                                              const double2 *dipvec, double2 em, double2 &q,
                                              double2 &e1, double2 &e2) {
    q = ifc ? charge[kc] : make_double2(0.0, 0.0);
    e1 = e2 = make_double2(0.0, 0.0);
    if (ifd) {
        const double2 d = cscal(dipstr[kc], 0.5 * k), v = dipvec[kc];
        e1 = cmul(d, cmul(cconj(v), cconj(em)));
        e2 = cmul(d, cmul(v, em));
    }
}

// ---------------------------------------------------------------------------
// P2M: a group of W lanes per leaf, lanes = sources, orders downward in
// groups of four whose 16 sums are formed by halving (halving_sum16).
// Bound by the FP64 pipe's about 30 instructions per (source, order) and as
// many shuffles.  2e6 points, zk 200, orders 17-20: 2.13 ms in the general
// kernel (idle half of the lanes in both).
// ---------------------------------------------------------------------------
template <int W>
__global__ void __launch_bounds__(256) helm_p2m_real_kernel(
    int nb, const int *__restrict__ nchild, const int *__restrict__ level,
    const int2 *__restrict__ sse, const double2 *__restrict__ centers,
    const HLevel *__restrict__ lv, const double2 *__restrict__ src,
    const double2 *__restrict__ charge, const double2 *__restrict__ dipstr,
    const double2 *__restrict__ dipvec, int ifc, int ifd, int nd, double k, int lmin,
    double2 *__restrict__ mp) {
    const int lane = threadIdx.x & (W - 1);
    const unsigned gmask = W == 32 ? 0xffffffffu : (0xffffu << (threadIdx.x & 16));
    const int nw = (gridDim.x * blockDim.x) / W;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) / W; b < nb; b += nw) {
        if (nchild[b] != 0) continue;
        const int l = level[b];
        if (l < lmin) continue;
        const HLevel L = lv[l];
        if (!L.flag) continue;
        const int2 r = sse[b];
        if (r.y <= r.x) continue;
        const int p = L.p;
        const double rs = L.rs, rs2 = rs * rs, ri = 1.0 / rs;
        double2 *M = const_cast<double2 *>(coef0(mp, L, b, nd));
        const double2 ctr = centers[b];
        for (int k0 = r.x; k0 < r.y; k0 += W) {
            const int kk = k0 + lane;
            const bool valid = kk < r.y;
            double2 em = make_double2(1.0, 0.0);
            double h = 0.0, x = 0.0;
            if (valid) {
                const double2 sp = src[kk];
                const double dx = sp.x - ctr.x, dy = sp.y - ctr.y;
                const double rr = sqrt(dx * dx + dy * dy);
                if (rr > 0.0) {
                    const double rinv = 1.0 / rr;
                    em = make_double2(dx * rinv, -dy * rinv);
                }
                x = k * rr;
                h = 0.5 * x * ri;
            }
            double jt, jt1;
            const int nt = jtop(p, h, -0.25 * x * x, rs, jt, jt1);
            const double hi = h > 0.0 ? 1.0 / h : 0.0;
            // down to j_{p+1}, j_{p+2} (a start above p + 1)
            double ja = jt, jb = jt1;  // j_m, j_{m+1} at m = max(nt, ...)
            int m = nt;
            for (; m > p + 1; m--) {
                const double jm = fma((double)m * hi, ja, -rs2 * jb);
                jb = ja;
                ja = jm;
            }
            const double2 pw0 = cpow_int(em, p), ep = cconj(em);
            for (int c = 0; c < nd; c++) {
                double2 q = make_double2(0.0, 0.0), e1 = q, e2 = q;
                if (valid)
                    src_strengths(ifc, ifd, k, (long long)kk * nd + c, charge, dipstr, dipvec, em,
                                  q, e1, e2);
                double2 pw = pw0;
                // b0 = j_n, b1 = j_{n+1} at n = p; a lane whose sequence
                // starts at order m < p holds zeros above m + 1
                double b0, b1;
                int ms = m;  // (order of ja)
                if (ms == p + 1) {
                    b1 = ja;
                    b0 = fma((double)ms * hi, ja, -rs2 * jb);
                } else if (ms == p) {
                    b0 = ja;
                    b1 = jb;
                } else {
                    b0 = ms == p - 1 ? jb : 0.0;
                    b1 = 0.0;
                }
                for (int n4 = p; n4 >= 0; n4 -= 4) {
                    double v[16];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const int n = n4 - t;
                        // j_{n-1}
                        double bm = 0.0;
                        if (n >= 1) {
                            if (n <= ms) bm = fma((double)n * hi, b0, -rs2 * b1);
                            else if (n - 1 == ms) bm = ja;
                            else if (n - 2 == ms) bm = jb;
                        }
                        double2 a, bb;
                        lin3(b0, bm * ri, b1 * rs, q, e1, e2, a, bb);
                        double2 cp, cm;
                        if (n > 0) {
                            cp = cmul(a, pw);
                            cm = cmul(bb, cconj(pw));
                            if (n & 1) cm = make_double2(-cm.x, -cm.y);
                        } else {
                            // q j_0 - (E1 + E2) j_1 rs
                            cp = make_double2(fma(-(e1.x + e2.x), b1 * rs, q.x * b0),
                                              fma(-(e1.y + e2.y), b1 * rs, q.y * b0));
                            cm = make_double2(0.0, 0.0);
                        }
                        if (n < 0) cp = cm = make_double2(0.0, 0.0);
                        v[4 * t] = cp.x;
                        v[4 * t + 1] = cp.y;
                        v[4 * t + 2] = cm.x;
                        v[4 * t + 3] = cm.y;
                        pw = cmul(pw, ep);
                        b1 = b0;
                        b0 = bm;
                    }
                    const double sum = halving_sum16<W>(v, lane & 15, gmask);
                    if (lane < 16) put16(M, n4 - (lane >> 2), 0, p, nd, c, lane, sum);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// P2L over list 4: warp per box, lanes = sources, upward H, orders in groups
// of four.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) helm_p2l_real_kernel(
    int nb, const int *__restrict__ level, const int *__restrict__ nlist4,
    const int *__restrict__ list4, const int2 *__restrict__ sse,
    const double2 *__restrict__ centers, const HLevel *__restrict__ lv,
    const double2 *__restrict__ src, const double2 *__restrict__ charge,
    const double2 *__restrict__ dipstr, const double2 *__restrict__ dipvec, int ifc,
    int ifd, int nd, double k, double2 *__restrict__ loc) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb; b += nw) {
        const int n4 = nlist4[b];
        if (n4 == 0) continue;
        const int l = level[b];
        if (l < 2) continue;
        const HLevel L = lv[l];
        if (!L.flag) continue;
        const int p = L.p;
        const double rs = L.rs, rs2 = rs * rs, ri = 1.0 / rs;
        double2 *E = const_cast<double2 *>(coef0(loc, L, b, nd));
        const double2 ctr = centers[b];
        // the sources of all list-4 leaves as one sequence over the lanes
        int tot = 0;
        for (int e = 0; e < n4; e++) {
            const int2 r = sse[list4[b * 5 + e]];
            tot += r.y - r.x;
        }
        for (int k0 = 0; k0 < tot; k0 += 32) {
            int gi = k0 + lane, kk = -1;
            if (gi < tot)
                for (int e = 0; e < n4; e++) {
                    const int2 r = sse[list4[b * 5 + e]];
                    if (gi < r.y - r.x) {
                        kk = r.x + gi;
                        break;
                    }
                    gi -= r.y - r.x;
                }
            const bool valid = kk >= 0;
            double2 em = make_double2(1.0, 0.0), h0 = make_double2(0.0, 0.0), h1 = h0;
            double w = 0.0;  // 2 rs / x
            if (valid) {
                const double2 sp = src[kk];
                const double dx = sp.x - ctr.x, dy = sp.y - ctr.y;
                const double rr2 = dx * dx + dy * dy, rr = sqrt(rr2), rinv = 1.0 / rr;
                em = make_double2(dx * rinv, -dy * rinv);
                const double x = k * rr, s = x * x;
                double2 g;
                if (s < hb::kSMax) hb::hankel01_sq<false>(s, 1.0 / s, h0, g);
                else hankel01_far(s, h0, g);
                h1 = cscal(g, x * rs);
                w = 2.0 * rs * rinv / k;
            }
            for (int c = 0; c < nd; c++) {
                double2 q = make_double2(0.0, 0.0), e1 = q, e2 = q;
                if (valid)
                    src_strengths(ifc, ifd, k, (long long)kk * nd + c, charge, dipstr, dipvec, em,
                                  q, e1, e2);
                double2 pw = make_double2(1.0, 0.0);
                double2 bm = make_double2(0.0, 0.0), b0 = h0, b1 = h1;  // h_{n-1}, h_n, h_{n+1}
                for (int nn = 0; nn <= p; nn += 4) {
                    double v[16];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const int n = nn + t;
                        double2 a, bb, cp, cm;
                        lin3(b0, cscal(bm, rs), cscal(b1, ri), q, e1, e2, a, bb);
                        if (n > 0) {
                            cp = cmul(a, pw);
                            cm = cmul(bb, cconj(pw));
                            if (n & 1) cm = make_double2(-cm.x, -cm.y);
                        } else {
                            cp = cmul(q, b0);
                            cfma(cp, make_double2(-(e1.x + e2.x) * ri, -(e1.y + e2.y) * ri), b1);
                            cm = make_double2(0.0, 0.0);
                        }
                        if (n > p) cp = cm = make_double2(0.0, 0.0);
                        v[4 * t] = cp.x;
                        v[4 * t + 1] = cp.y;
                        v[4 * t + 2] = cm.x;
                        v[4 * t + 3] = cm.y;
                        pw = cmul(pw, em);
                        const double f = w * (double)(n + 1);
                        const double2 b2 = make_double2(fma(f, b1.x, -rs2 * b0.x),
                                                        fma(f, b1.y, -rs2 * b0.y));
                        bm = b0;
                        b0 = b1;
                        b1 = b2;
                    }
                    const double sum = halving_sum16<32>(v, lane & 15, 0xffffffffu);
                    if (lane < 16) put16(E, nn + (lane >> 2), 0, p, nd, c, lane, sum);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// M2P + L2P.  G lanes (a power of two) share a point: they deal its list-3
// expansions among them, the last one adds the local expansion, and their sums
// are added by halving.  G = 1 unless the points leave the chip idle
// (far_lanes): the recurrences are serial, and a few thousand points are a few
// warps per SM.  The coefficients of the orders around n move through a window
// of registers, loaded one order ahead: with derivatives an order takes ten
// coefficients, of which two are new.
// Bound by the recurrences' latency: 0.80 ms with the general kernels, 0.47
// here at 2e6 points, zk 200; 1e5 clustered points 0.44 -> 0.21 ms, 2,001
// points with Hessians 0.21 -> 0.033 ms (one lane per point, coefficients
// loaded where they are used, a launch per point set).
// ---------------------------------------------------------------------------
struct AccR {
    double2 p, u, v, u2, v2;
};

// One expansion's coefficients with the real derivative factors
// a_n = (n >= 0 ? z2 : z1), b_n = (n >= 1 ? z1 : z2).  The window holds
// P[j] = C(n + j - H), M[j] = C(-n + j - H); up() and down() move n by one.
template <int PGH, bool UP>
struct CoefR {
    static constexpr int H = PGH - 1, K = 2 * H + 1;
    const double2 *c0;
    int p, nd;
    double z1, z2;
    double2 P[K], M[K], np, nm;
    __device__ __forceinline__ double2 at(int n) const {
        return (n < -p || n > p) ? make_double2(0.0, 0.0) : c0[(long long)n * nd];
    }
    __device__ __forceinline__ void ahead(int n) {  // what the step from n brings in
        np = at(UP ? n + 1 + H : n - 1 - H);
        nm = at(UP ? -n - 1 - H : -n + 1 + H);
    }
    __device__ __forceinline__ CoefR(const double2 *c, int p_, int nd_, double za, double zb, int n)
        : c0(c), p(p_), nd(nd_), z1(za), z2(zb) {
#pragma unroll
        for (int j = 0; j < K; j++) {
            P[j] = at(n + j - H);
            M[j] = at(-n + j - H);
        }
        ahead(n);
    }
    // to order n (from n - 1, or n + 1 downwards)
    __device__ __forceinline__ void step(int n) {
        constexpr bool pl = UP;  // P moves towards lower indexes
#pragma unroll
        for (int j = 0; j + 1 < K; j++) {
            if (pl) {
                P[j] = P[j + 1];
                M[K - 1 - j] = M[K - 2 - j];
            } else {
                P[K - 1 - j] = P[K - 2 - j];
                M[j] = M[j + 1];
            }
        }
        P[pl ? K - 1 : 0] = np;
        M[pl ? 0 : K - 1] = nm;
        ahead(n);
    }
    __device__ __forceinline__ double2 pos(int d) const { return P[H + d]; }  // C(n + d)
    __device__ __forceinline__ double2 neg(int d) const { return M[H + d]; }  // C(-n + d)
};

// Adds the order +n / -n terms (n >= 0) with the angular factor w^n = wn and
// the radial value b (real J or complex H): E_n = wn b, E_-n = (-1)^n
// conj(wn) b.  For n >= 1: a_n = z2, b_n = z1, a_-n = z1, b_-n = z2; the
// second shifts' products are a_n a_n+1 = z2^2, b_n b_n-1 = z1^2 (z1 z2 at
// n = 1: b_1 b_0), and mirrored for -n.
__device__ __forceinline__ void radial_add(double2 &a, double2 g, double b) {
    a = make_double2(fma(g.x, b, a.x), fma(g.y, b, a.y));
}
__device__ __forceinline__ void radial_add(double2 &a, double2 g, double2 b) { cfma(a, g, b); }

template <int PGH, bool UP, class B>
__device__ __forceinline__ void acc_real(AccR &A, const CoefR<PGH, UP> &C, int n, double2 wn, B b) {
    constexpr int d1 = PGH >= 2 ? 1 : 0, d2 = PGH >= 3 ? 2 : 0;  // (inside the window)
    if (n == 0) {
        radial_add(A.p, C.pos(0), b);
        if (PGH >= 2) {
            radial_add(A.u, cscal(C.pos(d1), C.z2), b);
            radial_add(A.v, cscal(C.pos(-d1), C.z2), b);
        }
        if (PGH >= 3) {
            radial_add(A.u2, cscal(C.pos(d2), C.z2 * C.z2), b);
            radial_add(A.v2, cscal(C.pos(-d2), C.z2 * C.z2), b);
        }
        return;
    }
    const double2 wm = (n & 1) ? make_double2(-wn.x, wn.y) : cconj(wn);  // (-1)^n conj(wn)
    auto two = [&](double2 &S, double2 cp, double fp, double2 cm, double fm) {
        double2 g = cmul(cscal(cp, fp), wn);
        cfma(g, cscal(cm, fm), wm);
        radial_add(S, g, b);
    };
    {
        double2 g = cmul(C.pos(0), wn);
        cfma(g, C.neg(0), wm);
        radial_add(A.p, g, b);
    }
    if (PGH >= 2) {
        two(A.u, C.pos(d1), C.z2, C.neg(d1), C.z1);
        two(A.v, C.pos(-d1), C.z1, C.neg(-d1), C.z2);
    }
    if (PGH >= 3) {
        const double s1 = C.z1 * C.z1, s2 = C.z2 * C.z2, s12 = C.z1 * C.z2;
        // a_-n a_-n+1: z1 z1, or z1 z2 at n = 1; b_n b_n-1 likewise
        const double f = n == 1 ? s12 : s1;
        two(A.u2, C.pos(d2), s2, C.neg(d2), f);
        two(A.v2, C.pos(-d2), f, C.neg(-d2), s2);
    }
}

// Lanes per point: as many (up to 8) as keep the threads of all points within
// what the chip holds at once of this kernel (16 warps per SM).
inline int far_lanes(long long points) {
    int g = 1;
    while (g < 8 && points * g * 2 <= (long long)kNumSM * 16 * 32) g *= 2;
    return g;
}

template <int PGH>
__global__ void __launch_bounds__(128) helm_far_real_kernel(
    HFarSet s0, HFarSet s1, int g0, const int *__restrict__ level,
    const double2 *__restrict__ centers, const int *__restrict__ nlist3,
    const int *__restrict__ list3, const HLevel *__restrict__ lv, int nlevels,
    const double2 *__restrict__ mp, const double2 *__restrict__ loc, int nd, int G, double k,
    int lmin) {
    const bool second = blockIdx.x >= g0;
    const HFarSet X = second ? s1 : s0;
    const long long n = (long long)X.n * G;
    const int blk = blockIdx.x - (second ? g0 : 0), nblk = second ? gridDim.x - g0 : g0;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const unsigned mask = (G == 1 ? 1u : (1u << G) - 1u) << (lane - sub);
    for (long long i = (long long)blk * blockDim.x + threadIdx.x; i < n;
         i += (long long)nblk * blockDim.x) {
        const int t = (int)(i / G);
        const int b = X.leaf[t];
        const int l = level[b];
        if (l < lmin) continue;  // (uniform over a point's lanes)
        const HLevel L = lv[l];
        const double2 x = X.pos[t];
        for (int c = 0; c < nd; c++) {
            AccR A;
            A.p = A.u = A.v = A.u2 = A.v2 = make_double2(0.0, 0.0);
            // M2P over list 3 (boxes of level l + 1)
            if (l + 1 <= nlevels && lv[l + 1].flag) {
                const int nl3 = nlist3[b];
                const HLevel L3 = lv[l + 1];
                const double rs = L3.rs, rs2 = rs * rs;
                const int N = L3.p + PGH - 1;
                for (int e = sub; e < nl3; e += G) {
                    const int jb = list3[b * 20 + e];
                    const double2 cc = centers[jb];
                    const double dx = x.x - cc.x, dy = x.y - cc.y;
                    const double rr = sqrt(dx * dx + dy * dy), rinv = 1.0 / rr;
                    const double2 w = make_double2(dx * rinv, dy * rinv);
                    const double xx = k * rr, s = xx * xx;
                    CoefR<PGH, true> C(coef0(mp, L3, jb, nd) + c, L3.p, nd, 0.5 * k / rs,
                                       0.5 * k * rs, 0);
                    double2 h0, g;
                    if (s < hb::kSMax) hb::hankel01_sq<false>(s, 1.0 / s, h0, g);
                    else hankel01_far(s, h0, g);
                    const double zr = 2.0 * rs * rinv / k;
                    acc_real(A, C, 0, w, h0);
                    double2 hm1 = h0, hc = cscal(g, xx * rs), wn = w;
                    for (int m = 1; m <= N; m++) {
                        C.step(m);
                        acc_real(A, C, m, wn, hc);
                        const double f = zr * (double)m;
                        const double2 hn = make_double2(fma(f, hc.x, -rs2 * hm1.x),
                                                        fma(f, hc.y, -rs2 * hm1.y));
                        hm1 = hc;
                        hc = hn;
                        wn = cmul(wn, w);
                    }
                }
            }
            // L2P of the leaf's own local expansion
            if (l >= 2 && L.flag && sub == G - 1) {
                const double rs = L.rs, rs2 = rs * rs;
                const double2 cc = centers[b];
                const double dx = x.x - cc.x, dy = x.y - cc.y;
                const double rr = sqrt(dx * dx + dy * dy);
                const double2 w = rr > 0.0 ? make_double2(dx / rr, dy / rr) : make_double2(1.0, 0.0);
                const int N = L.p + PGH - 1;
                const double xx = k * rr, h = 0.5 * xx / rs;
                double ja, jb;  // j_m, j_{m+1}
                int m = jtop(N, h, -0.25 * xx * xx, rs, ja, jb);
                const double hi = h > 0.0 ? 1.0 / h : 0.0;
                for (; m > N; m--) {
                    const double jm = fma((double)m * hi, ja, -rs2 * jb);
                    jb = ja;
                    ja = jm;
                }
                // (a sequence that starts below N: the orders above m + 1 are zero)
                const int top = min(m + 1, N);
                CoefR<PGH, false> C(coef0(loc, L, b, nd) + c, L.p, nd, 0.5 * k * rs, 0.5 * k / rs,
                                    top);
                if (m + 1 <= N) {
                    acc_real(A, C, m + 1, cpow_int(w, m + 1), jb);
                    C.step(m);
                }
                double2 wn = cpow_int(w, m);
                const double2 wc = cconj(w);
                for (; m >= 1; m--) {
                    acc_real(A, C, m, wn, ja);
                    const double jm = fma((double)m * hi, ja, -rs2 * jb);
                    jb = ja;
                    ja = jm;
                    wn = cmul(wn, wc);
                    C.step(m - 1);
                }
                acc_real(A, C, 0, wn, ja);
            }
            for (int o = 1; o < G; o <<= 1) {
                auto sum = [&](double2 &z) {
                    z.x += __shfl_xor_sync(mask, z.x, o);
                    z.y += __shfl_xor_sync(mask, z.y, o);
                };
                sum(A.p);
                if (PGH >= 2) {
                    sum(A.u);
                    sum(A.v);
                }
                if (PGH >= 3) {
                    sum(A.u2);
                    sum(A.v2);
                }
            }
            if (sub != 0) continue;
            // i / 4
            auto i4 = [](double2 z) { return make_double2(-0.25 * z.y, 0.25 * z.x); };
            X.pot[(long long)t * nd + c] = i4(A.p);
            if (PGH >= 2) {
                X.grad[((long long)t * 2 + 0) * nd + c] = i4(csub(A.u, A.v));
                X.grad[((long long)t * 2 + 1) * nd + c] = i4(hk::cmuli(cadd(A.u, A.v)));
            }
            if (PGH >= 3) {
                const double2 sm = cadd(A.u2, A.v2), kp = cscal(A.p, 0.5 * k * k);
                X.hess[((long long)t * 3 + 0) * nd + c] = i4(csub(sm, kp));
                X.hess[((long long)t * 3 + 1) * nd + c] = i4(hk::cmuli(csub(A.u2, A.v2)));
                X.hess[((long long)t * 3 + 2) * nd + c] =
                    i4(make_double2(-sm.x - kp.x, -sm.y - kp.y));
            }
        }
    }
}
