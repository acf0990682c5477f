// helm_tables.cuh -- the translation tables of every level of a Helmholtz
// evaluation, built on the device (included by helmholtz.cu).
//
// T(m), m = -N..N, for the shift from center1 to center2 = center1 + d:
// T(0) = B_0, T(m) = zm^m B_m, T(-m) = (-1)^m conj(zm)^m B_m with
// zm = -(dx - i dy) / |d| and B the scaled J (M2M, L2L) or H (M2L) sequence of
// k |d| (h2dmpmp / h2dlocloc / h2dmploc, helmrouts2d.c:736-1042).
//
// The offsets of a level have nine lengths: one of M2M, one of L2L and the
// seven of list 2.  A block takes one of them: thread 0 runs the sequence
// (the recurrences are serial; about 5 to 20 us, all levels at once), the
// threads turn it into the tables of the offsets of that length.  A tenth
// block per level writes the level's real factors.  On the host the tables
// took 1 to 2 ms for a wavenumber, tolerance and domain size not seen before
// and 0.11 ms of copying on every call (10 levels, 2e6 points).
#pragma once

// One level's tables: orders, scales and places (-1: not wanted).
struct HTabLev {
    int Nm, Nl, N2;          // largest |m| of the M2M, L2L and M2L tables
    double hb, bs, rc, rl;   // half a child's side, the side, the child's and own scale
    long long m2m, m2m_f, l2l, l2l_f, m2l, m2l_sc;                          // complex
    long long m2m_s, m2m_pw, m2m_in, m2m_out, l2l_s, l2l_pw, l2l_in, l2l_out, m2l_pw;  // real
    int pc, p;               // the child level's order and the own one
};
constexpr int kTabLevels = 16;  // levels per launch
struct HTabLevs {
    HTabLev l[kTabLevels];
};

// B_0..B_N (H_q(z) rs^q) to T0[q].
__device__ void table_seq_h(int N, double2 z, double rs, double2 *T0) {
    if (hk::cabs_(z) < 1.0e-200) {
        for (int q = 0; q <= N; q++) T0[q] = make_double2(0.0, 0.0);
        return;
    }
    double2 a, b;
    hk::hankel01(z, a, b);
    b = cscal(b, rs);
    T0[0] = a;
    if (N >= 1) T0[1] = b;
    const double2 zr = cscal(cinv(z), 2.0 * rs);
    const double rs2 = rs * rs;
    for (int q = 1; q < N; q++) {
        const double2 c = csub(cmul(cscal(zr, (double)q), b), cscal(a, rs2));
        a = b;
        b = c;
        T0[q + 1] = c;
    }
}

// Miller's recurrence for J_q(z) / rs^q: T0[q] = g_q and T0[-q].x = the
// number of rescalings by 1e-40 before it; the value is g_q 1e-40^(events
// after it) * norm.  Returns norm, and the number of rescalings in `events`.
__device__ double2 table_seq_j(int N, double2 z, double rs, double2 *T0, int &events) {
    events = 0;
    if (hk::cabs_(z) < 1.0e-200) {
        for (int q = N; q >= 0; q--) {
            T0[-q] = make_double2(0.0, 0.0);
            T0[q] = make_double2(q == 0 ? 1.0 : 0.0, 0.0);
        }
        return make_double2(1.0, 0.0);
    }
    const double2 zinv = cinv(z), zr = cscal(zinv, 2.0 * rs);
    const double rs2 = rs * rs;
    const bool lower = z.y < 0.0;
    const int ntop = jb_ntop(N + 3, zinv);
    double2 gp1 = make_double2(0.0, 0.0), gc = make_double2(1.0, 0.0);
    double2 psi = make_double2(0.0, 0.0);  // sum_{q>=1} (-/+ i)^q J_q, to the scale of g
    for (int q = ntop - 1; q >= 1; q--) {
        double2 gm1 = csub(cmul(cscal(zr, (double)q), gc), cscal(gp1, rs2));
        if (gm1.x * gm1.x + gm1.y * gm1.y > 1.0e40) {
            gc = cscal(gc, 1.0e-40);
            gm1 = cscal(gm1, 1.0e-40);
            psi = cscal(psi, 1.0e-40);
            events++;
        }
        psi = cadd(cscal(psi, rs), cmul(gc, zm_pow(q, lower)));
        if (q <= N) {
            T0[q] = gc;
            T0[-q] = make_double2((double)events, 0.0);
        }
        gp1 = gc;
        gc = gm1;
    }
    T0[0] = gc;
    // exp(-/+ i z) = J_0 + 2 sum (-/+ i)^q J_q
    psi = cadd(cscal(psi, 2.0 * rs), gc);
    const double2 ez = lower ? hk::cexp_(make_double2(-z.y, z.x)) : hk::cexp_(make_double2(z.y, -z.x));
    return hk::cdiv_(ez, psi);
}

__device__ __forceinline__ double dpow_int(double x, int n) {
    double r = 1.0;
    while (n > 0) {
        if (n & 1) r *= x;
        x *= x;
        n >>= 1;
    }
    return r;
}

__global__ void __launch_bounds__(128) helm_tables_kernel(const __grid_constant__ HTabLevs levs,
                                                          double2 zk, double2 *__restrict__ ct,
                                                          double *__restrict__ rt) {
    const HTabLev &L = levs.l[blockIdx.x / 10];
    const int role = blockIdx.x % 10;
    if (role == 9) {  // real factors: powers of one base each
        auto powers = [&](long long o, double base, int n) {
            if (o < 0) return;
            for (int e = threadIdx.x; e <= n; e += blockDim.x) rt[o + e] = dpow_int(base, e);
        };
        const double f = L.rc / L.rl;  // (an order's factor from child to parent)
        powers(L.m2m_s, f, L.p);
        powers(L.m2m_pw, L.rc, 2 * L.pc);
        powers(L.m2m_in, L.rc, L.pc);
        powers(L.m2m_out, f / L.rc, L.p);
        powers(L.l2l_s, f, L.pc);
        powers(L.l2l_pw, L.rl, 2 * L.pc);
        powers(L.l2l_in, 1.0 / L.rl, L.p);
        powers(L.l2l_out, f * L.rl, L.pc);
        powers(L.m2l_pw, L.rl, 2 * L.p);
        return;
    }
    const bool hank = role >= 2;
    const int N = role == 0 ? L.Nm : role == 1 ? L.Nl : L.N2;
    const long long fold = role == 0 ? L.m2m_f : role == 1 ? L.l2l_f : -1;
    const long long plain = role == 0 ? L.m2m : role == 1 ? L.l2l : L.m2l;
    if (fold < 0 && plain < 0) return;
    const long long len = 2 * N + 1;
    const double rs = role == 0 ? L.rc : L.rl;
    // the offsets of this length: (x, y) up to signs and order
    const int la = role < 5 ? 2 : 3, lb = role < 5 ? role - 2 : role - 5;
    const double ax = hank ? la * L.bs : L.hb, ay = hank ? lb * L.bs : L.hb;
    const double r = sqrt(ax * ax + ay * ay);
    auto m2l_at = [&](int ix, int iy) { return plain + ((iy + 3) * 7 + (ix + 3)) * len + N; };
    double2 *seq = ct + (fold >= 0 ? fold + N : hank ? m2l_at(la, lb) : plain + N);
    __shared__ double2 s_norm;
    __shared__ int s_events;
    if (threadIdx.x == 0) {
        int events = 0;
        if (hank) {
            table_seq_h(N, cscal(zk, r), rs, seq);
            s_norm = make_double2(1.0, 0.0);
        } else {
            s_norm = table_seq_j(N, cscal(zk, r), rs, seq, events);
        }
        s_events = events;
    }
    __syncthreads();
    for (int q = threadIdx.x; q <= N; q += blockDim.x) {
        double2 B = seq[q];
        if (!hank) {
            const int after = s_events - (q == 0 ? s_events : (int)seq[-q].x);
            for (int e = 0; e < after; e++) B = cscal(B, 1.0e-40);
            B = cmul(B, s_norm);
        }
        const double sg = (q & 1) ? -1.0 : 1.0;
        auto put = [&](long long o, double dx, double dy, double f) {
            const double2 w = cpow_int(make_double2(-dx / r, dy / r), q);
            ct[o + q] = cscal(cmul(w, B), f);
            ct[o - q] = cscal(cmul(cconj(w), B), sg * f);
        };
        if (!hank) {
            // child cs lies at (sx, sy) half sides from the parent; M2M shifts
            // the other way
            const double s = role == 0 ? -L.hb : L.hb;
            if (fold >= 0) {
                put(fold + N, -s, -s, dpow_int(rs, q));
            } else {
                for (int cs = 0; cs < 4; cs++)
                    put(plain + cs * len + N, (cs & 1) ? s : -s, (cs & 2) ? s : -s, 1.0);
            }
            continue;
        }
        const double sc = L.m2l_sc >= 0 ? 1.0 / dpow_int(rs, q) : 0.0;
        for (int k = 0; k < 8; k++) {
            // signs and order of (la, lb); the repeated ones write the same
            int ix = (k & 4) ? lb : la, iy = (k & 4) ? la : lb;
            if (k & 1) ix = -ix;
            if (k & 2) iy = -iy;
            const long long o = m2l_at(ix, iy);
            put(o, ix * L.bs, iy * L.bs, 1.0);
            if (L.m2l_sc >= 0) put(L.m2l_sc + (o - plain), ix * L.bs, iy * L.bs, sc);
        }
    }
    // offsets inside list 1
    if (role == 2)
        for (int e = threadIdx.x; e < 9 * len; e += blockDim.x) {
            const long long o = ((e / len / 3 + 2) * 7 + e / len % 3 + 2) * len + e % len;
            ct[plain + o] = make_double2(0.0, 0.0);
            if (L.m2l_sc >= 0) ct[L.m2l_sc + o] = make_double2(0.0, 0.0);
        }
}
