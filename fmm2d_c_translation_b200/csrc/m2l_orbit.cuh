// m2l_orbit.cuh -- FP64 M2L with the list-2 offsets folded by quarter turns
// (included by m2l.cu).
//
// The shift of the reference (l2dmploc, laprouts2d.c:886-994) over an offset
// t is L_i += t^-i sum_j B_ij (-1/t)^j M_j with one real matrix B.  For four
// sources at t_s = i^s t_0 (i the imaginary unit) and h^s_j = (-1/t_s)^j M^s_j,
//     t_s^-i = i^(-s i) t_0^-i,   so
//     L_i += t_0^-i sum_j B_ij D_(i mod 4),j,   D_r,j = sum_s i^(-s r) h^s_j :
// the rows of one residue of i mod 4 see one combination of the four
// sources, and B is applied once instead of four times.  The 27 offsets of a
// child position form ten such orbits: the ring of largest distance 2 is
// four full orbits, the outer ones are five pairs and one single.  The
// combinations are a four-point transform per coefficient (16 additions),
// and B's rows are grouped by residue: four tiles of eight rows hold rows
// 0 .. 31 (u-th row of residue r: r + 4 u), as many DMMAs per orbit as a
// plain ordering needs per offset at orders up to 31.  The rows above 31
// (NL of them) are summed by the lanes on the FP64 pipe instead of in tiles
// that would be mostly empty, and added up over the four lanes of a box at
// the end.
//
// A warp takes eight boxes of one segment (columns of the DMMAs) and one
// channel; a step's coefficients are loaded a step ahead (without that the
// loads' latency left the DMMA pipe 10 % busy and the kernel slower than the
// plain form).  Bound by that latency and the loads' wavefronts (53 % of the
// L1 data pipe, DMMA 28 %): order 37, 3e6 uniform points 3.06 -> 1.76 ms,
// order 28, 4e5 clustered points 0.37 -> 0.22 ms, the 8e6 points of a boundary
// curve (about seven sources per box, so most orbits hold one or two) 4.54 ->
// 3.87 ms.  The registers of the sums allow two blocks per SM with the rows
// above 31 and four without (three blocks spill, 2.12 ms at order 37; three
// without those rows 4.03 ms on the curve).
#pragma once

constexpr int kOrbits = 10;
constexpr int kOrbP = 40;  // coefficients covered

struct OrbitTables {
    int slot[4][kOrbits][4];  // [child position][orbit][quarter turns], -1: none
    double2 w1[4][kSlots][kOrbP];   // (-1/t)^j per slot
    double2 w2[4][kOrbits][kOrbP];  // t_0^-i per orbit
    double lt[4][kOrbits];          // ln |t_0|
};

OrbitTables *make_orbit_tables() {
    const SlotTables st = make_slot_tables();
    OrbitTables *o = new OrbitTables;
    for (int c = 0; c < 4; c++) {
        bool used[kSlots] = {false};
        int n = 0;
        auto turn = [&](int k) {  // slot of i t, -1 when not in list 2
            const int x = -st.dy[c][k], y = st.dx[c][k];
            return (x < -3 || x > 3 || y < -3 || y > 3) ? -1 : st.slot_of[c][x + 3][y + 3];
        };
        // full orbits first, then the pairs, then the single
        for (int want = 4; want >= 1; want--)
            for (int k = 0; k < kSlots; k++) {
                if (used[k]) continue;
                int m[4] = {k, -1, -1, -1}, len = 1;
                for (int s = 1; s < 4; s++) {
                    const int q = turn(m[s - 1]);
                    if (q < 0 || q == k) break;
                    m[s] = q;
                    len++;
                }
                if (len != want || n >= kOrbits) continue;
                for (int s = 0; s < 4; s++) {
                    o->slot[c][n][s] = m[s];
                    if (m[s] >= 0) used[m[s]] = true;
                }
                const double tx = st.dx[c][k], ty = st.dy[c][k], tn = 1.0 / (tx * tx + ty * ty);
                const double2 w = make_double2(tx * tn, -ty * tn);
                double2 v = make_double2(1.0, 0.0);
                for (int i = 0; i < kOrbP; i++) {
                    o->w2[c][n][i] = v;
                    v = cmul(v, w);
                }
                o->lt[c][n] = 0.5 * std::log(tx * tx + ty * ty);
                n++;
            }
        for (int k = 0; k < kSlots; k++) {
            const double tx = st.dx[c][k], ty = st.dy[c][k], tn = 1.0 / (tx * tx + ty * ty);
            const double2 w = make_double2(-tx * tn, ty * tn);
            double2 v = make_double2(1.0, 0.0);
            for (int j = 0; j < kOrbP; j++) {
                o->w1[c][k][j] = v;
                v = cmul(v, w);
            }
        }
    }
    return o;
}

// The tables on the current device (built once per device and process).
const OrbitTables *orbit_tables(cudaStream_t s) {
    static std::mutex mu;
    static const OrbitTables *tab[64] = {nullptr};
    int dev;
    FMM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if (!tab[dev]) {
        std::unique_ptr<OrbitTables> h(make_orbit_tables());
        OrbitTables *d = nullptr;
        FMM_CUDA(cudaMalloc(&d, sizeof(OrbitTables)));
        FMM_CUDA(cudaMemcpyAsync(d, h.get(), sizeof(OrbitTables), cudaMemcpyHostToDevice, s));
        FMM_CUDA(cudaStreamSynchronize(s));
        tab[dev] = d;
    }
    return tab[dev];
}

__device__ __forceinline__ double orbit_b(int i, int j, int p, const double *binom) {
    if (i > p || j > p) return 0.0;
    if (i == 0) return j == 0 ? 0.0 : 1.0;
    return j == 0 ? -1.0 / i : binom[(size_t)(i + j - 1) * (kLdc + 1) + (j - 1)];
}

template <int KS, int NL>
__global__ void __launch_bounds__(128, NL > 0 ? 2 : 4) m2l_orbit_kernel(
    SegTable seg, const int *__restrict__ boxes, const int *__restrict__ slots,
    const double *__restrict__ bs, int ndc, int p, const double *__restrict__ binom,
    const OrbitTables *__restrict__ ot, const double2 *__restrict__ mp,
    double2 *__restrict__ loc, int ntiles) {
    // A fragments of the residues' tiles, and the rows above 31
    __shared__ double s_a[4 * KS * 32];
    __shared__ double s_l[NL > 0 ? NL * KS * 4 : 1];
    __shared__ int s_tb[257];
    __shared__ int s_slot[4][kOrbits][4];
    for (int e = threadIdx.x; e < 4 * KS * 32; e += blockDim.x) {
        const int l = e & 31, ks = (e >> 5) % KS, r = (e >> 5) / KS;
        s_a[e] = orbit_b(r + 4 * (l >> 2), ks * 4 + (l & 3), p, binom);
    }
    for (int e = threadIdx.x; e < NL * KS * 4; e += blockDim.x)
        s_l[e] = orbit_b(32 + e / (KS * 4), e % (KS * 4), p, binom);
    for (int e = threadIdx.x; e <= seg.nseg && e < 257; e += blockDim.x) s_tb[e] = seg.tile_base[e];
    for (int e = threadIdx.x; e < 4 * kOrbits * 4; e += blockDim.x)
        (&s_slot[0][0][0])[e] = (&ot->slot[0][0][0])[e];
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int stride = (p + 1) * ndc;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // a tile's channels on neighbouring warps, which share its sectors in L1
    for (int unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < ntiles * ndc;
         unit += nwarps) {
        const int tile = unit / ndc, c = unit - tile * ndc;
        int lo = 0, hi = seg.nseg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_tb[mid] <= tile) lo = mid; else hi = mid;
        }
        const int q0 = seg.start[lo] + (tile - s_tb[lo]) * 8;
        const int qend = seg.start[lo] + seg.count[lo];
        const int cp = seg.cpos[lo];
        const double lr = log(bs[seg.level[lo]]);
        const int qg = q0 + g;
        const bool has_g = qg < qend;
        const int *qs = slots + (size_t)(has_g ? qg : q0) * kSlots;
        const double2 *Mc = mp + c;
        double acc[4][2][2];  // [residue][column][re/im], row residue + 4 g
        double2 accl[NL > 0 ? NL : 1];
        double2 slog = make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 2; e++) acc[r][e][0] = acc[r][e][1] = 0.0;
#pragma unroll
        for (int n = 0; n < NL; n++) accl[n] = make_double2(0.0, 0.0);
        int sn[4];  // the next orbit's sources
        auto members = [&](int o) {
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const int k = s_slot[cp][o][s];
                sn[s] = (k >= 0 && has_g) ? qs[k] : -1;
            }
        };
        members(0);
        for (int o = 0; o < kOrbits; o++) {
            int sb[4];
            bool mine = false;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                sb[s] = sn[s];
                mine = mine || sb[s] >= 0;
            }
            if (o + 1 < kOrbits) members(o + 1);
            if (__ballot_sync(0xffffffffu, mine) == 0) continue;
            // coefficients and weights of a K step, loaded one step ahead
            double2 m[4], w[4], mn[4], wn[4];
            auto load = [&](int ks) {
                const int j = ks * 4 + tig;
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    const bool v = sb[s] >= 0 && j <= p;
                    mn[s] = v ? Mc[(size_t)sb[s] * stride + (size_t)j * ndc] : make_double2(0.0, 0.0);
                    const int k = s_slot[cp][o][s];
                    wn[s] = __ldg(&ot->w1[cp][k >= 0 ? k : 0][j]);
                }
            };
            load(0);
            double tre[4][2], tim[4][2];
            double2 tl[NL > 0 ? NL : 1];
#pragma unroll
            for (int r = 0; r < 4; r++) tre[r][0] = tre[r][1] = tim[r][0] = tim[r][1] = 0.0;
#pragma unroll
            for (int n = 0; n < NL; n++) tl[n] = make_double2(0.0, 0.0);
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    m[s] = mn[s];
                    w[s] = wn[s];
                }
                if (ks + 1 < KS) load(ks + 1);
                double2 h[4];
#pragma unroll
                for (int s = 0; s < 4; s++) h[s] = cmul(m[s], w[s]);
                // D_r = sum_s i^(-s r) h_s
                const double2 a0 = cadd(h[0], h[2]), a1 = csub(h[0], h[2]);
                const double2 b0 = cadd(h[1], h[3]), b1 = csub(h[1], h[3]);
                const double2 D[4] = {cadd(a0, b0), make_double2(a1.x + b1.y, a1.y - b1.x),
                                      csub(a0, b0), make_double2(a1.x - b1.y, a1.y + b1.x)};
                if (ks == 0 && tig == 0) {  // + log|z0| M_0 in row 0
                    const double f = lr + ot->lt[cp][o];
                    slog.x = fma(f, D[0].x, slog.x);
                    slog.y = fma(f, D[0].y, slog.y);
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const double a = s_a[(r * KS + ks) * 32 + lane];
                    dmma(tre[r][0], tre[r][1], a, D[r].x);
                    dmma(tim[r][0], tim[r][1], a, D[r].y);
                }
#pragma unroll
                for (int n = 0; n < NL; n++) {
                    const double b = s_l[(n * KS + ks) * 4 + tig];
                    tl[n].x = fma(b, D[n & 3].x, tl[n].x);
                    tl[n].y = fma(b, D[n & 3].y, tl[n].y);
                }
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const double2 v = __ldg(&ot->w2[cp][o][r + 4 * g]);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    double *a = acc[r][e];
                    a[0] = fma(v.x, tre[r][e], fma(-v.y, tim[r][e], a[0]));
                    a[1] = fma(v.x, tim[r][e], fma(v.y, tre[r][e], a[1]));
                }
            }
#pragma unroll
            for (int n = 0; n < NL; n++) cfma(accl[n], __ldg(&ot->w2[cp][o][32 + n]), tl[n]);
        }
        // store: the first writer of these boxes' local expansions
#pragma unroll
        for (int e = 0; e < 2; e++) {
            // (column 2 tig + e's log sum is in its box's lane of tig 0)
            const double lx = __shfl_sync(0xffffffffu, slog.x, (2 * tig + e) * 4);
            const double ly = __shfl_sync(0xffffffffu, slog.y, (2 * tig + e) * 4);
            if (g == 0) {
                acc[0][e][0] += lx;
                acc[0][e][1] += ly;
            }
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int q = q0 + 2 * tig + e;
            if (q >= qend) continue;
            double2 *Lo = loc + (size_t)boxes[q] * stride + c;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int i = r + 4 * g;
                if (i <= p) Lo[(size_t)i * ndc] = make_double2(acc[r][e][0], acc[r][e][1]);
            }
        }
        if (NL > 0) {
#pragma unroll
            for (int n = 0; n < NL; n++) {
                double2 v = accl[n];
#pragma unroll
                for (int d = 1; d < 4; d <<= 1) {
                    v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
                    v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
                }
                if (tig == 0 && has_g && 32 + n <= p)
                    loc[(size_t)boxes[qg] * stride + (size_t)(32 + n) * ndc + c] = v;
            }
        }
    }
}

template <int KS, int NL>
void launch_orbit(const M2LWork &w, const Tree &T, int ndc, int p, const double *binom,
                  const double2 *mp, double2 *loc, cudaStream_t s) {
    const OrbitTables *ot = orbit_tables(s);
    const int ntiles = w.ntiles(8);
    const int64_t units = (int64_t)ntiles * ndc;
    if (units > INT32_MAX) throw FmmError(4, "M2L: too many boxes and channels");
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((units + 3) / 4, kNumSM * 16));
    m2l_orbit_kernel<KS, NL><<<blocks, 128, 0, s>>>(w.seg(8), w.boxes.get(), w.slots.get(),
                                                    T.d_boxsize.get(), ndc, p, binom, ot, mp, loc,
                                                    ntiles);
    FMM_CHECK_LAUNCH();
}

// Orders 16 .. 39 (below, the plain form's tiles are as few; above, the rows
// beyond 31 would fill tiles of their own).
bool m2l_orbit(const M2LWork &w, const Tree &T, int ndc, int p, const double *binom,
               const double2 *mp, double2 *loc, cudaStream_t s) {
    if (p < 16 || p > 39) return false;
    if (p < 20) launch_orbit<5, 0>(w, T, ndc, p, binom, mp, loc, s);
    else if (p < 24) launch_orbit<6, 0>(w, T, ndc, p, binom, mp, loc, s);
    else if (p < 28) launch_orbit<7, 0>(w, T, ndc, p, binom, mp, loc, s);
    else if (p < 32) launch_orbit<8, 0>(w, T, ndc, p, binom, mp, loc, s);
    else if (p < 36) launch_orbit<9, 4>(w, T, ndc, p, binom, mp, loc, s);
    else if (p < 38) launch_orbit<10, 6>(w, T, ndc, p, binom, mp, loc, s);
    else launch_orbit<10, 8>(w, T, ndc, p, binom, mp, loc, s);
    return true;
}
