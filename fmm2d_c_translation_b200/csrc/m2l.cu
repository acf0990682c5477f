// m2l.cu -- M2L over list 2 on the FP64 tensor cores (mma.sync m8n8k4 f64).
//
// The reference's multipole-to-local shift (l2dmploc,
// c_translation/src/laprouts2d.c:886-994) of a source box at c1 to a
// target box at c2 of the same level (box size r) factors as
//
//     L_i += w2^i [ B h~ ]_i  (+ log|z0| h~_0 for i = 0),  h~_j = w1^j M_j,
//
// with z0 = c1 - c2 = r t, w1 = -1/t, w2 = 1/t and the fixed real matrix
//     B_00 = 0,  B_0j = 1 (j >= 1),  B_i0 = -1/i,  B_ij = C(i+j-1, j-1).
// In a list-2 pair t is one of 40 lattice offsets, and the 8 target boxes
// of a tile that sit at the same position in their parents share the same
// 27 possible offsets.  A warp therefore owns 8 such boxes, walks the 27
// offsets, and for each one multiplies B (the A operand, fixed, staged in
// shared memory) by the 8 scaled source multipoles (the B operand, one
// column per box) with DMMA, then applies w2^i and accumulates the locals
// in registers.  Each box's local expansion has one writer (no atomics).
//
// Boxes are grouped into tiles by (level, child position) with one radix
// sort; the source of every (target, offset) slot is found once from
// list 2.  If any list-2 entry falls outside the 27 slots (not expected of
// the reference's trees) the caller falls back to the per-box kernel.
#include "laplace.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <mutex>
#include <stdlib.h>
#include <string.h>
#include <type_traits>
#include <vector>

namespace fmm2d {

namespace {

constexpr int kSlots = 27;

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// The 27 lattice offsets (dx, dy) of list 2 for a box at child position
// cpos (bit 0: right half of the parent, bit 1: upper half), in a fixed
// order; slot_of maps (cpos, dx + 3, dy + 3) to the slot or -1.
struct SlotTables {
    int dx[4][kSlots], dy[4][kSlots];
    int slot_of[4][7][7];
};

SlotTables make_slot_tables() {
    SlotTables t;
    for (int c = 0; c < 4; c++) {
        for (int a = 0; a < 7; a++)
            for (int b = 0; b < 7; b++) t.slot_of[c][a][b] = -1;
        const int px = c & 1, py = (c >> 1) & 1;
        int k = 0;
        for (int dy = -2 - py; dy <= 3 - py; dy++)
            for (int dx = -2 - px; dx <= 3 - px; dx++) {
                if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1) continue;
                t.dx[c][k] = dx;
                t.dy[c][k] = dy;
                t.slot_of[c][dx + 3][dy + 3] = k;
                k++;
            }
    }
    return t;
}

__constant__ int c_slot_dx[4][kSlots];
__constant__ int c_slot_dy[4][kSlots];
__constant__ int c_slot_of[4][7][7];

// Segment = (level, child position); tiles of 8 boxes within a segment.
struct SegTable {
    const int *tile_base;  // nseg + 1
    const int *start;      // nseg, into the sorted box list
    const int *count;      // nseg
    const int *level;      // nseg
    const int *cpos;       // nseg
    int nseg;
};

// NT > 0: only the terms with i + j < NT (the leading triangle of the
// shift; the split-precision M2L adds the rest on the tensor cores), every
// row of the locals still stored.
template <int MT, int KS, int CH, int NT = 0>
__global__ void __launch_bounds__(128, 4) m2l_dmma_kernel(
    SegTable seg, const int *__restrict__ boxes, const int *__restrict__ slots,
    const double *__restrict__ bs, int ndc, int c0, int p,
    const double *__restrict__ binom, const double2 *__restrict__ mp,
    double2 *__restrict__ loc, int ntiles) {
    // A-operand fragments of B: [mt][ks][lane]
    __shared__ double s_a[MT * KS * 32];
    __shared__ int s_tb[257];
    // (mt, ks) tiles with a term of the triangle
    auto live = [](int mt, int ks) { return NT == 0 || mt * 8 + ks * 4 < NT; };
    for (int e = threadIdx.x; e < MT * KS * 32; e += blockDim.x) {
        const int l = e & 31, ks = (e >> 5) % KS, mt = (e >> 5) / KS;
        const int i = mt * 8 + (l >> 2), j = ks * 4 + (l & 3);
        double v = 0.0;
        if (i <= p && j <= p && (NT == 0 || i + j < NT)) {
            if (i == 0)
                v = j == 0 ? 0.0 : 1.0;
            else
                v = j == 0 ? -1.0 / i : binom[(size_t)(i + j - 1) * (kLdc + 1) + (j - 1)];
        }
        s_a[e] = v;
    }
    for (int e = threadIdx.x; e <= seg.nseg && e < 257; e += blockDim.x) s_tb[e] = seg.tile_base[e];
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int stride = (p + 1) * ndc;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile < ntiles; tile += nwarps) {
        // segment of this tile
        int lo = 0, hi = seg.nseg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_tb[mid] <= tile) lo = mid; else hi = mid;
        }
        const int sg = lo;
        const int q0 = seg.start[sg] + (tile - s_tb[sg]) * 8;
        const int qend = seg.start[sg] + seg.count[sg];
        const int cp = seg.cpos[sg];
        const double lr = log(bs[seg.level[sg]]);
        // this lane's B-operand column box (g) and C columns (2 tig, 2 tig + 1)
        const int qg = q0 + g;
        const bool has_g = qg < qend;
        double acc[CH][MT][2][2];  // [ch][mt][e][re/im]
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int e = 0; e < 2; e++) acc[c][mt][e][0] = acc[c][mt][e][1] = 0.0;
        for (int k = 0; k < kSlots; k++) {
            const int sg_box = has_g ? slots[(size_t)qg * kSlots + k] : -1;
            // skip the offset when no box of the tile has a source there
            if (__ballot_sync(0xffffffffu, sg_box >= 0) == 0) continue;
            const double tx = (double)c_slot_dx[cp][k], ty = (double)c_slot_dy[cp][k];
            // w2 = 1/t, w1 = -1/t
            const double tn = 1.0 / (tx * tx + ty * ty);
            const double2 w2 = make_double2(tx * tn, -ty * tn);
            const double2 w1 = make_double2(-w2.x, -w2.y);
            const double lt = 0.5 * log(tx * tx + ty * ty);
            // w1^(tig) and w1^4 for the B fragments (j = 4 ks + tig)
            double2 w1p = make_double2(1.0, 0.0);
            for (int u = 0; u < tig; u++) w1p = cmul(w1p, w1);
            const double2 w1_2 = cmul(w1, w1), w1_4 = cmul(w1_2, w1_2);
            // w2^g and w2^8 for the C rows (i = 8 mt + g)
            double2 w2p = make_double2(1.0, 0.0);
            for (int u = 0; u < g; u++) w2p = cmul(w2p, w2);
            const double2 w2_2 = cmul(w2, w2), w2_4 = cmul(w2_2, w2_2), w2_8 = cmul(w2_4, w2_4);
            // sources of the C columns, for the log term of row 0
            const int sn0 = __shfl_sync(0xffffffffu, sg_box, (2 * tig) * 4);
            const int sn1 = __shfl_sync(0xffffffffu, sg_box, (2 * tig + 1) * 4);
#pragma unroll
            for (int c = 0; c < CH; c++) {
                double bre[KS], bim[KS];
                double2 wj = w1p;
#pragma unroll
                for (int ks = 0; ks < KS; ks++) {
                    const int j = ks * 4 + tig;
                    double2 h = make_double2(0.0, 0.0);
                    if (live(0, ks) && sg_box >= 0 && j <= p)
                        h = cmul(mp[(size_t)sg_box * stride + (size_t)j * ndc + c0 + c], wj);
                    bre[ks] = h.x;
                    bim[ks] = h.y;
                    wj = cmul(wj, w1_4);
                }
                double tre[MT][2], tim[MT][2];
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    tre[mt][0] = tre[mt][1] = tim[mt][0] = tim[mt][1] = 0.0;
#pragma unroll
                    for (int ks = 0; ks < KS; ks++) {
                        if (!live(mt, ks)) continue;
                        const double a = s_a[(mt * KS + ks) * 32 + lane];
                        dmma(tre[mt][0], tre[mt][1], a, bre[ks]);
                        dmma(tim[mt][0], tim[mt][1], a, bim[ks]);
                    }
                }
                double2 wi = w2p;
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    if (!live(mt, 0)) break;  // (rows of no triangle term stay zero)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const double2 tt = make_double2(tre[mt][e], tim[mt][e]);
                        const double2 v = cmul(wi, tt);
                        acc[c][mt][e][0] += v.x;
                        acc[c][mt][e][1] += v.y;
                    }
                    wi = cmul(wi, w2_8);
                }
                if (g == 0) {  // row i = 0 of mt = 0: + log|z0| M_0
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int sn = e == 0 ? sn0 : sn1;
                        if (sn >= 0) {
                            const double2 m0 = mp[(size_t)sn * stride + c0 + c];
                            acc[c][0][e][0] += (lr + lt) * m0.x;
                            acc[c][0][e][1] += (lr + lt) * m0.y;
                        }
                    }
                }
            }
        }
        // store: the first writer of these boxes' local expansions
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int q = q0 + 2 * tig + e;
            if (q >= qend) continue;
            const int b = boxes[q];
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                const int i = mt * 8 + g;
                if (i > p) continue;
#pragma unroll
                for (int c = 0; c < CH; c++)
                    loc[(size_t)b * stride + (size_t)i * ndc + c0 + c] =
                        make_double2(acc[c][mt][e][0], acc[c][mt][e][1]);
            }
        }
    }
}

template <int MT, int KS, int NT = 0>
void launch_dmma(const SegTable &sg, const int *boxes, const int *slots,
                 const double *bs, int ndc, int p, const double *binom,
                 const double2 *mp, double2 *loc, int ntiles, cudaStream_t s) {
    const int blocks = std::max(1, std::min((ntiles + 3) / 4, kNumSM * 16));
    const char *e = getenv("FMM2D_B200_M2L_CH2");
    const bool ch2 = e && e[0] == '1';
    for (int c0 = 0; c0 < ndc;) {
        if (ch2 && ndc - c0 >= 2 && MT <= 5) {
            m2l_dmma_kernel<MT, KS, 2, NT><<<blocks, 128, 0, s>>>(
                sg, boxes, slots, bs, ndc, c0, p, binom, mp, loc, ntiles);
            c0 += 2;
        } else {
            m2l_dmma_kernel<MT, KS, 1, NT><<<blocks, 128, 0, s>>>(
                sg, boxes, slots, bs, ndc, c0, p, binom, mp, loc, ntiles);
            c0 += 1;
        }
        FMM_CHECK_LAUNCH();
    }
}


// The tiles of one M2L evaluation: target boxes of levels >= 2 that hold
// points, grouped by (level, child position) = segment in box order, the
// source box of every (target, slot), and the segment tables for one or more
// tile sizes.
struct M2LWork {
    DevBuf<int> boxes, slots, segd;
    struct Tab {
        int tile, off, ntiles;  // tile size, offset of its table in segd
    };
    std::vector<Tab> tabs;
    std::vector<int> start, count;  // per segment
    int nseg = 0, ntarg = 0;
    int ntiles(int tile) const {
        for (const Tab &t : tabs)
            if (t.tile == tile) return t.ntiles;
        return 0;
    }
    SegTable seg(int tile) const {
        const int *h = segd.get();
        for (const Tab &t : tabs)
            if (t.tile == tile) h += t.off;
        return SegTable{h, h + nseg + 1, h + 2 * nseg + 1, h + 3 * nseg + 1, h + 4 * nseg + 1,
                        nseg};
    }
};

// Cache key of a planning object: its kind, tile size and skipped levels.
inline uint64_t m2l_key(int kind, int tile, uint64_t skip) {
    return ((uint64_t)kind << 56) | ((uint64_t)tile << 40) | (skip & ((1ull << 40) - 1));
}

void ensure_slot_tables(cudaStream_t s) {
    static std::mutex tables_mu;
    static bool tables_ready[64] = {false};
    int dev = 0;
    FMM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> tables_lock(tables_mu);
    if (!tables_ready[dev]) {
        const SlotTables st = make_slot_tables();
        FMM_CUDA(cudaMemcpyToSymbolAsync(c_slot_dx, st.dx, sizeof(st.dx), 0, cudaMemcpyHostToDevice, s));
        FMM_CUDA(cudaMemcpyToSymbolAsync(c_slot_dy, st.dy, sizeof(st.dy), 0, cudaMemcpyHostToDevice, s));
        FMM_CUDA(cudaMemcpyToSymbolAsync(c_slot_of, st.slot_of, sizeof(st.slot_of), 0, cudaMemcpyHostToDevice, s));
        FMM_CUDA(cudaStreamSynchronize(s));
        tables_ready[dev] = true;
    }
}

// Tile bases of the segments for tiles of `tile` boxes.
std::vector<int> tile_bases(const std::vector<int> &count, int tile) {
    std::vector<int> tb(count.size() + 1, 0);
    for (size_t k = 0; k < count.size(); k++) tb[k + 1] = tb[k] + (count[k] + tile - 1) / tile;
    return tb;
}

// Place of every box of levels >= 2 in segment order: level by level, the
// boxes that are child 0 of their parent first, then child 1, ...  (Boxes
// come in groups of four siblings, in child order, on every level.)
struct SegOrder {
    int start[kMaxLevels + 2];
    __device__ __forceinline__ int at(int b, int l) const {
        const int m = b - start[l], n4 = (start[l + 1] - start[l]) >> 2;
        return start[l] - start[2] + (m & 3) * n4 + (m >> 2);
    }
};

// Builds the segments, the slot table and the segment tables for the given
// tile sizes, leaving out the target levels set in skip_levels; false when a
// list-2 entry falls outside the 27 slots or there are too many segments.
// The boxes of a segment are placed by one prefix sum over flags kept in
// segment order, and the host reads the segments' ends and the check in one
// synchronisation.  (Sorting the boxes by segment, once per tile size, took
// 0.1 ms and two synchronisations each at any size.)
bool m2l_work(const Tree &T, const CauchyProblem &P, const std::vector<int> &tiles,
              cudaStream_t s, M2LWork &w, uint64_t skip_levels = 0) {
    const int L = T.nlevels;
    ensure_slot_tables(s);
    const int lo = T.lstart[2], n = T.nboxes - lo;
    const int nseg = 4 * (L - 1);
    w.nseg = nseg;
    w.start.assign(nseg, 0);
    w.count.assign(nseg, 0);
    if (nseg + 1 > 257) return false;
    SegOrder so;
    int most = 0;  // boxes of the levels that are not left out
    for (int l = 0; l <= L; l++) {
        so.start[l] = T.lstart[l];
        if (l >= 2 && !((skip_levels >> l) & 1ull)) most += T.lend[l] - T.lstart[l];
    }
    so.start[L + 1] = T.nboxes;
    if (most == 0) return true;
    const int2 *sse = T.srcse.get(), *tse = T.trgse.get();
    const int spgh = P.sset.pgh, tpgh = P.tset.pgh;
    const int *lev = T.level.get();
    DevBuf<int> flag(n, s), pos(n + 1, s), ends(nseg + 2, s), err(1, s);
    err.zero(s);
    w.boxes.alloc(most, s);
    w.slots.alloc((size_t)most * kSlots, s);
    int *fp = flag.get(), *pp = pos.get(), *ep = err.get(), *en = ends.get();
    for_each(n, s, [=] __device__(int64_t i) {
        const int b = lo + (int)i, l = lev[b];
        int np = 0;
        if (tpgh > 0) np += tse[b].y - tse[b].x;
        if (spgh > 0) np += sse[b].y - sse[b].x;
        fp[so.at(b, l)] = np > 0 && !((skip_levels >> l) & 1ull) ? 1 : 0;
    });
    exclusive_scan_i32(fp, pp, n, pp + n, s);
    // ---- the targets and the source box of every (target, slot), from list 2
    {
        int *bx = w.boxes.get(), *sl = w.slots.get();
        const int *n2 = T.nlist2.get(), *l2 = T.list2.get();
        const double2 *cen = T.centers.get();
        const double *bsd = T.d_boxsize.get();
        for_each(n, s, [=] __device__(int64_t i) {
            const int b = lo + (int)i, l = lev[b], f = so.at(b, l);
            if (!fp[f]) return;
            const int q = pp[f], c = (b - so.start[l]) & 3;
            bx[q] = b;
            int *row = sl + (size_t)q * kSlots;
            const double ri = 1.0 / bsd[l];
            const double2 cb = cen[b];
            unsigned have = 0;
            const int m = n2[b];
            for (int e = 0; e < m; e++) {
                const int sb = l2[kMaxList2 * b + e];
                if (sse[sb].y <= sse[sb].x) continue;  // no multipole
                const double2 cs = cen[sb];
                const int dx = (int)rint((cs.x - cb.x) * ri), dy = (int)rint((cs.y - cb.y) * ri);
                const int k = (dx >= -3 && dx <= 3 && dy >= -3 && dy <= 3)
                                  ? c_slot_of[c][dx + 3][dy + 3] : -1;
                if (k < 0) {
                    atomicExch(ep, 1);
                    continue;
                }
                have |= 1u << k;
                row[k] = sb;
            }
            for (int k = 0; k < kSlots; k++)
                if (!((have >> k) & 1u)) row[k] = -1;
        });
    }
    for_each(nseg + 2, s, [=] __device__(int64_t k) {
        if (k == nseg + 1) {
            en[k] = *ep;
        } else if (k == nseg) {
            en[k] = pp[n];
        } else {
            const int l = 2 + (int)k / 4, c = (int)k & 3;
            en[k] = pp[so.start[l] - lo + c * ((so.start[l + 1] - so.start[l]) >> 2)];
        }
    });
    std::vector<int> h(nseg + 2);
    read_small(h.data(), en, h.size() * sizeof(int), s);
    if (h[nseg + 1] != 0) return false;
    for (int k = 0; k < nseg; k++) {
        w.start[k] = h[k];
        w.count[k] = h[k + 1] - h[k];
    }
    w.ntarg = h[nseg];
    if (w.ntarg == 0) return true;
    std::vector<int> all;
    for (int tile : tiles) {
        const std::vector<int> tb = tile_bases(w.count, tile);
        w.tabs.push_back({tile, (int)all.size(), tb[nseg]});
        all.insert(all.end(), tb.begin(), tb.end());
        all.insert(all.end(), w.start.begin(), w.start.end());
        all.insert(all.end(), w.count.begin(), w.count.end());
        for (int k = 0; k < nseg; k++) all.push_back(2 + k / 4);
        for (int k = 0; k < nseg; k++) all.push_back(k % 4);
    }
    w.segd.alloc(all.size(), s);
    FMM_CUDA(cudaMemcpyAsync(w.segd.get(), all.data(), all.size() * sizeof(int),
                             cudaMemcpyHostToDevice, s));
    return true;
}

#include "m2l_orbit.cuh"

// ---------------------------------------------------------------------------
// FP32 M2L of the mixed-precision mode.  With t the slot offset in box
// units, the whole shift is one complex matrix per (child position, slot),
// level independent in the scaled form:
//     T_ij = w2^i B_ij w1^j  (T_00 = log|t|),
// and L_i += sum_slots sum_j T_ij M_j, plus log(r) M_0 in L_0.  One thread
// per target box, 128 boxes of one segment per block; the block stages
// each slot's matrix in shared memory (read as broadcasts) and every thread
// streams its source multipole (an FP32 copy) through the j loop, keeping
// the P1 x CH accumulators in registers (FP32 arithmetic, FP32
// accumulation over the 27 slots, stored as FP64).
// ---------------------------------------------------------------------------
constexpr int kFp32Tile = 128;

template <int P1, int CH>
__global__ void __launch_bounds__(kFp32Tile) m2l_fp32_kernel(
    SegTable seg, const int *__restrict__ boxes, const int *__restrict__ slots,
    const double *__restrict__ bs, int ndc, int c0, int p, const float2 *__restrict__ Tall,
    const float2 *__restrict__ mp32, double2 *__restrict__ loc, int ntiles) {
    __shared__ float2 sT[P1 * P1];
    __shared__ int s_tb[257];
    for (int e = threadIdx.x; e <= seg.nseg && e < 257; e += blockDim.x) s_tb[e] = seg.tile_base[e];
    __syncthreads();
    const int stride = (p + 1) * ndc;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int lo = 0, hi = seg.nseg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_tb[mid] <= tile) lo = mid; else hi = mid;
        }
        const int sg = lo;
        const int q = seg.start[sg] + (tile - s_tb[sg]) * kFp32Tile + threadIdx.x;
        const bool valid = q < seg.start[sg] + seg.count[sg];
        const int cp = seg.cpos[sg];
        const float lr = (float)log(bs[seg.level[sg]]);
        float2 acc[CH][P1];
        float2 s0[CH];
#pragma unroll
        for (int c = 0; c < CH; c++) {
            s0[c] = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < P1; i++) acc[c][i] = make_float2(0.f, 0.f);
        }
        for (int k = 0; k < kSlots; k++) {
            __syncthreads();  // the previous slot's matrix is no longer read
            const float2 *Tk = Tall + ((size_t)cp * kSlots + k) * P1 * P1;
            for (int e = threadIdx.x; e < P1 * P1; e += blockDim.x) sT[e] = Tk[e];
            __syncthreads();
            const int sb = valid ? slots[(size_t)q * kSlots + k] : -1;
            if (sb < 0) continue;
            const float2 *M = mp32 + (size_t)sb * stride + c0;
#pragma unroll
            for (int j = 0; j < P1; j++) {
                float2 m[CH];
#pragma unroll
                for (int c = 0; c < CH; c++)
                    m[c] = j <= p ? M[(size_t)j * ndc + c] : make_float2(0.f, 0.f);
                if (j == 0) {
#pragma unroll
                    for (int c = 0; c < CH; c++) {
                        s0[c].x += m[c].x;
                        s0[c].y += m[c].y;
                    }
                }
#pragma unroll
                for (int i = 0; i < P1; i++) {
                    const float2 t = sT[i * P1 + j];
#pragma unroll
                    for (int c = 0; c < CH; c++) {
                        acc[c][i].x = fmaf(t.x, m[c].x, fmaf(-t.y, m[c].y, acc[c][i].x));
                        acc[c][i].y = fmaf(t.x, m[c].y, fmaf(t.y, m[c].x, acc[c][i].y));
                    }
                }
            }
        }
        if (valid) {
            const int b = boxes[q];
#pragma unroll
            for (int c = 0; c < CH; c++) {
                acc[c][0].x += lr * s0[c].x;
                acc[c][0].y += lr * s0[c].y;
            }
#pragma unroll
            for (int i = 0; i < P1; i++) {
                if (i > p) break;
#pragma unroll
                for (int c = 0; c < CH; c++)
                    loc[(size_t)b * stride + (size_t)i * ndc + c0 + c] =
                        make_double2((double)acc[c][i].x, (double)acc[c][i].y);
            }
        }
    }
}

// The leading NR rows (local coefficients) of the same sums, which the
// tensor-core form leaves to FP32 (see the end of m2l_fp32): one thread per
// (box, row), so the 27 slots' matrices of the rows fit into shared memory at
// once and a thread's chain is its row's terms alone; every accumulator adds
// the same terms in the same order as m2l_fp32_kernel's.  Bound by the latency
// of the source rows' loads, which are issued one slot ahead.  Runs in blocks
// of m2l_tc_kernel's launch beside its tiles.  (A thread per box with the
// matrices staged slot by slot took 79 us for a tile, whatever it held.)
constexpr int rows_tile(int nr) { return 128 / nr; }  // boxes per block of 128 threads
constexpr int kRowsP1 = 20;

template <int CH, int NR>
__device__ __forceinline__ void m2l_rows(const SegTable &seg, const int *s_tb, float2 *sT,
                                         const int *__restrict__ boxes,
                                         const int *__restrict__ slots,
                                         const double *__restrict__ bs, int ndc, int c0, int p,
                                         const float2 *__restrict__ Tall,
                                         const float2 *__restrict__ mp32,
                                         double2 *__restrict__ loc, int first, int step,
                                         int ntiles) {
    constexpr int P1 = kRowsP1, TILE = rows_tile(NR);
    const int stride = (p + 1) * ndc;
    const int row = threadIdx.x % NR, bx = threadIdx.x / NR;
    int cp_in = -1;
    for (int tile = first; tile < ntiles; tile += step) {
        int lo = 0, hi = seg.nseg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_tb[mid] <= tile) lo = mid; else hi = mid;
        }
        const int cp = seg.cpos[lo];
        if (cp != cp_in) {
            __syncthreads();
            const float2 *Tc = Tall + (size_t)cp * kSlots * P1 * P1;
            for (int e = threadIdx.x; e < kSlots * NR * P1; e += blockDim.x)
                sT[e] = Tc[(size_t)(e / (NR * P1)) * P1 * P1 + e % (NR * P1)];
            cp_in = cp;
            __syncthreads();
        }
        const int q = seg.start[lo] + (tile - s_tb[lo]) * TILE + bx;
        if (bx >= TILE || q >= seg.start[lo] + seg.count[lo] || row > p) continue;
        const int *qs = slots + (size_t)q * kSlots;
        int sb[kSlots];
        unsigned mask = 0u;
#pragma unroll
        for (int k = 0; k < kSlots; k++) sb[k] = qs[k];
#pragma unroll
        for (int k = 0; k < kSlots; k++)
            if (sb[k] >= 0) mask |= 1u << k;
        float2 m[P1][CH], n[P1][CH];
        auto load = [&](int k) {
            const float2 *M = mp32 + (size_t)qs[k] * stride + c0;
#pragma unroll
            for (int j = 0; j < P1; j++)
#pragma unroll
                for (int c = 0; c < CH; c++)
                    n[j][c] = j <= p ? M[(size_t)j * ndc + c] : make_float2(0.f, 0.f);
        };
        float2 acc[CH], s0[CH];
#pragma unroll
        for (int c = 0; c < CH; c++) acc[c] = s0[c] = make_float2(0.f, 0.f);
        if (mask) load(__ffs(mask) - 1);
        while (mask) {
            const int k = __ffs(mask) - 1;
            mask &= mask - 1;
#pragma unroll
            for (int j = 0; j < P1; j++)
#pragma unroll
                for (int c = 0; c < CH; c++) m[j][c] = n[j][c];
            if (mask) load(__ffs(mask) - 1);
            const float2 *t0 = sT + (k * NR + row) * P1;
#pragma unroll
            for (int c = 0; c < CH; c++) {
                s0[c].x += m[0][c].x;
                s0[c].y += m[0][c].y;
            }
#pragma unroll
            for (int j = 0; j < P1; j++) {
                const float2 t = t0[j];
#pragma unroll
                for (int c = 0; c < CH; c++) {
                    acc[c].x = fmaf(t.x, m[j][c].x, fmaf(-t.y, m[j][c].y, acc[c].x));
                    acc[c].y = fmaf(t.x, m[j][c].y, fmaf(t.y, m[j][c].x, acc[c].y));
                }
            }
        }
        const int b = boxes[q];
#pragma unroll
        for (int c = 0; c < CH; c++) {
            if (row == 0) {
                const float lr = (float)log(bs[seg.level[lo]]);
                acc[c].x += lr * s0[c].x;
                acc[c].y += lr * s0[c].y;
            }
            loc[(size_t)b * stride + (size_t)row * ndc + c0 + c] =
                make_double2((double)acc[c].x, (double)acc[c].y);
        }
    }
}

// T_ij = w2^i B_ij w1^j per (child position, slot), FP64 built, FP32
// stored, padded to P1 x P1; cached per device and order.
const float2 *fp32_tables(int p, int P1, cudaStream_t s) {
    static std::mutex mu;
    static std::vector<std::pair<long, const float2 *>> cache;
    int dev;
    FMM_CUDA(cudaGetDevice(&dev));
    const long key = ((long)dev << 20) | ((long)p << 8) | P1;
    std::lock_guard<std::mutex> g(mu);
    for (auto &e : cache)
        if (e.first == key) return e.second;
    const SlotTables st = make_slot_tables();
    // binomials C(l, m) for l <= 2 P1
    const int nc = 2 * P1 + 2;
    std::vector<double> C((size_t)nc * nc, 0.0);
    for (int l = 0; l < nc; l++) {
        C[(size_t)l * nc] = 1.0;
        for (int m = 1; m <= l; m++)
            C[(size_t)l * nc + m] = C[(size_t)(l - 1) * nc + m - 1] + (m < l ? C[(size_t)(l - 1) * nc + m] : 0.0);
    }
    std::vector<float2> h((size_t)4 * kSlots * P1 * P1, make_float2(0.f, 0.f));
    for (int c = 0; c < 4; c++)
        for (int k = 0; k < kSlots; k++) {
            const double tx = st.dx[c][k], ty = st.dy[c][k];
            const double tn = 1.0 / (tx * tx + ty * ty);
            const double2 w2 = make_double2(tx * tn, -ty * tn), w1 = make_double2(-w2.x, -w2.y);
            float2 *Tk = h.data() + ((size_t)c * kSlots + k) * P1 * P1;
            double2 w2i = make_double2(1.0, 0.0);
            for (int i = 0; i <= p; i++) {
                double2 w1j = make_double2(1.0, 0.0);
                for (int j = 0; j <= p; j++) {
                    double b;
                    if (i == 0)
                        b = j == 0 ? 0.0 : 1.0;
                    else
                        b = j == 0 ? -1.0 / i : C[(size_t)(i + j - 1) * nc + (j - 1)];
                    double2 v = cscal(cmul(w2i, w1j), b);
                    if (i == 0 && j == 0) v = make_double2(0.5 * std::log(tx * tx + ty * ty), 0.0);
                    Tk[i * P1 + j] = make_float2((float)v.x, (float)v.y);
                    w1j = cmul(w1j, w1);
                }
                w2i = cmul(w2i, w2);
            }
        }
    float2 *d = nullptr;
    FMM_CUDA(cudaMalloc(&d, h.size() * sizeof(float2)));
    FMM_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(float2), cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaStreamSynchronize(s));
    cache.push_back({key, d});
    return d;
}

template <int P1>
void launch_fp32(const M2LWork &w, const Tree &T, const CauchyProblem &P, const float2 *Tab,
                 const float2 *mp32, double2 *loc, cudaStream_t s) {
    const int ntiles = w.ntiles(kFp32Tile);
    const int blocks = std::max(1, std::min(ntiles, kNumSM * 16));
    const SegTable sg = w.seg(kFp32Tile);
    const int *boxes = w.boxes.get();
    for (int c0 = 0; c0 < P.ndc;) {
        if (P.ndc - c0 >= 2) {
            m2l_fp32_kernel<P1, 2><<<blocks, kFp32Tile, 0, s>>>(
                sg, boxes, w.slots.get(), T.d_boxsize.get(), P.ndc, c0, P.p, Tab, mp32, loc,
                ntiles);
            c0 += 2;
        } else {
            m2l_fp32_kernel<P1, 1><<<blocks, kFp32Tile, 0, s>>>(
                sg, boxes, w.slots.get(), T.d_boxsize.get(), P.ndc, c0, P.p, Tab, mp32, loc,
                ntiles);
            c0 += 1;
        }
        FMM_CHECK_LAUNCH();
    }
}

// ---------------------------------------------------------------------------
// M2L of the mixed mode on the 5th-generation tensor cores (tcgen05, kind
// tf32, operands in shared memory, accumulator in tensor memory).
//
// In real form the slot operator is the 2P x 2P block matrix
// [[Re T, -Im T], [Im T, Re T]] (P = p + 1) acting on [Re M; Im M].  A tile
// is 128 rows = 128 / CH target boxes x CH channels of one segment; for each
// of the 27 slots the block gathers the rows' source multipoles (A, 128 x
// KP, KP = 2P rounded up to 8) and copies the slot's matrix (B, KP x KP,
// stored N-rows x K as the MMA's K-major B) into shared memory, and one
// thread issues D += A_hi B_hi + A_hi B_lo + A_lo B_hi (3 x TF32 split:
// x = hi + lo, both TF32-rounded; about 22 significant bits) accumulating
// all slots in the same tensor-memory tile.  The rows are read back with
// tcgen05.ld and stored as FP64.  Waits on the MMA-completion barrier are
// bounded; a wait that runs out sets *err and the kernel returns after
// releasing its tensor memory.
//
// Shared-memory operands use the no-swizzle K-major layout: 8-row x 16-byte
// core matrices, contiguous 128 bytes each; core matrix (row group g, K
// chunk c) at ((c * G + g) * 128) bytes, G = rows / 8.  So SBO (between row
// groups) = 128 bytes and LBO (between K chunks) = G * 128 bytes.
// ---------------------------------------------------------------------------
constexpr int kTcRows = 128;
constexpr int kTcMaxKP = 40;
// longest wait for an MMA-completion barrier (the MMAs of one slot take
// microseconds)
constexpr uint64_t kTcWaitNs = 2000000000ull;

// Bounded wait for the barrier phase with the given parity.
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity) {
    int never = 0;
    return mbar_wait_bounded(mbar, parity, &never, kTcWaitNs);
}

// byte offset of element (row, k) in a K-major no-swizzle operand of
// `rows` rows
__host__ __device__ __forceinline__ int tc_off(int row, int k, int rows) { return tc_fidx(row, k, rows) << 2; }

// The slots of a tile are pipelined D deep: the rows' source multipoles are
// loaded D slots ahead into registers, a slot's matrix comes by one bulk copy D
// slots ahead into one of 2 D buffers, and the operand rows have D buffers, so
// that with D = 2 storing one slot's rows overlaps the MMAs of the slot before.
// D = 2 (one block per SM) runs while every tile has an SM of its own and the
// chain of its 27 slots is what takes the time; with more tiles three blocks of
// D = 1 per SM overlap one another instead.  (One buffer, filled by all threads
// after the previous slot's MMAs, took 2.8 us per slot: 76 us for a single
// tile.)
//
// NR > 0: the rows below NR are left to m2l_rows, which runs in the blocks
// from ntcb on; NR = 0: row 0 (L_0, whose terms cancel across the slots) is
// summed in FP32 beside the MMAs.
template <int HALF, int D>
constexpr size_t tc_smem_bytes() {
    return (size_t)D * (2 * kTcRows * 2 * HALF + 2 * 2 * 4 * HALF * HALF) * sizeof(float);
}

struct TcArgs {
    SegTable seg, rseg;  // tiles of the rows' operand, of m2l_rows
    const int *boxes, *slots;
    const double *bs;
    int ndc, c0, p, ntiles, ntcb, nrtiles;
    const float *Bimg;
    const float2 *T0, *Trows, *mp32;
    double2 *loc;
    int *err;
};

template <int CH, int HALF, int NR, int D>
__global__ void __launch_bounds__(kTcRows, D == 1 ? 3 : 1) m2l_tc_kernel(const TcArgs A) {
    constexpr int kABufs = D, kBBufs = 2 * D;
    constexpr int KP = 2 * HALF;  // [Re 0..HALF-1 | Im 0..HALF-1]
    constexpr int kAFloats = 2 * kTcRows * KP, kBFloats = 2 * KP * KP;
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    float *sA = reinterpret_cast<float *>(tc_smem);       // [buffer][hi, lo]
    float *sB = sA + kABufs * kAFloats;                 // [buffer][hi, lo]
    constexpr int TPT = kTcRows / CH;
    __shared__ __align__(8) uint64_t s_mbar[kABufs + kBBufs];
    __shared__ uint32_t s_tmem;
    __shared__ int s_tb[257];
    __shared__ unsigned s_mask;
    __shared__ int s_qs[TPT * kSlots];
    __shared__ float2 s_t0[NR > 0 ? 1 : kSlots * (kTcMaxKP / 2)];
    const int tid = threadIdx.x, warp = tid >> 5;
    if constexpr (NR > 0) {
        if ((int)blockIdx.x >= A.ntcb) {
            for (int e = tid; e <= A.rseg.nseg && e < 257; e += blockDim.x)
                s_tb[e] = A.rseg.tile_base[e];
            __syncthreads();
            m2l_rows<CH, NR>(A.rseg, s_tb, reinterpret_cast<float2 *>(tc_smem), A.boxes, A.slots,
                             A.bs, A.ndc, A.c0, A.p, A.Trows, A.mp32, A.loc,
                             (int)blockIdx.x - A.ntcb, (int)gridDim.x - A.ntcb, A.nrtiles);
            return;
        }
    }
    const SegTable &seg = A.seg;
    for (int e = tid; e <= seg.nseg && e < 257; e += blockDim.x) s_tb[e] = seg.tile_base[e];
    if (tid == 0) {
        s_mask = 0u;
        for (int i = 0; i < kABufs + kBBufs; i++) mbar_init(smem_u32(&s_mbar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto a_bar = [&](int i) { return smem_u32(&s_mbar[i]); };
    auto b_bar = [&](int i) { return smem_u32(&s_mbar[kABufs + i]); };
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&s_tmem)),
                     "r"(64)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const int P = A.p + 1, stride = P * A.ndc;
    constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(KP >> 3) << 17) |
                               (8u << 24);
    constexpr uint32_t aLBO = (kTcRows / 8) * 128, bLBO = (KP / 8) * 128, SBO = 128;
    // uses of every buffer so far (thread-uniform; B's by thread 0)
    uint32_t na[kABufs] = {}, nb_issued[kBBufs] = {}, nb_done[kBBufs] = {};
    int last = -1;  // operand buffer of the last commit
    bool failed = false;
    int cp_loaded = -1;
    for (int tile = blockIdx.x; tile < A.ntiles; tile += NR > 0 ? A.ntcb : (int)gridDim.x) {
        int lo = 0, hi = seg.nseg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_tb[mid] <= tile) lo = mid; else hi = mid;
        }
        const int sg = lo;
        const int qend = seg.start[sg] + seg.count[sg];
        const int q0 = seg.start[sg] + (tile - s_tb[sg]) * TPT;
        const int nbox = min(TPT, qend - q0);
        const int bx = tid / CH, q = q0 + bx, c = A.c0 + tid % CH;
        const bool valid = bx < nbox;
        const int cp = seg.cpos[sg];
        // the sources of the tile's slots, and the mask of slots in use
        unsigned mymask = 0u;
        for (int e = tid; e < nbox * kSlots; e += kTcRows) {
            const int sb = A.slots[(size_t)q0 * kSlots + e];
            s_qs[e] = sb;
            if (sb >= 0) mymask |= 1u << (e % kSlots);
        }
        mymask = __reduce_or_sync(0xffffffffu, mymask);
        if ((tid & 31) == 0 && mymask) atomicOr(&s_mask, mymask);
        if (NR == 0 && cp != cp_loaded) {  // row 0 of this position's 27 matrices
            for (int e = tid; e < kSlots * P; e += blockDim.x)
                s_t0[(e / P) * (kTcMaxKP / 2) + e % P] =
                    A.T0[((size_t)cp * kSlots + e / P) * P + e % P];
        }
        cp_loaded = cp;
        __syncthreads();
        unsigned mask = s_mask;
        __syncthreads();  // all have read the mask; it is cleared for the next tile
        if (tid == 0) s_mask = 0u;
        float l0x = 0.f, l0y = 0.f;  // row 0 (L_0) on the CUDA cores
        float s0x = 0.f, s0y = 0.f;
        // source rows of the coming D slots
        float2 m0[HALF], m1[D == 2 ? HALF : 1];
        auto load = [&](int k, float2 *m) {
            const int sb = valid && k >= 0 ? s_qs[bx * kSlots + k] : -1;
            const float2 *M = A.mp32 + (size_t)(sb >= 0 ? sb : 0) * stride + c;
#pragma unroll
            for (int j = 0; j < HALF; j++)
                m[j] = (sb >= 0 && j < P) ? M[(size_t)j * A.ndc] : make_float2(0.f, 0.f);
        };
        // a slot's matrix (hi and lo images) into B buffer `buf`
        auto fetch = [&](int k, int buf) {
            if (tid != 0 || k < 0) return;
            mbar_arrive_expect_tx(b_bar(buf), kBFloats * sizeof(float));
            bulk_g2s(smem_u32(sB + buf * kBFloats),
                     A.Bimg + ((size_t)cp * kSlots + k) * kBFloats, kBFloats * sizeof(float),
                     b_bar(buf));
            nb_issued[buf]++;
        };
        // slots in order: k0 now, k1 (and with D = 2 k2) next
        auto pop = [&]() {
            if (!mask) return -1;
            const int k = __ffs(mask) - 1;
            mask &= mask - 1;
            return k;
        };
        int k0 = pop(), k1 = pop();
        // (every MMA of the tile before has completed: the buffers are free)
        fetch(k0, 0);
        load(k0, m0);
        if (D == 2) {
            fetch(k1, 1);
            load(k1, m1);
        }
        bool issued = false;
        for (int i = 0; k0 >= 0; i++) {
            const int ab = i & (kABufs - 1), bb = i & (kBBufs - 1);
            // the MMAs of slot i - D read this operand buffer (and B buffer
            // i + D)
            if (i >= D && !tc_wait(a_bar(ab), (na[ab] - 1) & 1)) failed = true;
            float *hi_ = sA + ab * kAFloats, *lo_ = hi_ + kTcRows * KP;
            // A row `tid`: [Re M_0..HALF-1 | Im M_0..HALF-1] (zero beyond p),
            // split into TF32 hi / lo
#pragma unroll
            for (int kc = 0; kc < KP; kc += 4) {
                float4 vh, vl;
                float *ph = &vh.x, *pl = &vl.x;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int kk = kc + u;
                    const float v = kk < HALF ? m0[kk].x : m0[kk - HALF].y;
                    const float h = tc_tf32(v);
                    ph[u] = h;
                    pl[u] = tc_tf32(v - h);
                }
                const int off = tc_off(tid, kc, kTcRows) >> 2;
                *reinterpret_cast<float4 *>(hi_ + off) = vh;
                *reinterpret_cast<float4 *>(lo_ + off) = vl;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (__syncthreads_or(failed)) {
                failed = true;
                break;
            }
            const int k2 = pop(), kn = D == 2 ? k2 : k1;  // kn: D slots on
            fetch(kn, (i + D) & (kBBufs - 1));  // (was slot i - D's)
            if (tid == 0) {
                if (!tc_wait(b_bar(bb), (nb_issued[bb] - 1) & 1)) {
                    failed = true;
                } else {
                    nb_done[bb] = nb_issued[bb];
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t aHi = smem_u32(hi_), aLo = smem_u32(lo_);
                    const uint32_t bHi = smem_u32(sB + bb * kBFloats), bLo = bHi + KP * KP * 4;
                    for (int ks = 0; ks < KP / 8; ks++) {
                        const uint32_t ao = 2 * ks * aLBO, bo = 2 * ks * bLBO;
                        tc_mma(tmem, tc_sdesc(aHi + ao, aLBO, SBO), tc_sdesc(bHi + bo, bLBO, SBO),
                               idesc, (issued || ks > 0) ? 1u : 0u);
                        tc_mma(tmem, tc_sdesc(aHi + ao, aLBO, SBO), tc_sdesc(bLo + bo, bLBO, SBO),
                               idesc, 1u);
                        tc_mma(tmem, tc_sdesc(aLo + ao, aLBO, SBO), tc_sdesc(bHi + bo, bLBO, SBO),
                               idesc, 1u);
                    }
                    tc_commit(a_bar(ab));
                }
            }
            na[ab]++;
            last = ab;
            issued = true;
            if (NR == 0 && valid && s_qs[bx * kSlots + k0] >= 0) {
                // row 0 on the CUDA cores while the MMAs run
                const float2 *t0 = s_t0 + (NR > 0 ? 0 : k0 * (kTcMaxKP / 2));
#pragma unroll
                for (int j = 0; j < HALF; j++) {
                    if (j < P) {
                        const float2 t = t0[j], m = m0[j];
                        l0x = fmaf(t.x, m.x, fmaf(-t.y, m.y, l0x));
                        l0y = fmaf(t.x, m.y, fmaf(t.y, m.x, l0y));
                    }
                }
                s0x += m0[0].x;
                s0y += m0[0].y;
            }
            if (D == 2) {
#pragma unroll
                for (int j = 0; j < HALF; j++) m0[j] = m1[D == 2 ? j : 0];
                load(kn, m1);
            } else {
                load(kn, m0);
            }
            k0 = k1;
            k1 = k2;
        }
        if (__syncthreads_or(failed)) {
            failed = true;
            break;
        }
        float d[KP];
#pragma unroll
        for (int i = 0; i < KP; i++) d[i] = 0.f;
        if (issued) {
            // (a commit covers every MMA issued before it)
            if (!tc_wait(a_bar(last), (na[last] - 1) & 1)) failed = true;
            if (__syncthreads_or(failed)) {
                failed = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
            for (int c8 = 0; c8 < KP / 8; c8++) {
                float v[8];
                tc_ld8(taddr + c8 * 8, v);
#pragma unroll
                for (int u = 0; u < 8; u++) d[c8 * 8 + u] = v[u];
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        if (valid) {
            const int b = A.boxes[q];
            const double lr = NR > 0 ? 0.0 : log(A.bs[seg.level[sg]]);
#pragma unroll
            for (int i = 0; i < HALF; i++) {
                if (i < NR || i >= P) continue;
                double re, im;
                if (i == 0) {
                    re = (double)l0x + lr * s0x;
                    im = (double)l0y + lr * s0y;
                } else {
                    re = d[i];
                    im = d[HALF + i];
                }
                A.loc[(size_t)b * stride + (size_t)i * A.ndc + c] = make_double2(re, im);
            }
        }
        // the next tile's MMAs overwrite the accumulator
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
    }
    if (failed) {
        if (tid == 0) {
            atomicExch(A.err, 1);
            // let the copies and MMAs still in flight finish before the
            // memory is released
            for (int i = 0; i < kBBufs; i++)
                if (nb_issued[i] != nb_done[i]) tc_wait(b_bar(i), (nb_issued[i] - 1) & 1);
        }
        if (last >= 0 && na[last] > 0) tc_wait(a_bar(last), (na[last] - 1) & 1);
    }
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(64)
                     : "memory");
    }
}

// m2l_rows alone: with more tiles than SMs its blocks would wait for the shared
// memory of the tensor-core form's.
template <int CH, int NR>
__global__ void __launch_bounds__(kTcRows) m2l_rows_kernel(const TcArgs A) {
    extern __shared__ __align__(16) unsigned char rows_smem[];
    __shared__ int s_tb[257];
    for (int e = threadIdx.x; e <= A.rseg.nseg && e < 257; e += blockDim.x)
        s_tb[e] = A.rseg.tile_base[e];
    __syncthreads();
    m2l_rows<CH, NR>(A.rseg, s_tb, reinterpret_cast<float2 *>(rows_smem), A.boxes, A.slots, A.bs,
                     A.ndc, A.c0, A.p, A.Trows, A.mp32, A.loc, (int)blockIdx.x, (int)gridDim.x,
                     A.nrtiles);
}

// B images per (child position, slot): the real form of T (rows = outputs
// i, K = inputs j), TF32 hi and lo, in the operand layout; cached per
// device and order.
float tf32_round_host(float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
    float r;
    memcpy(&r, &u, 4);
    return r;
}

// Also returns (t0) row 0 of each matrix, P complex FP32 values per
// (child position, slot), for the CUDA-core L_0 sum.
const float *tc_tables(int p, int KP, cudaStream_t s, const float2 **t0out) {
    static std::mutex mu;
    static std::vector<std::pair<long, const float *>> cache;
    static std::vector<std::pair<long, const float2 *>> cache0;
    int dev;
    FMM_CUDA(cudaGetDevice(&dev));
    const long key = ((long)dev << 20) | ((long)p << 8) | KP;
    std::lock_guard<std::mutex> g(mu);
    for (size_t e = 0; e < cache.size(); e++)
        if (cache[e].first == key) {
            *t0out = cache0[e].second;
            return cache[e].second;
        }
    const int P = p + 1;
    const SlotTables st = make_slot_tables();
    std::vector<float2> t0h((size_t)4 * kSlots * P);
    const int nc = 2 * P + 2;
    std::vector<double> C((size_t)nc * nc, 0.0);
    for (int l = 0; l < nc; l++) {
        C[(size_t)l * nc] = 1.0;
        for (int m = 1; m <= l; m++)
            C[(size_t)l * nc + m] =
                C[(size_t)(l - 1) * nc + m - 1] + (m < l ? C[(size_t)(l - 1) * nc + m] : 0.0);
    }
    std::vector<float> h((size_t)4 * kSlots * 2 * KP * KP, 0.f);
    std::vector<double2> T((size_t)P * P);
    for (int cp = 0; cp < 4; cp++)
        for (int k = 0; k < kSlots; k++) {
            const double tx = st.dx[cp][k], ty = st.dy[cp][k];
            const double tn = 1.0 / (tx * tx + ty * ty);
            const double2 w2 = make_double2(tx * tn, -ty * tn), w1 = make_double2(-w2.x, -w2.y);
            double2 w2i = make_double2(1.0, 0.0);
            for (int i = 0; i < P; i++) {
                double2 w1j = make_double2(1.0, 0.0);
                for (int j = 0; j < P; j++) {
                    double b;
                    if (i == 0)
                        b = j == 0 ? 0.0 : 1.0;
                    else
                        b = j == 0 ? -1.0 / i : C[(size_t)(i + j - 1) * nc + (j - 1)];
                    double2 v = cscal(cmul(w2i, w1j), b);
                    if (i == 0 && j == 0) v = make_double2(0.5 * std::log(tx * tx + ty * ty), 0.0);
                    T[(size_t)i * P + j] = v;
                    w1j = cmul(w1j, w1);
                }
                w2i = cmul(w2i, w2);
            }
            float *hi = h.data() + ((size_t)cp * kSlots + k) * 2 * KP * KP;
            float *lo = hi + KP * KP;
            float2 *t0 = t0h.data() + ((size_t)cp * kSlots + k) * P;
            for (int j = 0; j < P; j++)
                t0[j] = make_float2((float)T[j].x, (float)T[j].y);
            // rows / columns [Re 0..HALF-1 | Im 0..HALF-1], zero beyond p;
            // row 0 (L_0) is summed on the CUDA cores: rows 0 and HALF stay zero
            const int HALF = KP / 2;
            for (int n = 0; n < KP; n++)
                for (int kk = 0; kk < KP; kk++) {
                    const int i = n < HALF ? n : n - HALF, j = kk < HALF ? kk : kk - HALF;
                    if (i == 0 || i >= P || j >= P) continue;
                    const double2 t = T[(size_t)i * P + j];
                    double v;
                    if (n < HALF) v = kk < HALF ? t.x : -t.y;
                    else v = kk < HALF ? t.y : t.x;
                    const float f = (float)v;
                    const float fh = tf32_round_host(f);
                    const int off = tc_off(n, kk, KP) >> 2;
                    hi[off] = fh;
                    lo[off] = tf32_round_host(f - fh);
                }
        }
    float *d = nullptr;
    float2 *d0 = nullptr;
    FMM_CUDA(cudaMalloc(&d, h.size() * sizeof(float)));
    FMM_CUDA(cudaMalloc(&d0, t0h.size() * sizeof(float2)));
    FMM_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaMemcpyAsync(d0, t0h.data(), t0h.size() * sizeof(float2), cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaStreamSynchronize(s));
    cache.push_back({key, d});
    cache0.push_back({key, d0});
    *t0out = d0;
    return d;
}

}  // namespace

bool m2l_tensor_fp64(const Tree &T, const CauchyProblem &P, const double2 *mp,
                     double2 *loc, cudaStream_t s) {
    const int L = T.nlevels, p = P.p;
    if (L < 2 || p > 63) return false;
    bool ok = false;
    const auto wp = m2l_cached<M2LWork>(P.m2l_cache, m2l_key(1, 8, 0), ok,
                                        [&](M2LWork &x) { return m2l_work(T, P, {8}, s, x); });
    if (!ok) return false;
    const M2LWork &w = *wp;
    if (w.ntarg == 0) return true;
    const SegTable sg = w.seg(8);
    const int *boxes = w.boxes.get();
    const double *bs = T.d_boxsize.get();
    const double *binom = device_binomials(s);
    if (m2l_orbit(w, T, P.ndc, p, binom, mp, loc, s)) return true;
    const int ntiles = w.ntiles(8);
    const int ks = (p + 1 + 3) / 4;
    const int mt = (p + 1 + 7) / 8;
#define FMM_M2L_CASE(MT_, KS_)                                                   \
    if (mt <= MT_ && ks <= KS_) {                                                \
        launch_dmma<MT_, KS_>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, \
                              loc, ntiles, s);                                   \
        return true;                                                             \
    }
    FMM_M2L_CASE(2, 4)
    FMM_M2L_CASE(3, 5)
    FMM_M2L_CASE(3, 6)
    FMM_M2L_CASE(4, 8)
    FMM_M2L_CASE(5, 10)
    FMM_M2L_CASE(6, 12)
    FMM_M2L_CASE(8, 16)
#undef FMM_M2L_CASE
    return false;
}

// ---------------------------------------------------------------------------
// Split-precision M2L (eps below the mixed mode's range, all other passes
// FP64).  The scaled shift's terms T_ij M_j fall off with the total order
// n = i + j: for the nearest list-2 offsets (|t| = 2) and points at the
// box corners their share of the potential is about 0.707^n, and measured
// errors fall about 8x per 4 orders.  The leading triangle i + j < NT runs
// in FP64 on the DMMA kernel (the first writer of every local); the tail
// i + j >= NT runs as TF32 x 3 slot GEMMs on the tcgen05 tensor cores
// (slot_gemm_tc_level, about 2^-22 relative per product, one FP32
// accumulation over a tile's slots: the tail is small beside the result)
// and is added on top.  The tail's error falls about 0.59x per order of NT
// and eps about 0.47x per order of p, so NT grows faster than p:
// NT = 4 (p - 13) / 3 + 2 (rounded up to a multiple of 4) holds gradients
// and Hessians on clustered points within eps of the FP64 mode at 1e-9
// (p = 28, NT = 24) and 1e-10 (p = 31, NT = 28; 24 left Hessians 1.15e-10
// off).  At 1e-12 (p = 37) even NT = 32 left the Hessians of clustered
// points at 2e-11, twenty times the FP64 mode's error: orders above 31 keep
// the FP64 M2L.
// ---------------------------------------------------------------------------

// The tail images (i + j >= nt) of the 4 x 27 slot operators in real form,
// T_ij = w2^i B_ij w1^j (w2 = 1/t, w1 = -1/t, t the slot offset), TF32
// split; cached per device, order and nt.
const float *split_tail_tables(int p, int KP, int nt, cudaStream_t s) {
    static std::mutex mu;
    static std::vector<std::pair<long, const float *>> cache;
    int dev;
    FMM_CUDA(cudaGetDevice(&dev));
    const long key = ((long)dev << 24) | ((long)nt << 16) | ((long)p << 8) | KP;
    std::lock_guard<std::mutex> g(mu);
    for (auto &e : cache)
        if (e.first == key) return e.second;
    const int W = p + 1, nc = 2 * W + 2;
    std::vector<double> C((size_t)nc * nc, 0.0);
    for (int l = 0; l < nc; l++) {
        C[(size_t)l * nc] = 1.0;
        for (int m = 1; m <= l; m++)
            C[(size_t)l * nc + m] =
                C[(size_t)(l - 1) * nc + m - 1] + (m < l ? C[(size_t)(l - 1) * nc + m] : 0.0);
    }
    const SlotTables st = make_slot_tables();
    const size_t per = (size_t)(KP / 16) * 2 * KP * 16;  // floats per (position, slot)
    std::vector<float> h((size_t)4 * kSlots * per, 0.f);
    std::vector<double2> T((size_t)W * W);
    for (int cp = 0; cp < 4; cp++)
        for (int k = 0; k < kSlots; k++) {
            const double tx = st.dx[cp][k], ty = st.dy[cp][k];
            const double tn = 1.0 / (tx * tx + ty * ty);
            const double2 w2 = make_double2(tx * tn, -ty * tn), w1 = make_double2(-w2.x, -w2.y);
            double2 w2i = make_double2(1.0, 0.0);
            for (int i = 0; i < W; i++) {
                double2 w1j = make_double2(1.0, 0.0);
                for (int j = 0; j < W; j++) {
                    double b;
                    if (i == 0)
                        b = j == 0 ? 0.0 : 1.0;
                    else
                        b = j == 0 ? -1.0 / i : C[(size_t)(i + j - 1) * nc + (j - 1)];
                    T[(size_t)i * W + j] =
                        i + j >= nt ? cscal(cmul(w2i, w1j), b) : make_double2(0.0, 0.0);
                    w1j = cmul(w1j, w1);
                }
                w2i = cmul(w2i, w2);
            }
            float *img = h.data() + (size_t)(cp * kSlots + k) * per;
            for (int n = 0; n < 2 * W; n++)
                for (int kk = 0; kk < 2 * W; kk++) {
                    const double2 t = T[(size_t)(n < W ? n : n - W) * W + (kk < W ? kk : kk - W)];
                    const bool re_out = n < W, re_in = kk < W;
                    const double v = re_out ? (re_in ? t.x : -t.y) : (re_in ? t.y : t.x);
                    const float f = (float)v, fh = tf32_round_host(f);
                    const size_t at = slot_bimg_at(n, kk, KP);
                    img[at] = fh;
                    img[at + (size_t)KP * 16] = tf32_round_host(f - fh);
                }
        }
    float *d = nullptr;
    FMM_CUDA(cudaMalloc(&d, h.size() * sizeof(float)));
    FMM_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice, s));
    FMM_CUDA(cudaStreamSynchronize(s));
    cache.push_back({key, d});
    return d;
}

// The FP64 triangle on the DMMA kernel for the supported (MT, KS, NT).
template <int NT>
bool launch_split_triangle(const SegTable &sg, const int *boxes, const int *slots, const double *bs,
                           int ndc, int p, const double *binom, const double2 *mp, double2 *loc,
                           int ntiles, cudaStream_t s) {
    const int ks = (p + 1 + 3) / 4, mt = (p + 1 + 7) / 8;
#define FMM_SPLIT_CASE(MT_, KS_)                                                           \
    if (mt <= MT_ && ks <= KS_) {                                                          \
        launch_dmma<MT_, KS_, NT>(sg, boxes, slots, bs, ndc, p, binom, mp, loc, ntiles, s); \
        return true;                                                                       \
    }
    FMM_SPLIT_CASE(4, 8)
    FMM_SPLIT_CASE(5, 10)
    FMM_SPLIT_CASE(6, 12)
#undef FMM_SPLIT_CASE
    return false;
}

namespace {
struct SplitHold {
    SlotPlan spl;
};
}  // namespace

// 0: the order keeps the FP64 M2L
int split_triangle_order(int p) {
    const char *e = getenv("FMM2D_B200_SPLIT_NT");
    if (!e && p > 31) return 0;
    int nt = e ? atoi(e) : (4 * (p - 13) + 2) / 3 + 2;
    // the supported triangles: 8, 12, ..., 32
    if (nt < 8) nt = 8;
    nt = (nt + 3) / 4 * 4;
    return nt > 32 ? 0 : nt;
}

bool m2l_split_fp64(const Tree &T, const CauchyProblem &P, const double2 *mp, double2 *loc,
                    cudaStream_t s) {
    const int L = T.nlevels, p = P.p, W = p + 1;
    if (L < 2 || W < 20 || W > 48 || P.ndc > 128) return false;
    const int KP = slot_gemm_kp(W);
    const int nt = split_triangle_order(p);
    if (KP == 0 || nt == 0 || nt >= 2 * W - 1) return false;
    // planning first (nothing is launched when it fails)
    bool ok = false;
    const auto wp = m2l_cached<M2LWork>(P.m2l_cache, m2l_key(1, 8, 0), ok,
                                        [&](M2LWork &x) { return m2l_work(T, P, {8}, s, x); });
    if (!ok) return false;
    bool ok2 = false;
    const int tpt = 128 / P.ndc;
    const auto hp = m2l_cached<SplitHold>(P.m2l_cache, m2l_key(6, tpt, 0), ok2, [&](SplitHold &x) {
        return plan_slots(T, P.sset.pgh, P.tset.pgh, tpt, s, x.spl);
    });
    if (!ok2) return false;
    const M2LWork &w = *wp;
    if (w.ntarg == 0) return true;
    const int ntiles = w.ntiles(8);
    const float *bimg = split_tail_tables(p, KP, nt, s);
    // 1. the FP64 triangle, storing every local of levels >= 2 with points
    const double *binom = device_binomials(s);
    const SegTable sg = w.seg(8);
    const int *boxes = w.boxes.get();
    const double *bs = T.d_boxsize.get();
    bool launched = false;
    switch (nt) {
        case 8: launched = launch_split_triangle<8>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 12: launched = launch_split_triangle<12>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 16: launched = launch_split_triangle<16>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 20: launched = launch_split_triangle<20>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 24: launched = launch_split_triangle<24>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 28: launched = launch_split_triangle<28>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        case 32: launched = launch_split_triangle<32>(sg, boxes, w.slots.get(), bs, P.ndc, p, binom, mp, loc, ntiles, s); break;
        default: break;
    }
    if (!launched) return false;
    prof_set_count("m2l_split_nt", (double)nt);
    // 2. the tail on the tensor cores, level by level, added to the locals
    M2LCache *cache = P.m2l_cache;
    const bool deferred = cache && cache->deferred;
    DevBuf<int> err_own;
    if (!deferred) {
        err_own.alloc(1, s);
        FMM_CUDA(cudaMemsetAsync(err_own.get(), 0, sizeof(int), s));
    }
    int *errp = deferred ? cache->err : err_own.get();
    const size_t stride = (size_t)W * P.ndc;
    long long maxbox = 0;
    for (int l = 2; l <= L; l++) maxbox = std::max<long long>(maxbox, T.lend[l] - T.lstart[l]);
    DevBuf<float> arow((size_t)maxbox * P.ndc * 2 * KP, s);
    for (int l = 2; l <= L; l++) {
        const int g0 = 4 * (l - 2);
        if (g0 + 4 > hp->spl.nseg || hp->spl.tile_base[g0 + 4] == hp->spl.tile_base[g0]) continue;
        const int lo = T.lstart[l], nb = T.lend[l] - lo;
        slot_gemm_rows((long long)nb * P.ndc, P.ndc, W, KP, mp + (size_t)lo * stride, arow.get(), s);
        SlotGemmLevel g;
        g.level = l;
        g.lstart = lo;
        g.nd = P.ndc;
        g.W = W;
        g.KP = KP;
        g.arow = arow.get();
        g.bimg = bimg;
        g.out = loc + (size_t)lo * stride;
        g.oscale = 1.0;
        g.group = 27;
        if (!slot_gemm_tc_level(g, hp->spl, errp, s))
            throw FmmError(4, "split-precision M2L: unsupported tensor-core level shape");
    }
    if (!deferred && read_scalar(errp, s) != 0)
        throw FmmError(4, "tensor-core M2L: a wait for an MMA or operand barrier timed out");
    return true;
}

namespace {
struct SlotHold {
    M2LWork w;
    DevBuf<int2> dxy;
};
}  // namespace

bool plan_slots(const Tree &T, int spgh, int tpgh, int tile, cudaStream_t s, SlotPlan &sp) {
    sp = SlotPlan();
    if (T.nlevels < 2) return true;
    CauchyProblem P;
    P.sset.pgh = spgh;
    P.tset.pgh = tpgh;
    auto h = std::make_shared<SlotHold>();
    if (!m2l_work(T, P, {}, s, h->w)) return false;
    const M2LWork &w = h->w;
    sp.nseg = w.nseg;
    sp.ntarg = w.ntarg;
    sp.start = w.start;
    sp.count = w.count;
    if (w.ntarg == 0) return true;
    const SlotTables st = make_slot_tables();
    std::vector<int2> d(4 * kSlots);
    for (int c = 0; c < 4; c++)
        for (int k = 0; k < kSlots; k++) d[c * kSlots + k] = make_int2(st.dx[c][k], st.dy[c][k]);
    h->dxy.alloc(d.size(), s);
    // (a small pageable source is staged before the call returns)
    FMM_CUDA(cudaMemcpyAsync(h->dxy.get(), d.data(), d.size() * sizeof(int2),
                             cudaMemcpyHostToDevice, s));
    sp.boxes = w.boxes.get();
    sp.slots = w.slots.get();
    sp.dxy = h->dxy.get();
    sp.hold = h;
    retile_slots(sp, tile);
    return true;
}

void retile_slots(SlotPlan &sp, int tile) {
    sp.tile_base = tile_bases(sp.count, tile);
    sp.ntiles = sp.tile_base[sp.nseg];
}

namespace {
std::atomic<int> g_m2l_form[128];
}

// Form of the mixed-mode M2L for order p: FMM2D_B200_M2L ("simt", "tile"),
// else the setting for the order (fmm2d_b200_set_m2l_form, the autotuner),
// else windows on the tensor cores for the dense levels with slot tables
// for the rest.
int m2l_form(int p) {
    const char *mode = getenv("FMM2D_B200_M2L");
    if (mode && !strcmp(mode, "simt")) return kM2LSimt;
    if (mode && !strcmp(mode, "tile")) return kM2LTile;
    return (p >= 0 && p < 128) ? g_m2l_form[p].load() : kM2LWindow;
}

void set_m2l_form(int p, int form) {
    if (p >= 0 && p < 128) g_m2l_form[p].store(form);
}

bool m2l_fp32(const Tree &T, const CauchyProblem &P, const double2 *mp, double2 *loc,
              cudaStream_t s, float2 *mp32_out) {
    const int L = T.nlevels, p = P.p;
    if (L < 2 || p + 1 > 20) return false;
    const int form = m2l_form(p);
    const bool simt = form == kM2LSimt;
    const bool tile_only = form == kM2LTile;
    const int CH = P.ndc >= 2 ? 2 : 1;
    // FP32 copy of the multipoles of levels >= 2
    const int lo = T.lstart[2];
    const size_t stride = (size_t)(p + 1) * P.ndc;
    const size_t nv = (size_t)(T.nboxes - lo) * stride;
    DevBuf<float2> mp32_own;
    if (!mp32_out) mp32_own.alloc((size_t)T.nboxes * stride, s);
    float2 *mp32p = mp32_out ? mp32_out : mp32_own.get();
    {
        const double2 *src = mp + (size_t)lo * stride;
        float2 *dst = mp32p + (size_t)lo * stride;
        for_each((int64_t)nv, s, [=] __device__(int64_t i) {
            dst[i] = make_float2((float)src[i].x, (float)src[i].y);
        });
    }
    // the bounded waits' error flag: read at the end, or by the caller in
    // the deferred mode
    M2LCache *cache = P.m2l_cache;
    const bool deferred = cache && cache->deferred;
    DevBuf<int> err_own;
    if (!deferred && !P.m2l_err) err_own.alloc(1, s);
    int *errp = deferred ? cache->err : P.m2l_err ? P.m2l_err : err_own.get();
    if (errp != P.m2l_err) FMM_CUDA(cudaMemsetAsync(errp, 0, sizeof(int), s));
    const uint64_t done =
        (simt || tile_only) ? 0 : m2l_window_fp32(T, P, mp32p, loc, errp, s);
    const int wtile = simt ? kFp32Tile : kTcRows / CH;
    const bool hess = std::max(P.sset.n > 0 ? P.sset.pgh : 0, P.tset.n > 0 ? P.tset.pgh : 0) >= 3;
    const int nrows = simt || !m2l_exact_rows(p) ? 0 : (hess ? kM2LExactRowsHess : kM2LExactRows);
    bool ok = false;
    // (tiles of the tensor-core form, of its single remaining channels and
    // of the leading rows from one plan)
    const auto wp = m2l_cached<M2LWork>(cache, m2l_key(3, wtile + 1000 * nrows, done), ok, [&](M2LWork &x) {
        std::vector<int> tiles{wtile};
        if (!simt && CH == 2 && P.ndc % 2 != 0) tiles.push_back(kTcRows);
        if (nrows) tiles.push_back(rows_tile(nrows));
        return m2l_work(T, P, tiles, s, x, done);
    });
    if (!ok) return false;
    const M2LWork &w = *wp;
    if (w.ntarg > 0 && simt) {
        if (p + 1 <= 12)
            launch_fp32<12>(w, T, P, fp32_tables(p, 12, s), mp32p, loc, s);
        else
            launch_fp32<20>(w, T, P, fp32_tables(p, 20, s), mp32p, loc, s);
    } else if (w.ntarg > 0) {
        // tensor cores: K = N = 2 HALF with HALF = 12 (p < 12) or 20
        const int HALF = p + 1 <= 12 ? 12 : 20;
        const int KP = 2 * HALF;
        const float2 *tab0 = nullptr;
        const float *tab = tc_tables(p, KP, s, &tab0);
        // A TF32 x 3 product is accurate to about 2^-22, four times an FP32
        // product.  Measured on 10^5 uniform charges at eps 1e-6 (order 18),
        // the gradient at the sources then has a relative error of 1.6e-6
        // with the tensor-core forms against 2.0e-7 with the FP32 CUDA-core
        // form.  From order kM2LExactFrom on, the leading kM2LExactRows local
        // coefficients -- L_0 .. L_3, which carry most of the gradient at a
        // leaf's points -- are therefore summed in FP32 on the CUDA cores: on
        // the window levels from the windows (m2l_window.cu), on the other
        // levels by m2l_rows.
        auto launch = [&](auto deep, size_t deep_smem, auto wide, size_t wide_smem, auto rows,
                          int tile, int nr, int c0) {
            TcArgs a;
            a.seg = w.seg(tile);
            a.rseg = nr ? w.seg(rows_tile(nr)) : a.seg;
            a.boxes = w.boxes.get();
            a.slots = w.slots.get();
            a.bs = T.d_boxsize.get();
            a.ndc = P.ndc;
            a.c0 = c0;
            a.p = p;
            a.ntiles = w.ntiles(tile);
            const bool own = a.ntiles <= kNumSM;  // an SM for every tile
            a.ntcb = std::max(1, std::min(a.ntiles, kNumSM * 3));
            a.nrtiles = nr ? w.ntiles(rows_tile(nr)) : 0;
            a.Bimg = tab;
            a.T0 = tab0;
            a.Trows = nr ? fp32_tables(p, kRowsP1, s) : nullptr;
            a.mp32 = mp32p;
            a.loc = loc;
            a.err = errp;
            // one launch while every tile has an SM, else the rows apart
            const bool apart = nr && a.ntiles + a.nrtiles > kNumSM;
            const int blocks = a.ntcb + (apart ? 0 : a.nrtiles);
            if (own) {
                raise_smem_limit(deep, deep_smem);
                deep<<<blocks, kTcRows, deep_smem, s>>>(a);
            } else {
                raise_smem_limit(wide, wide_smem);
                wide<<<blocks, kTcRows, wide_smem, s>>>(a);
            }
            FMM_CHECK_LAUNCH();
            if (apart) {
                const size_t sm = (size_t)kSlots * nr * kRowsP1 * sizeof(float2);
                rows<<<std::min(a.nrtiles, kNumSM * 8), kTcRows, sm, s>>>(a);
                FMM_CHECK_LAUNCH();
            }
        };
        auto form = [&](auto ch, auto half, auto nr, auto rows, int tile, int c0) {
            constexpr int C = decltype(ch)::value, H = decltype(half)::value,
                          N = decltype(nr)::value;
            launch(m2l_tc_kernel<C, H, N, 2>, tc_smem_bytes<H, 2>(), m2l_tc_kernel<C, H, N, 1>,
                   tc_smem_bytes<H, 1>(), rows, tile, N, c0);
        };
        auto one = [&](auto ch, int tile, int c0) {
            constexpr int C = decltype(ch)::value;
            constexpr std::integral_constant<int, 0> none{};
            constexpr std::integral_constant<int, kM2LExactRows> nr{};
            constexpr std::integral_constant<int, kM2LExactRowsHess> nrh{};
            constexpr std::integral_constant<int, 12> h12{};
            constexpr std::integral_constant<int, 20> h20{};
            auto rows = m2l_rows_kernel<C, kM2LExactRows>;
            if (HALF == 12) form(ch, h12, none, rows, tile, c0);
            else if (nrows == kM2LExactRowsHess)
                form(ch, h20, nrh, m2l_rows_kernel<C, kM2LExactRowsHess>, tile, c0);
            else if (nrows) form(ch, h20, nr, rows, tile, c0);
            else form(ch, h20, none, rows, tile, c0);
        };
        int c0 = 0;
        if (CH == 2)
            for (; P.ndc - c0 >= 2; c0 += 2) one(std::integral_constant<int, 2>{}, wtile, c0);
        // remaining single channels, one channel per row
        for (; c0 < P.ndc; c0++) one(std::integral_constant<int, 1>{}, kTcRows, c0);
    }
    if (errp == err_own.get() && read_scalar(errp, s) != 0)
        throw FmmError(4, "tensor-core M2L: a wait for an MMA or operand barrier timed out");
    return true;
}

}  // namespace fmm2d
