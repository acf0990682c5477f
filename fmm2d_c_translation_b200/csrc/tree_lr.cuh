// tree_lr.cuh -- colleagues and level restriction of a key-built tree in one
// cooperative launch (included by tree.cu).
//
// computecoll (tree_routs2d.c:140-195) and pts_tree_fix_lr (pts_tree2d.c:
// 767-964) are sequences of short steps over the boxes of one level, each
// depending on the one before: about seven per level, most of them a few
// microseconds of dependent loads.  As launches, with a host synchronisation
// per level for the counts, they took 1.08 ms on 4e5 clustered points (12
// levels; here 0.43), 0.87 ms on 5e4 (0.35), 2.76 ms on the 8e6 points of a
// boundary curve (18 levels; 2.10, bound by the colleagues' loads).  Here they
// are phases of one kernel with a grid-wide barrier between them; counts stay
// on the device, and one status read at the end gives the host the new level
// ranges.  The boxes' arrays are sized with room for the added boxes; when that
// does not suffice the kernel stops before writing past the end and the host
// builds again with more room.
#pragma once

// The arrays of one numbering of the boxes (the reorganisations copy from
// one set to the other).
struct LrSet {
    double2 *cen;
    int *lev, *par, *nch, *chi, *flg;
    int2 *rs, *rt;
};

// What the kernel reports (host layout).
struct LrOut {
    int status;   // 1: the boxes did not fit
    int nboxes;
    int set;      // set that holds the result
    int big;      // bit 0 / 1: a leaf of more than kLeafSort sources / targets
    int lstart[kRefLevels], lend[kRefLevels];
};

// One block of 1024 threads per SM: a quarter of the arrivals at each of the
// grid barriers (four blocks of 256: 2.48 ms on the boundary curve's points).
constexpr int kLrThreads = 1024;
constexpr int kLrBlocks = kNumSM;

struct LrArgs {
    LrSet a, b;
    int *nnb, *nb;
    KeyView ks, kt;
    const double *dcol, *d1, *d2, *d3, *bsl;  // per level: distances, box sizes
    int L, nroots, nboxes, cap, leaf_sort;
    int lstart[kRefLevels], lend[kRefLevels];
    int *any;      // [0]: flagged boxes, [1]: flag++ boxes; zero at the start
    int *levcnt;   // [kRefLevels] split boxes per level; zero at the start
    int *blkcnt;   // [2][kLrBlocks] items selected per block
    LrOut *out;
};

__device__ __forceinline__ int lr_block_sum(int v, int *sh) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < kLrThreads / 32; w++) t += sh[w];
    return t;
}

// Colleagues of the boxes [lo, hi) of one level: W lanes per four siblings,
// whose candidates -- the children of their parent's colleagues, in order, at
// most 36 -- are the same boxes.  Bound by the chain of dependent loads
// (parent, colleagues, children, centers; the next siblings' first two are
// loaded ahead).
template <int W>
__device__ __forceinline__ void lr_colleagues_w(const LrSet &S, int *nnb, int *nb, int lo, int hi,
                                                double d, int gt, int nt) {
    constexpr int NU = (36 + W - 1) / W;
    constexpr unsigned kMask = W == 32 ? 0xffffffffu : (1u << (W & 31)) - 1u;
    const int sub = threadIdx.x & (W - 1), sh0 = threadIdx.x & 31 & ~(W - 1);
    const unsigned lt = (1u << sub) - 1u;
    const int ng = (hi - lo) >> 2, step = nt / W;
    // (whole warps stay in the loop: the ballots take all lanes)
    const int rounds = (ng + step - 1) / step;
    int g = gt / W, dad = 0, n = 0;
    if (g < ng) {
        dad = S.par[lo + 4 * g];
        n = 4 * nnb[dad];
    }
    for (int r = 0; r < rounds; r++) {
        const int b0 = g < ng ? lo + 4 * g : -1;
        int kb[NU];
        double2 ck[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const int e = sub + W * u;
            kb[u] = e < n ? S.chi[4 * nb[9 * dad + (e >> 2)] + (e & 3)] : -1;
        }
        g += step;
        int dad2 = 0, n2 = 0;
        if (r + 1 < rounds && g < ng) {
            dad2 = S.par[lo + 4 * g];
            n2 = 4 * nnb[dad2];
        }
#pragma unroll
        for (int u = 0; u < NU; u++) ck[u] = kb[u] >= 0 ? S.cen[kb[u]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int b = b0 + j;
            const double2 cb = b0 >= 0 ? S.cen[b] : make_double2(0.0, 0.0);
            int base = 0;
#pragma unroll
            for (int u = 0; u < NU; u++) {
                const bool ok = kb[u] >= 0 && within(ck[u], cb, d);
                const unsigned m = (__ballot_sync(0xffffffffu, ok) >> sh0) & kMask;
                const int pos = base + __popc(m & lt);
                if (ok && pos < 9) nb[9 * b + pos] = kb[u];
                base += __popc(m);
            }
            if (b0 < 0) continue;
            const int cnt = min(base, 9);
            if (sub == 0) nnb[b] = cnt;
            for (int k = sub; k < 9; k += W)
                if (k >= cnt) nb[9 * b + k] = -1;
        }
        dad = dad2;
        n = n2;
    }
}

// A warp per four siblings while that gives every warp at most two rounds
// (fewer loads in a row: clusters' levels), else eight lanes, which keep four
// chains in flight per warp.  Measured: the colleagues and flags of 4e5
// clustered points 0.49 ms with 32 lanes, 0.61 with 8; of 10^7 + 10^7 uniform
// points 0.38 and 0.32 ms.
__device__ __forceinline__ void lr_colleagues(const LrSet &S, int *nnb, int *nb, int lo, int hi,
                                              double d, int gt, int nt) {
    if ((hi - lo) >> 2 <= 2 * (nt >> 5))
        lr_colleagues_w<32>(S, nnb, nb, lo, hi, d, gt, nt);
    else
        lr_colleagues_w<8>(S, nnb, nb, lo, hi, d, gt, nt);
}

// Splits the selected (flag > 0) items of a list of n1 + n2 boxes (box lo + i
// below n1, else tlo + i - n1), four children per box appended in item
// order from box nb0 on; blkcnt holds the blocks' counts of their chunks.
__device__ __forceinline__ void lr_split(const LrArgs &A, const LrSet &S, int lo, int n1, int tlo,
                                         int n2, int nb0, const int *blkcnt, int *sh) {
    const int n = n1 + n2, chunk = (n + (int)gridDim.x - 1) / (int)gridDim.x;
    const int i0 = min(n, (int)blockIdx.x * chunk), i1 = min(n, i0 + chunk);
    int pre = 0;
    for (int w = threadIdx.x; w < (int)blockIdx.x; w += kLrThreads) pre += blkcnt[w];
    int run = lr_block_sum(pre, sh);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int ib = i0; ib < i1; ib += kLrThreads) {
        const int i = ib + (int)threadIdx.x;
        const int b = i < n1 ? lo + i : tlo + (i - n1);
        const bool hit = i < i1 && S.flg[b] > 0;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        __syncthreads();
        if (lane == 0) sh[warp] = __popc(m);
        __syncthreads();
        int off = run + __popc(m & ((1u << lane) - 1u));
#pragma unroll
        for (int w = 0; w < kLrThreads / 32; w++) {
            if (w < warp) off += sh[w];
            run += sh[w];
        }
        if (!hit) continue;
        const int base = nb0 + 4 * off;
        const double2 c = S.cen[b];
        const int nl = S.lev[b] + 1, cf = S.flg[b] == 1 ? 3 : 0;
        const double bs = A.bsl[nl];
        S.nch[b] = 4;
        // point ranges of the children: by the digit of their level
        auto split = [&](const KeyView &kv, int2 r, int2 *o) {
            int at = r.x;
            for (int j = 0; j < 4; j++) {
                int e = r.y;
                if (j < 3) {
                    int x = at, y = r.y;
                    while (x < y) {
                        const int mid = x + ((y - x) >> 1);
                        if (key_digit(kv, mid, nl) < j + 1) x = mid + 1; else y = mid;
                    }
                    e = x;
                }
                o[base + j] = make_int2(at, e);
                at = e;
            }
        };
        split(A.ks, S.rs[b], S.rs);
        split(A.kt, S.rt[b], S.rt);
        *reinterpret_cast<int4 *>(S.chi + 4 * (size_t)b) =
            make_int4(base, base + 1, base + 2, base + 3);
        for (int j = 0; j < 4; j++) {
            const int kb = base + j;
            S.cen[kb] = child_center(c, bs, j);
            S.par[kb] = b;
            S.nch[kb] = 0;
            S.lev[kb] = nl;
            S.flg[kb] = cf;
            *reinterpret_cast<int4 *>(S.chi + 4 * (size_t)kb) = make_int4(-1, -1, -1, -1);
        }
    }
}

// pts_tree_reorg: box b's number when every level's range is followed by its
// tail, both in their order.
struct LrMap {
    int ls[kRefLevels], le[kRefLevels], ts[kRefLevels], te[kRefLevels], ns[kRefLevels];
    __device__ __forceinline__ int at(int b, int l) const {
        if (l < 2) return b;
        if (b >= ls[l] && b < le[l]) return ns[l] + (b - ls[l]);
        return ns[l] + (le[l] - ls[l]) + (b - ts[l]);
    }
};

__global__ void __launch_bounds__(kLrThreads, 1) tree_lr_kernel(LrArgs A) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ LrMap M;
    __shared__ int sh[kLrThreads / 32];
    const int tid = threadIdx.x, gt = blockIdx.x * kLrThreads + tid, nt = gridDim.x * kLrThreads;
    const int L = A.L;
    int *nnb = A.nnb, *nb = A.nb;
    LrSet S = A.a, O = A.b;
    int nboxes = A.nboxes, status = 0;
    for (int l = tid; l <= L; l += kLrThreads) {
        M.ls[l] = A.lstart[l];
        M.le[l] = A.lend[l];
        M.ts[l] = M.te[l] = 0;
    }
    __syncthreads();
    // colleagues of every level
    auto all_colleagues = [&]() {
        for (int b = gt; b < A.nroots; b += nt) {
            nnb[b] = 1;
            nb[9 * b] = b;
            for (int k = 1; k < 9; k++) nb[9 * b + k] = -1;
        }
        for (int l = 1; l <= L; l++) {
            grid.sync();
            lr_colleagues(S, nnb, nb, M.ls[l], M.le[l], A.dcol[l], gt, nt);
        }
    };
    // the copy into the other set in the new numbering; flags other than
    // flag++ are cleared, and a remaining flag++ box is noted in any[1]
    auto reorg = [&]() {
        if (tid == 0) {
            int cur = M.ls[min(2, L)];
            for (int l = 0; l <= L; l++) {
                M.ns[l] = l < 2 ? M.ls[l] : cur;
                if (l >= 2) cur += (M.le[l] - M.ls[l]) + (M.te[l] - M.ts[l]);
            }
        }
        __syncthreads();
        for (int b = gt; b < nboxes; b += nt) {
            const int l = S.lev[b], m = M.at(b, l);
            O.rs[m] = S.rs[b];
            O.rt[m] = S.rt[b];
            O.cen[m] = S.cen[b];
            O.lev[m] = l;
            O.nch[m] = S.nch[b];
            const int f = S.flg[b] == 3 ? 3 : 0;
            O.flg[m] = f;
            if (f) A.any[1] = 1;
            const int pb = S.par[b];
            O.par[m] = pb < 0 ? -1 : M.at(pb, l - 1);
            const int4 c = *reinterpret_cast<const int4 *>(S.chi + 4 * (size_t)b);
            *reinterpret_cast<int4 *>(O.chi + 4 * (size_t)m) =
                c.x < 0 ? make_int4(-1, -1, -1, -1)
                        : make_int4(M.at(c.x, l + 1), M.at(c.y, l + 1), M.at(c.z, l + 1),
                                    M.at(c.w, l + 1));
        }
        __syncthreads();
        if (tid == 0)
            for (int l = 2; l <= L; l++) {
                const int n = (M.le[l] - M.ls[l]) + (M.te[l] - M.ts[l]);
                M.ls[l] = M.ns[l];
                M.le[l] = M.ns[l] + n;
            }
        __syncthreads();
        for (int l = tid; l <= L; l += kLrThreads) M.ts[l] = M.te[l] = 0;
        const LrSet t = S;
        S = O;
        O = t;
        __syncthreads();
    };
    for (int b = gt; b < nboxes; b += nt) S.flg[b] = 0;
    all_colleagues();
    bool go = L >= 2;
    if (go) {
        grid.sync();
        // flag: leaves among the granddad's colleagues that touch the dad
        // (the same for four siblings: one thread per group and colleague)
        const int lo = M.ls[2], n = (M.le[L] - lo) / 4 * 9;
        for (int t = gt; t < n; t += nt) {
            const int b = lo + 4 * (t / 9), k = t % 9;
            const int dad = S.par[b], gd = S.par[dad];
            if (k >= nnb[gd]) continue;
            const int jb = nb[9 * gd + k];
            if (S.nch[jb] == 0 && within(S.cen[jb], S.cen[dad], A.d1[S.lev[b]])) {
                S.flg[jb] = 1;
                A.any[0] = 1;
            }
        }
        grid.sync();
        go = *(volatile int *)A.any != 0;
    }
    if (go) {
        for (int l = L; l >= 1; l--) {
            // flag+: leaves among the dad's colleagues that touch a flagged box
            const int lo = M.ls[l], n = (M.le[l] - lo) * 9;
            const double dist = A.d2[l];
            for (int t = gt; t < n; t += nt) {
                const int b = lo + t / 9, k = t % 9;
                const int f = S.flg[b];
                if (f != 1 && f != 2) continue;
                const int dad = S.par[b];
                if (k >= nnb[dad]) continue;
                const int jb = nb[9 * dad + k];
                if (S.nch[jb] == 0 && S.flg[jb] == 0 && within(S.cen[jb], S.cen[b], dist))
                    S.flg[jb] = 2;
            }
            grid.sync();
        }
        // split the flagged boxes of the original levels 1 .. L-2
        {
            const int lo = M.ls[1], n = L >= 3 ? M.le[L - 2] - lo : 0;
            const int chunk = (n + (int)gridDim.x - 1) / (int)gridDim.x;
            const int i0 = min(n, (int)blockIdx.x * chunk), i1 = min(n, i0 + chunk);
            int c = 0;
            for (int i = i0 + tid; i < i1; i += kLrThreads)
                if (S.flg[lo + i] > 0) {
                    c++;
                    atomicAdd(&A.levcnt[S.lev[lo + i]], 1);
                }
            c = lr_block_sum(c, sh);
            if (tid == 0) A.blkcnt[blockIdx.x] = c;
            grid.sync();
            if (tid == 0) {
                int at = nboxes;
                for (int l = 1; l <= L - 2; l++) {
                    M.ts[l + 1] = at;
                    at += 4 * ((volatile int *)A.levcnt)[l];
                    M.te[l + 1] = at;
                }
                sh[0] = at;
            }
            __syncthreads();
            const int nb1 = sh[0];
            __syncthreads();
            if (nb1 > A.cap) {
                status = 1;
                go = false;
            } else {
                lr_split(A, S, lo, n, 0, 0, nboxes, A.blkcnt, sh);
                nboxes = nb1;
            }
        }
    }
    if (go) {
        grid.sync();
        reorg();
        grid.sync();
        all_colleagues();
        grid.sync();
        go = ((volatile int *)A.any)[1] != 0;
    }
    if (go) {
        for (int l = 2; l <= L - 2; l++) {
            // updateflags (tree_routs2d.c:197-252) on the level and its tail:
            // a flag++ box is split only when a child of one of its
            // colleagues has children and touches it
            const int lo = M.ls[l], n1 = M.le[l] - lo, tlo = M.ts[l], n2 = M.te[l] - tlo;
            const int n = n1 + n2, chunk = (n + (int)gridDim.x - 1) / (int)gridDim.x;
            const int i0 = min(n, (int)blockIdx.x * chunk), i1 = min(n, i0 + chunk);
            const double dist = A.d3[l];
            int c = 0;
            for (int i = i0 + tid; i < i1; i += kLrThreads) {
                const int b = i < n1 ? lo + i : tlo + (i - n1);
                const int f0 = S.flg[b];
                int f = f0 > 0 ? 1 : 0;
                if (f0 == 3) {
                    f = 0;
                    const double2 cb = S.cen[b];
                    for (int k = 0; k < nnb[b] && !f; k++) {
                        const int jb = nb[9 * b + k];
                        for (int j = 0; j < 4; j++) {
                            const int kb = S.chi[4 * jb + j];
                            if (kb >= 0 && S.nch[kb] > 0 && within(S.cen[kb], cb, dist)) {
                                f = 1;
                                break;
                            }
                        }
                    }
                    S.flg[b] = f;
                }
                c += f;
            }
            c = lr_block_sum(c, sh);
            int *bc = A.blkcnt + (l & 1) * kLrBlocks;
            if (tid == 0) bc[blockIdx.x] = c;
            grid.sync();
            int tot = 0;
            for (int w = tid; w < (int)gridDim.x; w += kLrThreads) tot += bc[w];
            tot = lr_block_sum(tot, sh);
            if (tid == 0) {
                M.ts[l + 1] = nboxes;
                M.te[l + 1] = nboxes + 4 * tot;
            }
            __syncthreads();
            if (tot == 0) continue;
            if (nboxes + 4 * tot > A.cap) {
                status = 1;
                break;
            }
            lr_split(A, S, lo, n1, tlo, n2, nboxes, bc, sh);
            nboxes += 4 * tot;
            grid.sync();
            // colleagues of the new boxes from their dad's (current) list
            lr_colleagues(S, nnb, nb, M.ts[l + 1], M.te[l + 1], A.dcol[l + 1], gt, nt);
            grid.sync();
        }
        if (status == 0) {
            grid.sync();
            reorg();
            grid.sync();
            all_colleagues();
        }
    }
    // leaves of more points than one warp sorts
    int big = 0;
    for (int b = gt; b < nboxes; b += nt)
        if (S.nch[b] == 0) {
            const int2 r = S.rs[b], t = S.rt[b];
            if (r.y - r.x > A.leaf_sort) big |= 1;
            if (t.y - t.x > A.leaf_sort) big |= 2;
        }
    if (big) atomicOr(&A.out->big, big);
    if (gt == 0) {
        A.out->status = status;
        A.out->nboxes = nboxes;
        A.out->set = S.cen == A.a.cen ? 0 : 1;
        for (int l = 0; l <= L; l++) {
            A.out->lstart[l] = M.ls[l];
            A.out->lend[l] = M.le[l];
        }
    }
}
