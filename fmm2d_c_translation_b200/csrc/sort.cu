// sort.cu -- stable LSD radix sort of (uint32 key, uint32 value) pairs.
//
// Used by the tree builder: to order the points by their path keys (the
// child digits of every level, most significant first), and to put the
// points of large leaves back in input order, which is the stable
// permutation the reference's repeated partition
// (c_translation/src/pts_tree2d.c:670-765) produces.
//
// 8-bit digits.  One pass over the keys counts the digits of every pass;
// then each pass reads and writes the pairs once: a tile counts its digits,
// publishes the counts, finds the counts of the tiles before it by looking
// back over what they published (Merrill and Garland's decoupled look-back),
// ranks its items stably in shared memory (warp match for ties inside a
// warp, per-warp counts across warps, a running per-digit count across
// rounds) and writes them out in digit order, so that consecutive threads
// write consecutive addresses of the same digit run.  Tiles take their
// number from a counter, so the tiles before a running one have all begun;
// a wait that lasts too long all the same ends with the thread counting the
// earlier keys itself.  Up to one tile, all passes run in one block.
//
// Counting and scanning per pass instead (a histogram, three scan launches
// and a scatter per digit) took 15 launches for the three digits of 10^5
// points and read the keys twice per pass.  Keys and levels of the tree: 300
// points 0.18 -> 0.11 ms, 10^5 0.24 -> 0.15, 4e5 clustered 0.77 -> 0.45,
// 10^7 + 10^7 1.92 -> 1.74 ms.
#include "common.cuh"
#include "sort.cuh"

#include <algorithm>
#include <stdlib.h>
#include <string.h>

namespace fmm2d {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRadix = 256;
constexpr int kMaxPasses = 4;
constexpr int kMaxSpin = 1 << 20;

// Tile states: 2 flag bits over a count, of 30 bits in the 32-bit form and of
// 62 in the 64-bit one, which 2^30 and more items take.
template <class St>
struct TileState {
    static constexpr int kBits = 8 * sizeof(St) - 2;
    static constexpr St kOwn = (St)1 << kBits, kIncl = (St)2 << kBits, kCount = kOwn - 1;
};

// Digit counts of every pass.
__global__ void __launch_bounds__(kThreads) radix_hist_kernel(const uint32_t *__restrict__ keys,
                                                              int64_t n, int lo_bit, int passes,
                                                              int *__restrict__ hist) {
    __shared__ int h[kMaxPasses][kRadix];
    for (int p = 0; p < passes; p++) h[p][threadIdx.x] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * kThreads;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) {
        const uint32_t k = keys[i] >> lo_bit;
        for (int p = 0; p < passes; p++) atomicAdd(&h[p][(k >> (8 * p)) & 0xff], 1);
    }
    __syncthreads();
    for (int p = 0; p < passes; p++)
        if (h[p][threadIdx.x]) atomicAdd(&hist[p * kRadix + threadIdx.x], h[p][threadIdx.x]);
}

// Exclusive scan of one value per thread over the block.
__device__ __forceinline__ int block_excl(int v, int *wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int pre = 0;
    for (int w = 0; w < warp; w++) pre += wsum[w];
    return pre + incl - v;
}

template <int ROUNDS>
struct TileSmem {
    uint32_t sk[kThreads * ROUNDS], sv[kThreads * ROUNDS];
    int lstart[kRadix];  // tile-local start of each digit
    int gdelta[kRadix];  // global position - local position
    int run[kRadix];
    int wc[kWarps][kRadix];
    int wsum[kWarps];
    int tile;
};

// Ranks the tile's items (kr, vr in round order) stably by the digit at
// `shift` into S.sk, S.sv; S.lstart holds the digits' starts.
template <int ROUNDS>
__device__ __forceinline__ void rank_tile(TileSmem<ROUNDS> &S, const uint32_t *kr,
                                          const uint32_t *vr, int cnt, int shift) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    S.run[tid] = 0;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        if (r * kThreads >= cnt) break;
#pragma unroll
        for (int w = 0; w < kWarps; w++) S.wc[w][tid] = 0;
        __syncthreads();
        const bool valid = r * kThreads + tid < cnt;
        const int d = valid ? (int)((kr[r] >> shift) & 0xff) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(peers & lt_mask);
        if (valid && rank == 0) S.wc[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            int pos = S.lstart[d] + S.run[d] + rank;
            for (int w = 0; w < warp; w++) pos += S.wc[w][d];
            S.sk[pos] = kr[r];
            S.sv[pos] = vr[r];
        }
        __syncthreads();
        int add = 0;
#pragma unroll
        for (int w = 0; w < kWarps; w++) add += S.wc[w][tid];
        S.run[tid] += add;
    }
    __syncthreads();
}

// One pass over all tiles; vin null: the values are the positions.
template <int ROUNDS, class St>
__global__ void __launch_bounds__(kThreads) radix_pass_kernel(
    const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
    uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, int64_t n, int shift,
    const int *__restrict__ hist, int *__restrict__ next, volatile St *state) {
    constexpr int kTile = kThreads * ROUNDS;
    constexpr St kOwn = TileState<St>::kOwn, kIncl = TileState<St>::kIncl;
    __shared__ TileSmem<ROUNDS> S;
    const int tid = threadIdx.x;
    if (tid == 0) S.tile = atomicAdd(next, 1);
    S.run[tid] = 0;
    __syncthreads();
    const int tile = S.tile;
    const int64_t base = (int64_t)tile * kTile;
    const int cnt = n - base < kTile ? (int)(n - base) : kTile;
    uint32_t kr[ROUNDS], vr[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int o = r * kThreads + tid;
        kr[r] = o < cnt ? kin[base + o] : 0u;
        vr[r] = o < cnt ? (vin ? vin[base + o] : (uint32_t)(base + o)) : 0u;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; r++)
        if (r * kThreads + tid < cnt) atomicAdd(&S.run[(kr[r] >> shift) & 0xff], 1);
    __syncthreads();
    const int own = S.run[tid];
    volatile St *st = state + (size_t)tile * kRadix + tid;
    *st = (tile == 0 ? kIncl : kOwn) | (St)own;
    const int lst = block_excl(own, S.wsum);
    const int gst = block_excl(hist[tid], S.wsum);  // the digit's first place
    S.lstart[tid] = lst;
    __syncthreads();
    rank_tile<ROUNDS>(S, kr, vr, cnt, shift);
    // the digit's items in the tiles before this one
    uint32_t before = 0;
    int spins = 0;
    for (int t = tile - 1; t >= 0;) {
        const St v = state[(size_t)t * kRadix + tid];
        if (v >= kOwn) {
            before += (uint32_t)(v & TileState<St>::kCount);
            if (v >= kIncl) break;
            t--;
        } else if (++spins > kMaxSpin) {
            before = 0;
            for (int64_t i = 0; i < base; i++) before += ((kin[i] >> shift) & 0xff) == (uint32_t)tid;
            break;
        }
    }
    if (tile > 0) *st = kIncl | (St)(before + (uint32_t)own);
    S.gdelta[tid] = gst + (int)before - lst;
    __syncthreads();
    for (int i = tid; i < cnt; i += kThreads) {
        const uint32_t key = S.sk[i];
        const int64_t g = (int64_t)S.gdelta[(key >> shift) & 0xff] + i;
        kout[g] = key;
        vout[g] = S.sv[i];
    }
}

// All passes of at most one tile in one block.
constexpr int kOneRounds = 16;
__global__ void __launch_bounds__(kThreads) radix_one_kernel(
    const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, int n, int lo_bit,
    int key_bits) {
    __shared__ TileSmem<kOneRounds> S;
    const int tid = threadIdx.x;
    uint32_t kr[kOneRounds], vr[kOneRounds];
#pragma unroll
    for (int r = 0; r < kOneRounds; r++) {
        const int o = r * kThreads + tid;
        kr[r] = o < n ? kin[o] : 0u;
        vr[r] = o < n ? (vin ? vin[o] : (uint32_t)o) : 0u;
    }
    for (int shift = lo_bit; shift < key_bits; shift += 8) {
        S.run[tid] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kOneRounds; r++)
            if (r * kThreads + tid < n) atomicAdd(&S.run[(kr[r] >> shift) & 0xff], 1);
        __syncthreads();
        const int lst = block_excl(S.run[tid], S.wsum);
        S.lstart[tid] = lst;
        __syncthreads();
        rank_tile<kOneRounds>(S, kr, vr, n, shift);
#pragma unroll
        for (int r = 0; r < kOneRounds; r++) {
            const int o = r * kThreads + tid;
            if (o < n) {
                kr[r] = S.sk[o];
                vr[r] = S.sv[o];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kOneRounds; r++) {
        const int o = r * kThreads + tid;
        if (o < n) {
            kout[o] = kr[r];
            vout[o] = vr[r];
        }
    }
}

template <int ROUNDS, class St>
void sort_passes(const uint32_t *kin, const uint32_t *vin, uint32_t *const k[2],
                 uint32_t *const v[2], int64_t n, int lo_bit, int passes, cudaStream_t s) {
    const int64_t tile = (int64_t)kThreads * ROUNDS;
    const int ntiles = (int)((n + tile - 1) / tile);
    // per pass the tile states, then digit counts and the tile counter
    const size_t per = (size_t)ntiles * kRadix, head = (size_t)passes * (kRadix + 1);
    DevBuf<int> work(passes * per * (sizeof(St) / sizeof(int)) + head, s);
    work.zero(s);
    St *state = reinterpret_cast<St *>(work.get());
    int *hist = reinterpret_cast<int *>(state + passes * per), *next = hist + passes * kRadix;
    const int blocks = (int)std::min<int64_t>((n + 2047) / 2048, kNumSM * 4);
    radix_hist_kernel<<<blocks, kThreads, 0, s>>>(kin, n, lo_bit, passes, hist);
    FMM_CHECK_LAUNCH();
    for (int p = 0; p < passes; p++) {
        radix_pass_kernel<ROUNDS, St><<<ntiles, kThreads, 0, s>>>(
            p == 0 ? kin : k[(p - 1) & 1], p == 0 ? vin : v[(p - 1) & 1], k[p & 1], v[p & 1], n,
            lo_bit + 8 * p, hist + p * kRadix, next + p, state + p * per);
        FMM_CHECK_LAUNCH();
    }
}

}  // namespace

int radix_sort_into(const uint32_t *kin, const uint32_t *vin, uint32_t *const k[2],
                    uint32_t *const v[2], int64_t n, int key_bits, cudaStream_t s, int lo_bit) {
    if (n <= 0) return 0;
    const int passes = std::max(1, (key_bits - lo_bit + 7) / 8);
    if (passes > kMaxPasses) throw FmmError(4, "sort: more than 32 key bits");
    if (n <= kThreads * kOneRounds) {
        radix_one_kernel<<<1, kThreads, 0, s>>>(kin, vin, k[0], v[0], (int)n, lo_bit, key_bits);
        FMM_CHECK_LAUNCH();
        return 0;
    }
    // 64-bit states from 2^30 items on (FMM2D_B200_SORT_WIDE=1: always); tiles
    // of 1,024 items while larger ones would leave SMs without one
    const char *e = getenv("FMM2D_B200_SORT_WIDE");
    const bool wide = n > (int64_t)TileState<uint32_t>::kCount || (e && !strcmp(e, "1"));
    const bool small = n < (int64_t)kThreads * 16 * kNumSM;
    auto sort = wide ? (small ? sort_passes<4, unsigned long long> : sort_passes<16, unsigned long long>)
                     : (small ? sort_passes<4, uint32_t> : sort_passes<16, uint32_t>);
    sort(kin, vin, k, v, n, lo_bit, passes, s);
    return (passes - 1) & 1;
}

void radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *keys_tmp,
                      uint32_t *vals_tmp, int64_t n, int key_bits,
                      cudaStream_t s, int lo_bit) {
    if (n <= 1 || key_bits <= lo_bit) return;
    if (n <= kThreads * kOneRounds) {
        // (one block reads everything before it writes)
        radix_one_kernel<<<1, kThreads, 0, s>>>(keys, vals, keys, vals, (int)n, lo_bit, key_bits);
        FMM_CHECK_LAUNCH();
        return;
    }
    uint32_t *const k[2] = {keys_tmp, keys}, *const v[2] = {vals_tmp, vals};
    if (radix_sort_into(keys, vals, k, v, n, key_bits, s, lo_bit) == 0) {
        FMM_CUDA(cudaMemcpyAsync(keys, keys_tmp, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        FMM_CUDA(cudaMemcpyAsync(vals, vals_tmp, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
}

}  // namespace fmm2d
