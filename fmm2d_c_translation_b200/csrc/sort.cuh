// sort.cuh -- stable radix sort of (key, value) pairs on the device.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmm2d {

// Stable sort of n (key, value) pairs by bits [lo_bit, key_bits) of key
// (8-bit digits from lo_bit up).  keys_tmp / vals_tmp are scratch arrays of
// n elements; the result is left in keys / vals.
void radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *keys_tmp,
                      uint32_t *vals_tmp, int64_t n, int key_bits,
                      cudaStream_t s, int lo_bit = 0);

// The same sort out of place: the pairs (kin, vin), or (kin, position) when
// vin is null, sorted into k[r], v[r]; returns r (0 or 1).  k[0] and v[0] are
// written while kin and vin are still read, so they must be other arrays.
int radix_sort_into(const uint32_t *kin, const uint32_t *vin, uint32_t *const k[2],
                    uint32_t *const v[2], int64_t n, int key_bits, cudaStream_t s,
                    int lo_bit = 0);

}  // namespace fmm2d
