// Packed genotype words (16 codes of two bits), shared by the kernels that lay genotypes out for the tensor cores.
#pragma once
#include <cstdint>

namespace sg {

// 16 packed codes (00 two copies, 01 missing, 10 one, 11 none) to copies, in place
__device__ __forceinline__ uint32_t pack_copies(uint32_t x, int fill, uint32_t valid) {
  const uint32_t lo = x & 0x55555555u, hi = (x >> 1) & 0x55555555u, miss = lo & ~hi;
  uint32_t one = hi & ~lo, two = ~(hi | lo) & 0x55555555u;
  if (fill == 1) one |= miss;
  if (fill == 2) two |= miss;
  return (one & valid) | ((two & valid) << 1);
}

// the fields of the first ``left`` samples of a word (bit 2 i for sample i)
__device__ __forceinline__ uint32_t valid_fields(int64_t left) {
  return left >= 16 ? 0x55555555u : left <= 0 ? 0u : 0x55555555u & ((1u << (2 * left)) - 1u);
}

// 16 x 16 fields of two bits transposed: swaps of the off-diagonal d x d blocks
__device__ __forceinline__ void transpose_fields(uint32_t (&w)[16]) {
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) {
    const uint32_t mask = d == 8 ? 0x0000FFFFu : d == 4 ? 0x00FF00FFu : d == 2 ? 0x0F0F0F0Fu : 0x33333333u;
#pragma unroll
    for (int p = 0; p < 16; ++p)
      if (!(p & d)) {
        const uint32_t t = ((w[p] >> (2 * d)) ^ w[p + d]) & mask;
        w[p + d] ^= t;
        w[p] ^= t << (2 * d);
      }
  }
}

}  // namespace sg
