// Bit-stream reads of the packed masks and the list rule of GEMM-Q, for the kernels that build work lists and for the GEMM
// kernel that finds its first tile without one.
#pragma once

#include <cstdint>

namespace fo {
namespace {

// 32 bits of the little-endian bit stream `seg` starting at bit `pos`; bytes at or beyond `limit`
// (the number of readable bytes from `seg`) read as zero.
__device__ __forceinline__ uint32_t load_bits32(const uint8_t* seg, int64_t pos, int64_t limit) {
  const int64_t byte0 = pos >> 3;
  const int sh = static_cast<int>(pos & 7);
  uint64_t acc = 0;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int64_t bi = byte0 + i;
    const uint64_t v = (bi < limit) ? seg[bi] : 0u;
    acc |= v << (8 * i);
  }
  return static_cast<uint32_t>(acc >> sh);
}
__device__ __forceinline__ int get_bit(const uint8_t* seg, int64_t pos, int64_t limit) {
  const int64_t bi = pos >> 3;
  if (bi >= limit) return 0;
  return (seg[bi] >> (pos & 7)) & 1;
}

// up to 64 bits of the stream starting at bit `pos` (9 independent byte loads, clamped like load_bits32)
__device__ __forceinline__ uint64_t load_bits64(const uint8_t* seg, int64_t pos, int64_t limit, int nbits) {
  const int64_t byte0 = pos >> 3;
  const int sh = static_cast<int>(pos & 7);
  uint64_t lo = 0, hi = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t bi = byte0 + i;
    const uint64_t v = (bi < limit) ? seg[bi] : 0u;
    lo |= v << (8 * i);
  }
  if (byte0 + 8 < limit) hi = seg[byte0 + 8];
  uint64_t r = sh ? ((lo >> sh) | (hi << (64 - sh))) : lo;
  if (nbits < 64) r &= (1ull << nbits) - 1ull;
  return r;
}

constexpr int kPairCost = 20, kSingleCost = 13;

// Time at which the last CTA ends when `n` CTAs draw `pairs` two-block tiles and then `singles` single-block tiles
// in list order, every tile going to the CTA that is free first.
__device__ __forceinline__ int gemm_q_makespan(int pairs, int singles, int n) {
  const int full = pairs / n, r = pairs % n;
  int t_a = full * kPairCost, c_a = n - r;        // CTAs free after the full rounds
  int t_b = (full + 1) * kPairCost, c_b = r;      // CTAs that run one more two-block tile
  int end = (full + (r ? 1 : 0)) * kPairCost;
  int m = singles;
  while (m > 0) {
    if (c_a > 0 && (c_b == 0 || t_a <= t_b)) {
      m -= c_a;
      t_a += kSingleCost;
      end = end > t_a ? end : t_a;
    } else {
      m -= c_b;
      t_b += kSingleCost;
      end = end > t_b ? end : t_b;
    }
  }
  return end;
}

}  // namespace
}  // namespace fo
