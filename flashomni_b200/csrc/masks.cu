// Mask path: bit packing (packbits / segment_packbits) and the compaction of the packed
// block masks into the work lists the attention and GEMM kernels consume.
//
// Bit layout (same as include/flashomni/attention/prefill.cuh:1284-1294,1385-1394 and
// include/flashomni/gemm/w16a16/gemm.cuh:50-58 of the reference): per request b the segment starts
// at byte `indptr[b]`; q-block bit index = qb*H + h; kv-block bit index = (qb*H + h)*nkv + kvb;
// bit i of a segment = (seg[i >> 3] >> (i & 7)) & 1.
//
// All kernels here are integer / byte work bound by HBM and launch latency; they never touch
// memory outside the extents given (reads are clamped to the packed buffers' byte sizes) and
// report malformed input through a status word instead of faulting.
#include "cast_fp8.cuh"
#include "internal.h"
#include "mask_bits.cuh"

namespace fo {

// ---------------------------------------------------------------------------------------------
// packbits
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack8(const uint8_t* p, int64_t avail, bool little, bool aligned8) {
  // Packs up to 8 input bytes (non-zero -> 1). `avail` = number of valid inputs (1..8).
  uint32_t out = 0;
  if (aligned8 && avail >= 8) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const uint32_t w[2] = {v.x, v.y};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t byte = (w[i >> 2] >> ((i & 3) * 8)) & 0xFFu;
      const uint32_t bit = byte != 0u;
      out |= bit << (little ? i : 7 - i);
    }
  } else {
    const int n = avail < 8 ? static_cast<int>(avail) : 8;
    for (int i = 0; i < n; ++i) {
      const uint32_t bit = p[i] != 0;
      out |= bit << (little ? i : 7 - i);
    }
  }
  return out;
}

// Four output bytes from 32 input bytes held in two 16-byte words: per 32-bit word the "byte is non-zero" flags are
// gathered with one multiply (flag of byte i at bit 8 i; the product with 2^24 + 2^17 + 2^10 + 2^3 puts flag i at bit
// 24 + i, all partial products land on distinct bits).
__device__ __forceinline__ uint32_t nibble_of(uint32_t w) {
  const uint32_t t = ((((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u) >> 7;
  return (t * 0x01020408u) >> 24;
}
__device__ __forceinline__ uint32_t pack32(const uint4& a, const uint4& b, bool little) {
  uint32_t r = (nibble_of(a.x) | (nibble_of(a.y) << 4)) | ((nibble_of(a.z) | (nibble_of(a.w) << 4)) << 8) |
               ((nibble_of(b.x) | (nibble_of(b.y) << 4)) << 16) | ((nibble_of(b.z) | (nibble_of(b.w) << 4)) << 24);
  if (!little) r = __byte_perm(__brev(r), 0, 0x0123);  // reverse the bits inside every byte, keep the byte order
  return r;
}

// One thread per four output bytes (32 inputs, two 16-byte loads in flight) where alignment and length allow it,
// byte by byte otherwise.
__global__ void packbits_kernel(const uint8_t* __restrict__ x, int64_t n, int little, uint8_t* __restrict__ y) {
  const int64_t nbytes = (n + 7) >> 3;
  const int64_t nwords = (nbytes + 3) >> 2;
  const bool x16 = (reinterpret_cast<uintptr_t>(x) & 15u) == 0, y4 = (reinterpret_cast<uintptr_t>(y) & 3u) == 0;
  const bool x8 = (reinterpret_cast<uintptr_t>(x) & 7u) == 0;
  for (int64_t w = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; w < nwords;
       w += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i0 = w * 4;
    if (x16 && y4 && (i0 + 4) * 8 <= n) {
      const uint4 a = *reinterpret_cast<const uint4*>(x + i0 * 8), b = *reinterpret_cast<const uint4*>(x + i0 * 8 + 16);
      *reinterpret_cast<uint32_t*>(y + i0) = pack32(a, b, little != 0);
    } else {
      for (int64_t i = i0; i < i0 + 4 && i < nbytes; ++i)
        y[i] = static_cast<uint8_t>(pack8(x + i * 8, n - i * 8, little != 0, x8));
    }
  }
}

// The same per segment; the segment of an output byte is found by binary search over the byte indptr.
__device__ __forceinline__ int seg_of(const int32_t* __restrict__ new_indptr, int num_segments, int64_t i) {
  int lo = 0, hi = num_segments;  // new_indptr[lo] <= i < new_indptr[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (static_cast<int64_t>(new_indptr[mid]) <= i) lo = mid; else hi = mid;
  }
  return lo;
}
__global__ void segment_packbits_kernel(const uint8_t* __restrict__ x, const int32_t* __restrict__ indptr,
                                        const int32_t* __restrict__ new_indptr, int num_segments,
                                        int64_t out_bytes, int little, uint8_t* __restrict__ y) {
  const int64_t nwords = (out_bytes + 3) >> 2;
  const bool y4 = (reinterpret_cast<uintptr_t>(y) & 3u) == 0;
  for (int64_t w = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; w < nwords;
       w += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i0 = w * 4;
    const int lo = seg_of(new_indptr, num_segments, i0);
    const int64_t seg_in0 = indptr[lo], seg_in1 = indptr[lo + 1];
    const int64_t src0 = seg_in0 + (i0 - new_indptr[lo]) * 8;
    // fast path: the four bytes lie in one segment, all 32 inputs exist, loads and the store are aligned
    if (y4 && i0 + 4 <= out_bytes && i0 + 4 <= static_cast<int64_t>(new_indptr[lo + 1]) && src0 + 32 <= seg_in1 &&
        (reinterpret_cast<uintptr_t>(x + src0) & 15u) == 0) {
      const uint4 a = *reinterpret_cast<const uint4*>(x + src0), b = *reinterpret_cast<const uint4*>(x + src0 + 16);
      *reinterpret_cast<uint32_t*>(y + i0) = pack32(a, b, little != 0);
      continue;
    }
    for (int64_t i = i0; i < i0 + 4 && i < out_bytes; ++i) {
      const int sg = seg_of(new_indptr, num_segments, i);
      const int64_t src = static_cast<int64_t>(indptr[sg]) + (i - new_indptr[sg]) * 8;
      const int64_t avail = static_cast<int64_t>(indptr[sg + 1]) - src;
      if (avail <= 0) { y[i] = 0; continue; }
      const bool aligned = (reinterpret_cast<uintptr_t>(x + src) & 7u) == 0;
      y[i] = static_cast<uint8_t>(pack8(x + src, avail, little != 0, aligned));
    }
  }
}

cudaError_t launch_packbits(const uint8_t* x, int64_t n, int little, uint8_t* y, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int64_t nwords = (((n + 7) >> 3) + 3) >> 2;
  const int threads = 256;
  int64_t blocks = (nwords + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  packbits_kernel<<<static_cast<int>(blocks), threads, 0, stream>>>(x, n, little, y);
  return cudaGetLastError();
}

cudaError_t launch_segment_packbits(const uint8_t* x, const int32_t* indptr, const int32_t* new_indptr,
                                    int num_segments, int64_t out_bytes, int little, uint8_t* y,
                                    cudaStream_t stream) {
  if (out_bytes <= 0 || num_segments <= 0) return cudaSuccess;
  const int64_t nwords = (out_bytes + 3) >> 2;
  const int threads = 256;
  int64_t blocks = (nwords + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  segment_packbits_kernel<<<static_cast<int>(blocks), threads, 0, stream>>>(x, indptr, new_indptr, num_segments,
                                                                            out_bytes, little, y);
  return cudaGetLastError();
}

// The same without a byte indptr in hand: every CTA derives it from the element indptr (a few segments: one scan in shared
// memory) and packs its share; CTA 0 also writes the byte indptr and, to host memory that the device can write, the
// total (-1: an indptr that decreases or leaves the n values of x, nothing is packed). What bounds the step is the
// caller's wait. With at most one CTA per SM each reports to a word of its own when its bytes are written, and the caller polls
// these words instead of waiting for the stream: two calls for the masks of 2 x 36 q-blocks x 24 heads 33.3 -> 31.2 us on a
// B200, of 604 q-blocks x 40 heads 38.2 -> 36.0 (ten launches and a copy in place of this kernel: 191.5 us). Returning when
// CTA 0 knows the total would take 24.8, but the caller's other streams would then read bytes that are still being written.
constexpr int kPackSegs = 1024;
template <typename Idx>
__global__ void __launch_bounds__(256) segment_packbits_sized_kernel(const uint8_t* __restrict__ x, int64_t n,
                                                                     const Idx* __restrict__ indptr, int num_segments, int64_t capacity, int little,
                                                                     uint8_t* __restrict__ y, int32_t* __restrict__ new_indptr,
                                                                     long long* __restrict__ words, int every_block) {
  __shared__ int64_t s_in[kPackSegs + 1];
  __shared__ int32_t s_new[kPackSegs + 1];
  __shared__ int s_bad;
  const int tid = threadIdx.x;
  if (tid == 0) s_bad = 0;
  for (int i = tid; i <= num_segments; i += 256) s_in[i] = static_cast<int64_t>(indptr[i]);
  __syncthreads();
  if (tid < 32) {
    int64_t carry = 0;
    bool bad = false;
    for (int base = 0; base < num_segments; base += 32) {
      const int i = base + tid;
      const int64_t len = i < num_segments ? s_in[i + 1] - s_in[i] : 0;
      bad = bad || len < 0;
      int64_t v = (len + 7) >> 3;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t up = __shfl_up_sync(0xffffffffu, v, o);
        if (tid >= o) v += up;
      }
      if (i < num_segments) s_new[i + 1] = static_cast<int32_t>(carry + v);
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    bad = __any_sync(0xffffffffu, bad) || carry > 0x7fffffffLL || carry > capacity || s_in[0] < 0 || s_in[num_segments] > n;
    if (tid == 0) {
      s_new[0] = 0;
      s_bad = bad ? 1 : 0;
    }
  }
  __syncthreads();
  const int64_t out_bytes = s_bad ? 0 : s_new[num_segments];
  if (blockIdx.x == 0 && !s_bad)
    for (int i = tid; i <= num_segments; i += 256) new_indptr[i] = s_new[i];
  const int64_t nwords = (out_bytes + 3) >> 2;
  const bool y4 = (reinterpret_cast<uintptr_t>(y) & 3u) == 0;
  for (int64_t w = blockIdx.x * 256ll + tid; w < nwords; w += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t i0 = w * 4;
    const int lo = seg_of(s_new, num_segments, i0);
    const int64_t src0 = s_in[lo] + (i0 - s_new[lo]) * 8;
    if (y4 && i0 + 4 <= s_new[lo + 1] && src0 + 32 <= s_in[lo + 1] && (reinterpret_cast<uintptr_t>(x + src0) & 15u) == 0) {
      const uint4 a = *reinterpret_cast<const uint4*>(x + src0), b = *reinterpret_cast<const uint4*>(x + src0 + 16);
      *reinterpret_cast<uint32_t*>(y + i0) = pack32(a, b, little != 0);
      continue;
    }
    for (int64_t i = i0; i < i0 + 4 && i < out_bytes; ++i) {
      const int sg = seg_of(s_new, num_segments, i);
      const int64_t src = s_in[sg] + (i - s_new[sg]) * 8;
      const int64_t avail = s_in[sg + 1] - src;
      const bool aligned = (reinterpret_cast<uintptr_t>(x + src) & 7u) == 0;
      y[i] = static_cast<uint8_t>(pack8(x + src, avail, little != 0, aligned));
    }
  }
  __syncthreads();
  if (tid == 0 && (every_block || blockIdx.x == 0)) {  // the host may be polling: what this block has written comes first
    __threadfence_system();
    static_cast<volatile long long*>(words)[blockIdx.x] = s_bad ? -1ll : static_cast<long long>(out_bytes);
  }
}

int segment_packbits_sized_blocks(int64_t capacity) {
  const int64_t blocks = ((capacity >> 2) + 255) / 256;
  return blocks > 148 * 8 ? 148 * 8 : (blocks < 1 ? 1 : static_cast<int>(blocks));
}

cudaError_t launch_segment_packbits_sized(const uint8_t* x, int64_t n, const void* indptr, int indptr_is_64, int num_segments,
                                          int64_t capacity, int little, uint8_t* y, int32_t* new_indptr, long long* words,
                                          int every_block, cudaStream_t stream) {
  if (num_segments > kPackSegs) return cudaErrorInvalidValue;
  const int blocks = segment_packbits_sized_blocks(capacity);
  if (indptr_is_64)
    segment_packbits_sized_kernel<int64_t><<<blocks, 256, 0, stream>>>(x, n, static_cast<const int64_t*>(indptr), num_segments, capacity, little,
                                                                      y, new_indptr, words, every_block);
  else
    segment_packbits_sized_kernel<int32_t><<<blocks, 256, 0, stream>>>(x, n, static_cast<const int32_t*>(indptr), num_segments, capacity, little,
                                                                      y, new_indptr, words, every_block);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Attention mask compaction
// ---------------------------------------------------------------------------------------------
// Candidate c enumerates (b, qb, hl) in ascending (b, qb, hl) order, hl in [0, head_count).
struct Cand {
  int b, qb, h;       // h = head_begin + hl (index used for mask bits)
  int nq, nkv;
  bool valid;
};

constexpr int kMaxBatchSmem = 1024;
constexpr int64_t kCompactL2Bytes = 48ll << 20;   // K + V bytes of the heads of one group (a share of the 126 MB L2)
constexpr int64_t kCompactFineBuckets = 8192;  // groups * (max_nkv + 1) up to which items are ordered by length inside a group

// Fills smem prefix of candidates per request. Thread 0 computes (B is small), all read after sync.
__device__ __forceinline__ void build_cand_prefix(const CompactArgs& a, int64_t* s_prefix) {
  if (threadIdx.x == 0) {
    int64_t acc = 0;
    s_prefix[0] = 0;
    for (int b = 0; b < a.batch; ++b) {
      const int64_t ql = static_cast<int64_t>(a.qo_indptr[b + 1]) - a.qo_indptr[b];
      const int64_t nq = ql > 0 ? (ql + a.sbq - 1) / a.sbq : 0;
      acc += nq * a.head_count;
      s_prefix[b + 1] = acc;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ Cand decode_cand(const CompactArgs& a, const int64_t* s_prefix, int64_t c) {
  Cand r;
  int lo = 0, hi = a.batch;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_prefix[mid] <= c) lo = mid; else hi = mid;
  }
  r.b = lo;
  const int64_t local = c - s_prefix[lo];
  r.qb = static_cast<int>(local / a.head_count);
  r.h = a.head_begin + static_cast<int>(local % a.head_count);
  const int64_t ql = static_cast<int64_t>(a.qo_indptr[lo + 1]) - a.qo_indptr[lo];
  const int64_t kl = static_cast<int64_t>(a.kv_indptr[lo + 1]) - a.kv_indptr[lo];
  r.nq = static_cast<int>((ql + a.sbq - 1) / a.sbq);
  r.nkv = kl > 0 ? static_cast<int>((kl + a.sbkv - 1) / a.sbkv) : 0;
  r.valid = c < s_prefix[a.batch];
  return r;
}

// Pass 1: one warp per candidate. cnt[c] = number of kept kv-blocks if the q-block is active, else -1.
__global__ void compact_count_kernel(CompactArgs a) {
  __shared__ int64_t s_prefix[kMaxBatchSmem + 1];
  build_cand_prefix(a, s_prefix);
  const int lane = threadIdx.x & 31;
  const int64_t warps_per_grid = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t c = blockIdx.x * static_cast<int64_t>(blockDim.x >> 5) + (threadIdx.x >> 5); c < a.n_cand;
       c += warps_per_grid) {
    const Cand cd = decode_cand(a, s_prefix, c);
    int result;
    if (a.is_full) {
      result = cd.nkv;
    } else {
      const int64_t ioff = a.info_indptr[cd.b];
      const int64_t koff = a.kv_info_indptr[cd.b];
      const int64_t qbit = static_cast<int64_t>(cd.qb) * a.num_heads + cd.h;
      const int active = get_bit(a.sparse_info + ioff, qbit, a.info_bytes - ioff);
      if (!active) {
        result = -1;
      } else {
        const int64_t row0 = qbit * cd.nkv;
        int cnt = 0;
        for (int w = lane * 32; w < cd.nkv; w += 32 * 32) {
          uint32_t bits = load_bits32(a.sparse_kv_info + koff, row0 + w, a.kv_info_bytes - koff);
          const int rem = cd.nkv - w;
          if (rem < 32) bits &= (1u << rem) - 1u;
          cnt += __popc(bits);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        result = cnt;
      }
    }
    if (lane == 0) a.cnt[c] = result;
  }
}

// Pass 2: single CTA. Exclusive scans of the active flags (item index) and of the kept counts
// (offset into kv_idx), then the processing order: items grouped by (request, head), q-blocks ascending
// inside a group, by a stable counting sort: W warps own contiguous candidate slices, each with its own
// histogram in shared memory; bucket starts are (items of smaller keys) + (same bucket, earlier
// slices); every warp then places its slice in ascending candidate order, 32 at a time.
__global__ void __launch_bounds__(1024) compact_scan_kernel(CompactArgs a, int sort_warps, int by_length, int heads_per_group) {
  extern __shared__ __align__(16) int s_whist[];  // [sort_warps + 1][batch * head_count]; first the scan's staging
  __shared__ int s_warp_items[32];
  __shared__ long long s_warp_kept[32];
  __shared__ int s_carry_items;
  __shared__ long long s_carry_kept;
  __shared__ int64_t s_prefix[kMaxBatchSmem + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) { s_carry_items = 0; s_carry_kept = 0; }
  __syncthreads();
  // kScanPer consecutive candidates per thread and pass: a thread scans its own run, the CTA scans the run totals
  constexpr int kScanPer = 8;
  constexpr int kPassCand = 1024 * kScanPer, kPassPad = kPassCand + kPassCand / 32;
  // staging of a pass, over the dynamic shared memory that the sort below uses afterwards
  long long* s_off = reinterpret_cast<long long*>(s_whist);           // [kPassPad] kept-list offsets
  int* s_val = reinterpret_cast<int*>(s_off + kPassPad);              // [kPassPad] candidate counts
  int* s_pos = s_val + kPassPad;                                      // [kPassPad] item positions
  for (int64_t base = 0; base < a.n_cand; base += static_cast<int64_t>(blockDim.x) * kScanPer) {
    const int64_t c0 = base + static_cast<int64_t>(tid) * kScanPer;
    // The counts of a pass come in with coalesced loads and the results leave with coalesced stores; between them
    // they sit in shared memory, where a thread finds its eight consecutive entries (index i at i + i / 32: the
    // accesses of a warp then fall on 32 different banks).
    const int64_t pass_n = (a.n_cand - base) < kPassCand ? (a.n_cand - base) : kPassCand;
    for (int i = tid; i < pass_n; i += blockDim.x) s_val[i + (i >> 5)] = a.cnt[base + i];
    __syncthreads();
    int vals[kScanPer];
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      const int i = tid * kScanPer + k;
      vals[k] = (c0 + k < a.n_cand) ? s_val[i + (i >> 5)] : -1;
    }
    int run_i = 0;
    long long run_k = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      run_i += vals[k] >= 0;
      run_k += vals[k] >= 0 ? vals[k] : 0;
    }
    int xi = run_i;
    long long xk = run_k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yi = __shfl_up_sync(0xffffffffu, xi, o);
      const long long yk = __shfl_up_sync(0xffffffffu, xk, o);
      if (lane >= o) { xi += yi; xk += yk; }
    }
    if (lane == 31) { s_warp_items[warp] = xi; s_warp_kept[warp] = xk; }
    __syncthreads();
    if (warp == 0) {
      int wi = s_warp_items[lane];
      long long wk = s_warp_kept[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int yi = __shfl_up_sync(0xffffffffu, wi, o);
        const long long yk = __shfl_up_sync(0xffffffffu, wk, o);
        if (lane >= o) { wi += yi; wk += yk; }
      }
      s_warp_items[lane] = wi;  // inclusive over warps
      s_warp_kept[lane] = wk;
    }
    __syncthreads();
    int pre_i = s_carry_items + (warp ? s_warp_items[warp - 1] : 0) + xi - run_i;
    long long pre_k = s_carry_kept + (warp ? s_warp_kept[warp - 1] : 0) + xk - run_k;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      if (c0 + k < a.n_cand) {
        const bool flag = vals[k] >= 0;
        const int i = tid * kScanPer + k;
        s_pos[i + (i >> 5)] = flag ? pre_i : -1;
        s_off[i + (i >> 5)] = pre_k;
        pre_i += flag;
        pre_k += flag ? vals[k] : 0;
      }
    }
    __syncthreads();
    for (int i = tid; i < pass_n; i += blockDim.x) {
      a.item_pos[base + i] = s_pos[i + (i >> 5)];
      a.kv_off[base + i] = s_off[i + (i >> 5)];
    }
    if (tid == 0) {
      s_carry_items += s_warp_items[31];
      s_carry_kept += s_warp_kept[31];
    }
    __syncthreads();
  }
  const int n_items = s_carry_items;
  const long long total_kept = s_carry_kept;
  if (tid == 0) {
    a.counters[0] = n_items;
    a.counters[1] = static_cast<int>(total_kept > 0x7fffffffLL ? 0x7fffffff : total_kept);
    a.counters[2] = (total_kept > a.max_kept || n_items > a.max_items) ? kDevBadIndex : kDevOk;
    a.counters[3] = a.max_nkv;
    a.kv_ptr[n_items <= a.max_items ? n_items : 0] = static_cast<int>(total_kept);
  }
  // ---- processing order: stable counting sort by (request, group of heads), so that the CTAs that run at the
  // same time work on the same few heads and share their K / V tiles in L2. A group is `heads_per_group`
  // consecutive heads: as many as keep their K and V in L2 together (launch_attn_compact).
  // With `by_length` the items of a group are ordered by descending list length (ties: canonical order):
  // the items drawn last are then the short ones of the group and the launch ends without a long straggler.
  const int per_group = by_length ? a.max_nkv + 1 : 1;
  const int grp_per_req = (a.head_count + heads_per_group - 1) / heads_per_group;
  const int nb = a.batch * grp_per_req * per_group;
  if (!by_length) {
    // Single heads with their q-blocks ascending: the candidates read in (request, head, q-block) order instead of
    // (request, q-block, head); the running count of active ones is the position. One more scan, no sort.
    build_cand_prefix(a, s_prefix);
    if (a.head_count <= 512) {
      // Threads laid out head-fastest: thread (chunk k, head h) walks the q-blocks of its chunk for its head, so the
      // threads of a chunk read consecutive positions (one row of heads at a time). Count, prefix per head over the
      // chunks and over the heads, then the same walk again writing the positions out.
      int* s_cnt = reinterpret_cast<int*>(s_whist);          // [chunks][H] counts, then exclusive starts
      const int H = a.head_count;
      const int chunks = static_cast<int>(blockDim.x) / H;
      int* s_tot = s_cnt + chunks * H;                       // [H] items of a head, then the head's start
      const int h = tid % H, ck = tid / H;
      int req_base = 0;
      for (int b = 0; b < a.batch; ++b) {
        const int64_t c_req = s_prefix[b];
        const int nq = static_cast<int>((s_prefix[b + 1] - s_prefix[b]) / H);
        const int qpc = (nq + chunks - 1) / chunks;
        const int q0 = ck * qpc, q1 = (q0 + qpc < nq) ? q0 + qpc : nq;
        int mine = 0;
        if (ck < chunks)
          for (int qb = q0; qb < q1; ++qb) mine += a.item_pos[c_req + static_cast<int64_t>(qb) * H + h] >= 0;
        if (ck < chunks) s_cnt[ck * H + h] = mine;
        __syncthreads();
        if (tid < H) {   // exclusive prefix over the chunks of head `tid`
          int run = 0;
          for (int k = 0; k < chunks; ++k) {
            const int t = s_cnt[k * H + tid];
            s_cnt[k * H + tid] = run;
            run += t;
          }
          s_tot[tid] = run;
        }
        __syncthreads();
        if (warp == 0) {  // exclusive prefix over the heads
          int carry = 0;
          for (int h0 = 0; h0 < H; h0 += 32) {
            const int v = (h0 + lane < H) ? s_tot[h0 + lane] : 0;
            int x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int y = __shfl_up_sync(0xffffffffu, x, o);
              if (lane >= o) x += y;
            }
            if (h0 + lane < H) s_tot[h0 + lane] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
          }
          if (lane == 0) s_carry_items = carry;   // items of this request
        }
        __syncthreads();
        if (ck < chunks) {
          int pos = req_base + s_tot[h] + s_cnt[ck * H + h];
          for (int qb = q0; qb < q1; ++qb) {
            const int ip = a.item_pos[c_req + static_cast<int64_t>(qb) * H + h];
            if (ip >= 0) {
              if (pos < a.max_items) a.order[pos] = ip;
              ++pos;
            }
          }
        }
        req_base += s_carry_items;
        __syncthreads();
      }
      return;
    }
    if (tid == 0) s_carry_items = 0;
    __syncthreads();
    for (int64_t base = 0; base < a.n_cand; base += static_cast<int64_t>(blockDim.x) * kScanPer) {
      const int64_t j0 = base + static_cast<int64_t>(tid) * kScanPer;
      int ip[kScanPer];
#pragma unroll
      for (int k = 0; k < kScanPer; ++k) {
        const int64_t j = j0 + k;
        ip[k] = -1;
        if (j < a.n_cand) {
          int lo = 0, hi = a.batch;
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_prefix[mid] <= j) lo = mid; else hi = mid;
          }
          const int64_t local = j - s_prefix[lo];
          const int64_t nq = (s_prefix[lo + 1] - s_prefix[lo]) / a.head_count;
          const int64_t h = local / nq, qb = local % nq;
          ip[k] = a.item_pos[s_prefix[lo] + qb * a.head_count + h];
        }
      }
      int run = 0;
#pragma unroll
      for (int k = 0; k < kScanPer; ++k) run += ip[k] >= 0;
      int x = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_warp_items[warp] = x;
      __syncthreads();
      if (warp == 0) {
        int w = s_warp_items[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, w, o);
          if (lane >= o) w += y;
        }
        s_warp_items[lane] = w;
      }
      __syncthreads();
      int pos = s_carry_items + (warp ? s_warp_items[warp - 1] : 0) + x - run;
#pragma unroll
      for (int k = 0; k < kScanPer; ++k) {
        if (ip[k] >= 0) {
          if (pos < a.max_items) a.order[pos] = ip[k];
          ++pos;
        }
      }
      __syncthreads();
      if (tid == 0) s_carry_items += s_warp_items[31];
      __syncthreads();
    }
    return;
  }
  if (sort_warps <= 0) {  // too many (request, group, length) buckets for the shared-memory histograms: canonical order
    for (int i = tid; i < n_items && i < a.max_items; i += blockDim.x) a.order[i] = i;
    return;
  }
  int* s_total = s_whist + sort_warps * nb;  // [nb] bucket totals, then bucket starts
  for (int i = tid; i < (sort_warps + 1) * nb; i += blockDim.x) s_whist[i] = 0;
  build_cand_prefix(a, s_prefix);
  auto key_of = [&](int64_t c, int len) -> int {   // len = cnt[c], already fetched by the caller
    int lo = 0, hi = a.batch;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_prefix[mid] <= c) lo = mid; else hi = mid;
    }
    const int grp = lo * grp_per_req + static_cast<int>((c - s_prefix[lo]) % a.head_count) / heads_per_group;
    if (!by_length) return grp;
    len = len < 0 ? 0 : (len > a.max_nkv ? a.max_nkv : len);
    return grp * per_group + (a.max_nkv - len);
  };
  const int64_t slice = ((a.n_cand + sort_warps - 1) / sort_warps + 31) / 32 * 32;
  const int64_t my0 = static_cast<int64_t>(warp) * slice;
  const int64_t my1 = (my0 + slice < a.n_cand) ? my0 + slice : a.n_cand;
  constexpr int kAhead = 4;  // candidate counts fetched ahead: the loads of four steps are in flight together
  if (warp < sort_warps) {
    int* h = s_whist + warp * nb;
    for (int64_t c0 = my0 + lane; c0 < my1; c0 += 32 * kAhead) {
      int v[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) v[k] = (c0 + 32 * k < my1) ? a.cnt[c0 + 32 * k] : -1;
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
        if (v[k] >= 0) atomicAdd(&h[key_of(c0 + 32 * k, v[k])], 1);
    }
  }
  __syncthreads();
  // per bucket: exclusive prefix over the slices; the bucket total goes to s_total
  for (int k = tid; k < nb; k += blockDim.x) {
    int run = 0;
    for (int w = 0; w < sort_warps; ++w) {
      const int t = s_whist[w * nb + k];
      s_whist[w * nb + k] = run;
      run += t;
    }
    s_total[k] = run;
  }
  __syncthreads();
  // bucket starts in ascending key order (exclusive scan by warp 0)
  if (warp == 0) {
    int carry = 0;
    for (int k0 = 0; k0 < nb; k0 += 32) {
      const int k = k0 + lane;
      const int v = (k < nb) ? s_total[k] : 0;
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (k < nb) s_total[k] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  __syncthreads();
  for (int i = tid; i < sort_warps * nb; i += blockDim.x) s_whist[i] += s_total[i % nb];
  __syncthreads();
  if (warp < sort_warps) {
    int* h = s_whist + warp * nb;
    for (int64_t base0 = my0; base0 < my1; base0 += 32 * kAhead) {
      int cv[kAhead], ip[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int64_t c = base0 + 32 * k + lane;
        cv[k] = (c < my1) ? a.cnt[c] : -1;
        ip[k] = (c < my1) ? a.item_pos[c] : -1;
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
      const int64_t base = base0 + 32 * k;
      if (base >= my1) break;
      const int64_t c = base + lane;
      const bool flag = (c < my1) && cv[k] >= 0;
      const int v = flag ? key_of(c, cv[k]) : -1 - lane;
      const unsigned grp = __match_any_sync(0xffffffffu, v);
      const int rank_in_grp = __popc(grp & ((1u << lane) - 1u));
      const int leader = __ffs(grp) - 1;
      int start = 0;
      if (flag && lane == leader) {
        start = h[v];
        h[v] = start + __popc(grp);
      }
      start = __shfl_sync(0xffffffffu, start, leader);
      if (flag) {
        const int pos = start + rank_in_grp;
        if (pos < a.max_items) a.order[pos] = ip[k];
      }
      __syncwarp();
      }
    }
  }
}

// Pass 3: one warp per candidate; writes the item record and expands its kept kv-blocks (ascending).
__global__ void compact_fill_kernel(CompactArgs a) {
  __shared__ int64_t s_prefix[kMaxBatchSmem + 1];
  build_cand_prefix(a, s_prefix);
  const int lane = threadIdx.x & 31;
  const int64_t warps_per_grid = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t c = blockIdx.x * static_cast<int64_t>(blockDim.x >> 5) + (threadIdx.x >> 5); c < a.n_cand;
       c += warps_per_grid) {
    const int pos = a.item_pos[c];
    if (pos < 0 || pos >= a.max_items) continue;
    const Cand cd = decode_cand(a, s_prefix, c);
    const long long off = a.kv_off[c];
    const int kept = a.cnt[c];
    if (off + kept > a.max_kept) continue;  // flagged by the scan pass
    if (lane == 0) {
      a.items[4 * pos + 0] = cd.b;
      a.items[4 * pos + 1] = cd.h;
      a.items[4 * pos + 2] = cd.qb;
      a.items[4 * pos + 3] = kept;
      a.kv_ptr[pos] = static_cast<int>(off);
    }
    int written = 0;
    if (a.is_full) {
      for (int j = lane; j < cd.nkv; j += 32) a.kv_idx[off + j] = j;
    } else {
      const int64_t koff = a.kv_info_indptr[cd.b];
      const int64_t row0 = (static_cast<int64_t>(cd.qb) * a.num_heads + cd.h) * cd.nkv;
      for (int w0 = 0; w0 < cd.nkv; w0 += 32 * 32) {
        const int w = w0 + lane * 32;
        uint32_t bits = 0;
        if (w < cd.nkv) {
          bits = load_bits32(a.sparse_kv_info + koff, row0 + w, a.kv_info_bytes - koff);
          const int rem = cd.nkv - w;
          if (rem < 32) bits &= (1u << rem) - 1u;
        }
        const int pc = __popc(bits);
        int x = pc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        int dst = written + x - pc;
        while (bits) {
          const int bpos = __ffs(bits) - 1;
          bits &= bits - 1;
          a.kv_idx[off + dst++] = w + bpos;
        }
        written += __shfl_sync(0xffffffffu, x, 31);
      }
    }
  }
}

// Groups of heads: as many consecutive heads as keep their K and V tiles in L2 together (kCompactL2Bytes for
// 128-row x 128-column 16-bit blocks, max_nkv of them per head and tensor), evenly sized. Inside a group the
// items are ordered by descending list length while the histograms (groups x lengths) stay below
// kCompactFineBuckets; otherwise the groups are single heads with their q-blocks ascending.
static void order_rule(const CompactArgs& a, int* by_length, int* heads_per_group) {
  int64_t hpg = kCompactL2Bytes / (static_cast<int64_t>(a.max_nkv > 0 ? a.max_nkv : 1) * 65536);
  hpg = hpg < 1 ? 1 : (hpg > a.head_count ? a.head_count : hpg);
  const int64_t grp_per_req = (a.head_count + hpg - 1) / hpg;
  hpg = (a.head_count + grp_per_req - 1) / grp_per_req;
  *by_length = static_cast<int64_t>(a.batch) * grp_per_req * (a.max_nkv + 1) <= kCompactFineBuckets ? 1 : 0;
  *heads_per_group = *by_length ? static_cast<int>(hpg) : 1;
}

cudaError_t launch_attn_compact(const CompactArgs& a, cudaStream_t stream) {
  if (a.batch > kMaxBatchSmem) return cudaErrorInvalidValue;
  if (a.n_cand <= 0) {
    return cudaMemsetAsync(a.counters, 0, 4 * sizeof(int), stream);
  }
  const int threads = 256, wpb = threads / 32;
  int64_t blocks = (a.n_cand + wpb - 1) / wpb;
  if (blocks > 148 * 8) blocks = 148 * 8;
  // Sort histograms: as many warps as fit in ~160 KB of shared memory, plus one row of bucket totals; with more
  // groups than fit, the kernel leaves the items in canonical order.
  int by_length, hpg;
  order_rule(a, &by_length, &hpg);
  const int64_t groups = static_cast<int64_t>(a.batch) * ((a.head_count + hpg - 1) / hpg);
  const int64_t nb = by_length ? groups * (a.max_nkv + 1) : groups;
  int64_t sort_warps = nb > 0 ? (160 * 1024) / (nb * 4) - 1 : 0;
  if (sort_warps > 32) sort_warps = 32;
  if (sort_warps < 1) sort_warps = 0;
  size_t scan_smem = static_cast<size_t>((sort_warps + 1) * nb * 4) * (sort_warps > 0 ? 1 : 0);
  const size_t stage_smem = static_cast<size_t>(8192 + 8192 / 32) * 16;   // the scan's staging: 8 + 4 + 4 bytes per candidate
  if (scan_smem < stage_smem) scan_smem = stage_smem;
  {
    cudaError_t ea = cudaFuncSetAttribute(compact_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 164 * 1024);
    if (ea != cudaSuccess) return ea;
  }
  compact_count_kernel<<<static_cast<int>(blocks), threads, 0, stream>>>(a);
  compact_scan_kernel<<<1, 1024, scan_smem, stream>>>(a, static_cast<int>(sort_warps), by_length, hpg);
  compact_fill_kernel<<<static_cast<int>(blocks), threads, 0, stream>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Attention work units (self-contained records; split of long kv lists)
// ---------------------------------------------------------------------------------------------
// Walks the items in processing order and writes one 32-byte record per unit of work, holding everything the
// attention kernel's roles need (no chain of dependent loads at a unit boundary):
//   [0] n          kv blocks of the unit (0: an active q-block that keeps nothing)
//   [1] kv_off     offset of the unit's first entry in kv_idx
//   [2] h | b << 16   mask head (< 65536), request (< 32768)
//   [3] q_row0     first row of the q-block in the q / o tensors
//   [4] q_valid | ragged << 16   rows (tokens) of the q-block that exist (1..sbq); columns of the request's partial
//                  last kv block if the unit's list ends with it, else 0
//   [5] kv_row0    first kv row of the request
//   [6] causal     qb * sbq + kv_len - q_len: the last kv position that the q-block's first token may attend to
//                  under a causal mask (token t of the block: causal + t)
//   [7] slot << 16 | part << 8 | n_parts   (a whole item: n_parts = 1, slot = 0xffff)
// A kv list is cut into n_parts = ceil(n_kept / chunk_max) parts of (almost) equal length only when there is room for
// partial results (max_slots > 0) and the launch has more than min_items and at most num_streams items: chunk_max = max(min_chunk,
// ceil(total_kept / num_streams), ceil(max_nkv / 255)); otherwise every item is one unit.
// unit_counters: n_units, partial slots in use, chunk_max, status. arrive[slot] = 0 for every slot.
constexpr int kUnitSortMax = 2048;

__global__ void __launch_bounds__(1024) attn_units_kernel(UnitArgs a) {
  __shared__ int s_warp_u[32], s_warp_p[32];
  __shared__ int s_carry_u, s_carry_p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool list_ok = a.counters[2] == kDevOk;
  int n_items = a.counters[0];
  if (!list_ok || n_items < 0) n_items = 0;
  if (n_items > a.max_items) n_items = static_cast<int>(a.max_items);
  const long long total_kept = a.counters[1];
  int chunk_max = 0x7fffffff;
  if (n_items > a.min_items && a.max_slots > 0 && n_items <= a.num_streams) {
    long long c = (total_kept + a.num_streams - 1) / a.num_streams;
    if (c < a.min_chunk) c = a.min_chunk;
    const long long c255 = (static_cast<long long>(a.max_nkv) + 254) / 255;
    if (c < c255) c = c255;
    chunk_max = static_cast<int>(c);
  }
  for (int64_t i = tid; i < a.max_slots; i += blockDim.x) a.arrive[i] = 0;
  if (tid == 0) { s_carry_u = 0; s_carry_p = 0; }
  __syncthreads();
  for (int base = 0; base < n_items; base += blockDim.x) {
    const int pos = base + tid;
    int it = 0, n = 0, np = 0;
    int4 rec = make_int4(0, 0, 0, 0);
    if (pos < n_items) {
      it = a.order[pos];
      rec = *reinterpret_cast<const int4*>(a.items + 4 * it);  // (b, mask head, qb, n_kept)
      n = rec.w > 0 ? rec.w : 0;
      np = n > chunk_max ? (n + chunk_max - 1) / chunk_max : 1;
    }
    const int sp = np > 1 ? np : 0;
    int xu = np, xp = sp;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yu = __shfl_up_sync(0xffffffffu, xu, o);
      const int yp = __shfl_up_sync(0xffffffffu, xp, o);
      if (lane >= o) { xu += yu; xp += yp; }
    }
    if (lane == 31) { s_warp_u[warp] = xu; s_warp_p[warp] = xp; }
    __syncthreads();
    if (warp == 0) {
      int wu = s_warp_u[lane], wp = s_warp_p[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int yu = __shfl_up_sync(0xffffffffu, wu, o);
        const int yp = __shfl_up_sync(0xffffffffu, wp, o);
        if (lane >= o) { wu += yu; wp += yp; }
      }
      s_warp_u[lane] = wu;
      s_warp_p[lane] = wp;
    }
    __syncthreads();
    const int off_u = s_carry_u + (warp ? s_warp_u[warp - 1] : 0) + xu - np;
    const int off_p = s_carry_p + (warp ? s_warp_p[warp - 1] : 0) + xp - sp;
    if (pos < n_items) {
      const int q0 = a.qo_indptr[rec.x], q_len = a.qo_indptr[rec.x + 1] - q0;
      const int k0 = a.kv_indptr[rec.x], kv_len = a.kv_indptr[rec.x + 1] - k0;
      const int kvp = a.kv_ptr[it];
      int q_valid = q_len - rec.z * a.sbq;
      q_valid = q_valid > a.sbq ? a.sbq : (q_valid < 0 ? 0 : q_valid);
      int ragged = 0;
      const int tail_cols = kv_len % a.sbkv;
      // lists are ascending: only the item's last entry can be the request's partial block
      if (tail_cols != 0 && n > 0 && a.kv_idx[kvp + n - 1] == kv_len / a.sbkv) ragged = tail_cols;
      for (int p = 0; p < np; ++p) {
        const int j0 = static_cast<int>(static_cast<long long>(n) * p / np);
        const int j1 = static_cast<int>(static_cast<long long>(n) * (p + 1) / np);
        if (off_u + p < a.max_units) {
          int4* dst = reinterpret_cast<int4*>(a.units + 8 * static_cast<int64_t>(off_u + p));
          const int sp_word = np > 1 ? (((off_p + p) & 0xffff) << 16) | (p << 8) | np : (0xffff << 16) | 1;
          dst[0] = make_int4(j1 - j0, kvp + j0, rec.y | (rec.x << 16), q0 + rec.z * a.sbq);
          dst[1] = make_int4(q_valid | ((p == np - 1 ? ragged : 0) << 16), k0, rec.z * a.sbq + kv_len - q_len, sp_word);
        }
      }
    }
    __syncthreads();
    if (tid == 0) { s_carry_u += s_warp_u[31]; s_carry_p += s_warp_p[31]; }
    __syncthreads();
  }
  // When lists were cut, the units are put in descending order of their length (stable: equal lengths keep the
  // order above), so that the CTAs, which draw units in list order, take the short ones last. Every thread holds
  // its records in registers before any is written back.
  const int n_units = s_carry_u;
  if (chunk_max != 0x7fffffff && n_units <= kUnitSortMax && n_units <= a.max_units) {
    __shared__ int s_len[kUnitSortMax];
    int4 r0[kUnitSortMax / 1024], r1[kUnitSortMax / 1024];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kUnitSortMax / 1024; ++k) {
      const int u = tid + k * 1024;
      if (u < n_units) {
        const int4* src = reinterpret_cast<const int4*>(a.units + 8 * static_cast<int64_t>(u));
        r0[k] = src[0];
        r1[k] = src[1];
        s_len[u] = r0[k].x;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kUnitSortMax / 1024; ++k) {
      const int u = tid + k * 1024;
      if (u < n_units) {
        const int len = r0[k].x;
        int pos = 0;
        for (int v = 0; v < n_units; ++v) {
          const int lv = s_len[v];
          pos += (lv > len || (lv == len && v < u)) ? 1 : 0;
        }
        int4* dst = reinterpret_cast<int4*>(a.units + 8 * static_cast<int64_t>(pos));
        dst[0] = r0[k];
        dst[1] = r1[k];
      }
    }
  }
  if (tid == 0) {
    a.unit_counters[0] = s_carry_u;
    a.unit_counters[1] = s_carry_p;
    a.unit_counters[2] = chunk_max;
    a.unit_counters[3] = (!list_ok || s_carry_u > a.max_units || s_carry_p > a.max_slots || s_carry_p > 0xffff) ? kDevBadIndex : kDevOk;
  }
}

// The same records when no list can be cut (no room for partial results): every item is exactly one unit at its
// position in the processing order, so the items are independent of one another: one thread per item, any number
// of CTAs.
__global__ void __launch_bounds__(256) attn_units_whole_kernel(UnitArgs a) {
  const bool list_ok = a.counters[2] == kDevOk;
  int n_items = a.counters[0];
  if (!list_ok || n_items < 0) n_items = 0;
  if (n_items > a.max_items) n_items = static_cast<int>(a.max_items);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.unit_counters[0] = n_items;
    a.unit_counters[1] = 0;
    a.unit_counters[2] = 0x7fffffff;
    a.unit_counters[3] = (!list_ok || n_items > a.max_units) ? kDevBadIndex : kDevOk;
  }
  for (int64_t pos = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; pos < n_items && pos < a.max_units;
       pos += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int it = a.order[pos];
    const int4 rec = *reinterpret_cast<const int4*>(a.items + 4 * it);  // (b, mask head, qb, n_kept)
    const int n = rec.w > 0 ? rec.w : 0;
    const int q0 = a.qo_indptr[rec.x], q_len = a.qo_indptr[rec.x + 1] - q0;
    const int k0 = a.kv_indptr[rec.x], kv_len = a.kv_indptr[rec.x + 1] - k0;
    const int kvp = a.kv_ptr[it];
    int q_valid = q_len - rec.z * a.sbq;
    q_valid = q_valid > a.sbq ? a.sbq : (q_valid < 0 ? 0 : q_valid);
    int ragged = 0;
    const int tail_cols = kv_len % a.sbkv;
    if (tail_cols != 0 && n > 0 && a.kv_idx[kvp + n - 1] == kv_len / a.sbkv) ragged = tail_cols;
    int4* dst = reinterpret_cast<int4*>(a.units + 8 * pos);
    dst[0] = make_int4(n, kvp, rec.y | (rec.x << 16), q0 + rec.z * a.sbq);
    dst[1] = make_int4(q_valid | (ragged << 16), k0, rec.z * a.sbq + kv_len - q_len, (0xffff << 16) | 1);
  }
}

cudaError_t launch_attn_units(const UnitArgs& a, cudaStream_t stream) {
  if (a.max_slots <= 0) {
    int64_t blocks = (a.max_items + 255) / 256;
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks < 1) blocks = 1;
    attn_units_whole_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(a);
    return cudaGetLastError();
  }
  attn_units_kernel<<<1, 1024, 0, stream>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Small masks: every list above (items, kept blocks, order, unit records) in ONE launch
// ---------------------------------------------------------------------------------------------
// What bounds it: latency. A mask of a few thousand (q-block, head) pairs is some KB; the chain count -> scan -> fill
// -> units spends its time in four launches and in the dependent steps of a one-CTA scan. Here every CTA reads the
// WHOLE mask and counts every candidate into shared memory (redundant and cheap), after which a warp finds the place
// of its own candidate without talking to anybody: one sweep over the counts gives the number of active candidates
// and of kept blocks in front of it (its item and its offset in kv_idx) and the number of smaller sort keys (its
// position in the processing order). No scan, no sort, no second pass.
// A key is (bucket << 12 | candidate): the buckets of the counting sort above, ties by candidate, so the lists are
// the same word for word. With `zero_out` a warp whose q-block is not active (or whose lists do not fit) zeroes that
// block of the output, which saves the caller a pass over the whole tensor.
// Measured on a B200, whole attention call, against the chain and a zeroed allocation: 36 q-blocks x 24 heads x 36
// kv-blocks at density 0.5 134.8 -> 112.2 us, all blocks 302.2 -> 280.3 us; 3 x 4 x 3 blocks 56.6 -> 36.2 us.
constexpr int kSmallThreads = 512, kSmallBatch = 64;
constexpr int64_t kSmallCand = 4096, kSmallBits = 1 << 18;

__device__ __forceinline__ void attn_lists_small_body(const CompactArgs& a, const UnitArgs& u, const ZeroArgs& z,
                                                      const ZeroLater& later, int by_length, int heads_per_group, int cta) {
  extern __shared__ __align__(16) uint32_t s_dyn[];   // [n_cand] keys, then [n_cand] counts
  __shared__ int s_first[kSmallBatch + 1];            // first candidate of a request
  __shared__ int s_q0[kSmallBatch], s_ql[kSmallBatch], s_k0[kSmallBatch], s_kl[kSmallBatch];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = static_cast<int>(a.n_cand), H = a.head_count;
  uint32_t* s_key = s_dyn;
  int* s_cnt = reinterpret_cast<int*>(s_dyn + n);
  if (tid < a.batch) {
    s_q0[tid] = a.qo_indptr[tid];
    s_ql[tid] = a.qo_indptr[tid + 1] - s_q0[tid];
    s_k0[tid] = a.kv_indptr[tid];
    s_kl[tid] = a.kv_indptr[tid + 1] - s_k0[tid];
  }
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int b = 0; b < a.batch; ++b) {
      s_first[b] = acc;
      acc += s_ql[b] > 0 ? (s_ql[b] + a.sbq - 1) / a.sbq * H : 0;
    }
    s_first[a.batch] = acc;
  }
  __syncthreads();
  const int n_real = s_first[a.batch] < n ? s_first[a.batch] : n;
  const int grp_per_req = (H + heads_per_group - 1) / heads_per_group;
  auto request_of = [&](int c) -> int {
    int lo = 0, hi = a.batch;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_first[mid] <= c) lo = mid; else hi = mid;
    }
    return lo;
  };
  for (int c = tid; c < n; c += kSmallThreads) {
    int cnt = -1;
    uint32_t key = 0xffffffffu;
    if (c < n_real) {
      const int b = request_of(c);
      const int local = c - s_first[b], qb = local / H, hl = local - qb * H;
      const int nkv = s_kl[b] > 0 ? (s_kl[b] + a.sbkv - 1) / a.sbkv : 0;
      if (a.is_full) {
        cnt = nkv;
      } else {
        const int64_t ioff = a.info_indptr[b], koff = a.kv_info_indptr[b];
        const int64_t qbit = static_cast<int64_t>(qb) * a.num_heads + a.head_begin + hl;
        if (get_bit(a.sparse_info + ioff, qbit, a.info_bytes - ioff)) {
          cnt = 0;
          for (int w = 0; w < nkv; w += 64) {
            const int rem = nkv - w;
            cnt += __popcll(load_bits64(a.sparse_kv_info + koff, qbit * nkv + w, a.kv_info_bytes - koff, rem < 64 ? rem : 64));
          }
        }
      }
      if (cnt >= 0) {
        int bucket;
        if (by_length) {
          const int len = cnt > a.max_nkv ? a.max_nkv : cnt;
          bucket = (b * grp_per_req + hl / heads_per_group) * (a.max_nkv + 1) + (a.max_nkv - len);
        } else {  // single heads, q-blocks ascending
          bucket = s_first[b] + hl * ((s_first[b + 1] - s_first[b]) / H) + qb;
        }
        key = (static_cast<uint32_t>(bucket) << 12) | static_cast<uint32_t>(c);
      }
    }
    s_cnt[c] = cnt;
    s_key[c] = key;
  }
  __syncthreads();
  const int c = cta * (kSmallThreads / 32) + warp;
  if (c >= n) return;
  const int kept = s_cnt[c];
  const uint32_t key = s_key[c];
  int pos = 0, off = 0, rank = 0, tot_items = 0, tot_kept = 0;
  for (int i = lane; i < n; i += 32) {
    const int v = s_cnt[i];
    const int act = v >= 0 ? 1 : 0, kv = v > 0 ? v : 0;
    tot_items += act;
    tot_kept += kv;
    if (i < c) { pos += act; off += kv; }
    rank += s_key[i] < key ? 1 : 0;
  }
  pos = __reduce_add_sync(0xffffffffu, pos);
  off = __reduce_add_sync(0xffffffffu, off);
  rank = __reduce_add_sync(0xffffffffu, rank);
  tot_items = __reduce_add_sync(0xffffffffu, tot_items);
  tot_kept = __reduce_add_sync(0xffffffffu, tot_kept);
  const int status = (tot_kept > a.max_kept || tot_items > a.max_items) ? kDevBadIndex : kDevOk;
  if (c == 0 && lane == 0) {
    a.counters[0] = tot_items;
    a.counters[1] = tot_kept;
    a.counters[2] = status;
    a.counters[3] = a.max_nkv;
    a.kv_ptr[tot_items <= a.max_items ? tot_items : 0] = tot_kept;
    u.unit_counters[0] = status == kDevOk ? tot_items : 0;
    u.unit_counters[1] = 0;
    u.unit_counters[2] = 0x7fffffff;
    u.unit_counters[3] = (status != kDevOk || tot_items > u.max_units) ? kDevBadIndex : kDevOk;
    if (later.rec != nullptr) *later.count = status != kDevOk || tot_items > u.max_units ? n_real : n_real - tot_items;
  }
  if (c >= n_real) return;
  const int b = request_of(c);
  const int local = c - s_first[b], qb = local / H, hl = local - qb * H;
  int q_valid = s_ql[b] - qb * a.sbq;
  q_valid = q_valid > a.sbq ? a.sbq : q_valid;
  // a q-block that nobody computes: not active, or in lists that do not fit (the attention ignores all of those)
  const bool fits = status == kDevOk && tot_items <= u.max_units;
  if (later.rec != nullptr && (kept < 0 || !fits) && lane == 0)
    later.rec[fits ? c - pos : c] = make_int2(s_q0[b] + qb * a.sbq, (q_valid << 16) | hl);
  if (z.out != nullptr && (kept < 0 || !fits)) {
    const int vecs = z.head_bytes >> 4;   // 16-byte words of one token's share of this mask head
    uint8_t* dst = z.out + static_cast<int64_t>(s_q0[b] + qb * a.sbq) * z.token_bytes + static_cast<int64_t>(hl) * z.head_bytes;
    for (int i = lane; i < q_valid * vecs; i += 32) {
      const int t = i / vecs;
      *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(t) * z.token_bytes + 16 * (i - t * vecs)) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (kept < 0) return;
  if (off + static_cast<int64_t>(kept) > a.max_kept || pos >= a.max_items || rank >= u.max_units) return;  // flagged above
  const int nkv = s_kl[b] > 0 ? (s_kl[b] + a.sbkv - 1) / a.sbkv : 0;
  const int64_t koff = a.is_full ? 0 : a.kv_info_indptr[b];
  const int64_t row0 = (static_cast<int64_t>(qb) * a.num_heads + a.head_begin + hl) * nkv;
  if (lane == 0) {
    const int h = a.head_begin + hl;
    *reinterpret_cast<int4*>(a.items + 4 * pos) = make_int4(b, h, qb, kept);
    a.kv_ptr[pos] = off;
    a.order[rank] = pos;
    // the request's partial last block, if the list ends with it
    const int tail_cols = s_kl[b] % a.sbkv;
    int ragged = 0;
    if (tail_cols != 0 && kept > 0 && nkv > 0 &&
        (a.is_full || get_bit(a.sparse_kv_info + koff, row0 + nkv - 1, a.kv_info_bytes - koff)))
      ragged = tail_cols;
    int4* dst = reinterpret_cast<int4*>(u.units + 8 * static_cast<int64_t>(rank));
    dst[0] = make_int4(kept, off, h | (b << 16), s_q0[b] + qb * a.sbq);
    dst[1] = make_int4(q_valid | (ragged << 16), s_k0[b], qb * a.sbq + s_kl[b] - s_ql[b], (0xffff << 16) | 1);
  }
  if (a.is_full) {
    for (int j = lane; j < nkv; j += 32) a.kv_idx[off + j] = j;
    return;
  }
  int written = 0;
  for (int w0 = 0; w0 < nkv; w0 += 32 * 32) {
    const int w = w0 + lane * 32;
    uint32_t bits = 0;
    if (w < nkv) {
      bits = load_bits32(a.sparse_kv_info + koff, row0 + w, a.kv_info_bytes - koff);
      const int rem = nkv - w;
      if (rem < 32) bits &= (1u << rem) - 1u;
    }
    const int pc = __popc(bits);
    int x = pc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    int dst = written + x - pc;
    while (bits) {
      const int bpos = __ffs(bits) - 1;
      bits &= bits - 1;
      a.kv_idx[off + dst++] = w + bpos;
    }
    written += __shfl_sync(0xffffffffu, x, 31);
  }
}

// kCast: the CTAs past the list builders cast fp8 K and V (0: there are none; else 1 + e5m2 + 2 * bf16). The lists are pure
// latency and the cast pure bandwidth; one behind the other they took 17 us in front of the attention of 3959 tokens with 8
// kv heads on a B200, together 9.8.
template <int kCast>
__global__ void __launch_bounds__(kSmallThreads) attn_lists_small_kernel(CompactArgs a, UnitArgs u, ZeroArgs z, ZeroLater later, CastArgs cast,
                                                                         int list_ctas, int by_length, int heads_per_group) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the attention kernel may set itself up meanwhile
  if (kCast != 0 && static_cast<int>(blockIdx.x) >= list_ctas) {
    const int i = static_cast<int>(blockIdx.x) - list_ctas, ctas = (static_cast<int>(gridDim.x) - list_ctas) / 2, t = i < ctas ? 0 : 1;
    cast_fp8_body<((kCast - 1) & 1) != 0, ((kCast - 1) & 2) != 0>(cast.src[t], cast.n, cast.dst[t], i - t * ctas, ctas);
    return;
  }
  attn_lists_small_body(a, u, z, later, by_length, heads_per_group, static_cast<int>(blockIdx.x));
}

// What the kernel can take: keys have 12 bits for the candidate, and every CTA reads the whole mask (kSmallBits = 32 KB).
// Cut lists and larger masks take the chain above. The lists of a layer step go this way up to here: the chain is six
// launches for them.
bool attn_lists_small_fits(const CompactArgs& a, const UnitArgs& u) {
  return a.n_cand > 0 && a.n_cand <= kSmallCand && a.batch <= kSmallBatch && u.max_slots <= 0 && a.max_nkv < (1 << 18) &&
         (a.is_full || a.n_cand * a.max_nkv <= kSmallBits);
}

// The line lies where the redundant work stays below the launches it saves: it doubles where the CTAs (one per SM, 16
// candidates each) need a second round. Lists alone, graph replays on a B200, chain against one launch: 2048 candidates
// 22-26 and 12-14.5 us, 2560 23.3-24.2 and 20.3-22.1, 3072 21-27 and 23-30, 4096 23-29 and 29-31. To the limit of the
// kernel it goes where the chain has more to do: many requests (4096 candidates of 16 requests 34-35 and 33-34 us, of 64
// 55-59 and 39), all blocks (21-23 and 20.5), and an output to zero, which the chain zeroes whole.
bool attn_lists_small_applies(const CompactArgs& a, const UnitArgs& u, const ZeroArgs& z) {
  return attn_lists_small_fits(a, u) && (a.n_cand <= 2560 || a.batch >= 16 || a.is_full || z.out != nullptr);
}

cudaError_t launch_attn_lists_small(const CompactArgs& a, const UnitArgs& u, const ZeroArgs& z, const ZeroLater& later,
                                    const CastArgs& cast, cudaStream_t stream) {
  int by_length, hpg;
  order_rule(a, &by_length, &hpg);
  const int wpb = kSmallThreads / 32;
  const int blocks = static_cast<int>((a.n_cand + wpb - 1) / wpb);
  const size_t smem = static_cast<size_t>(a.n_cand) * 8;
  if (cast.src[0] == nullptr) {
    attn_lists_small_kernel<0><<<blocks, kSmallThreads, smem, stream>>>(a, u, z, later, cast, blocks, by_length, hpg);
  } else {
    int64_t per = (cast.n / 16 + kSmallThreads - 1) / kSmallThreads;   // cast CTAs for each of K and V
    per = per > 148 * 2 ? 148 * 2 : (per < 1 ? 1 : per);
    const int grid = blocks + 2 * static_cast<int>(per);
    switch (1 + (cast.e5m2 ? 1 : 0) + (cast.is_bf16 ? 2 : 0)) {
      case 1: attn_lists_small_kernel<1><<<grid, kSmallThreads, smem, stream>>>(a, u, z, later, cast, blocks, by_length, hpg); break;
      case 2: attn_lists_small_kernel<2><<<grid, kSmallThreads, smem, stream>>>(a, u, z, later, cast, blocks, by_length, hpg); break;
      case 3: attn_lists_small_kernel<3><<<grid, kSmallThreads, smem, stream>>>(a, u, z, later, cast, blocks, by_length, hpg); break;
      default: attn_lists_small_kernel<4><<<grid, kSmallThreads, smem, stream>>>(a, u, z, later, cast, blocks, by_length, hpg); break;
    }
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// GEMM work lists (single CTA: the candidate counts are a few thousand at most)
// ---------------------------------------------------------------------------------------------
// GEMM-Q: tile records (b, iy, ix0, ix1). Per row block (b, iy) the active column blocks are taken two
// at a time in ascending order; a leftover single block has ix1 = -1. All two-block records come first,
// the single-block records after them, each part in ascending (b, iy) order: the GEMM hands tiles to its
// CTAs in list order, and the half-size tiles at the end fill the last wave. The last `k` two-block records
// are cut into two single-block records each, k chosen so that the launch ends earliest when `n_ctas` CTAs draw
// the records in list order (gemm_q_split_rule: a two-block tile costs 20 time units, a single-block tile 13).
// counters[0] = number of records, counters[1] = number of active 128x128 tiles, counters[3] = number
// of two-block records. The kernel walks the row blocks twice: totals first, then the records; with at most one row block
// per thread (the usual case) the second walk has everything in registers.
// Both list kernels are all latency and sit in front of the GEMM when the caller did not prepare the list: they let it
// start its set-up at once (programmatic dependent launch; the GEMM waits for the list before reading it).
__device__ __forceinline__ void gemm_q_tiles_body(const GemmListArgs& a) {
  __shared__ int s_warp[32];
  __shared__ int s_warp_t[32];
  __shared__ int s_carry, s_carry_t, s_pairs_total, s_best;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int warps = static_cast<int>(blockDim.x) >> 5;   // 32, or the 16 of layer_lists_kernel: only their sums are scanned
  const int mt = a.m / 128, nt = a.n / 128;
  const int rows = a.batch * mt;
  const bool one_walk = rows <= static_cast<int>(blockDim.x);
  int cnt = 0, x = 0, xt = 0;
  const uint8_t* seg = nullptr;
  int64_t limit = 0, bit0 = 0;
  uint64_t rowbits = 0;
  bool fast = false;
  for (int pass = 0; pass < 2; ++pass) {
    if (tid == 0) { s_carry = 0; s_carry_t = 0; }
    __syncthreads();
    const int pairs_total = pass == 0 ? 0 : s_pairs_total;
    const int n_split = pass == 0 ? 0 : (s_best & 0xffff);   // two-block records cut into singles
    const int pairs_kept = pairs_total - n_split;
    for (int base = 0; base < rows; base += blockDim.x) {
      const int r = base + tid;
      const bool have = pass == 1 && one_walk;   // s_warp / s_warp_t still hold the scan, too
      if (!have) cnt = 0;
      if (r < rows && !have) {
        const int b = r / mt, iy = r % mt;
        if (a.is_full) {
          cnt = nt;
        } else {
          const int64_t ioff = a.info_indptr[b];
          seg = a.sparse_info + ioff;
          limit = a.info_bytes - ioff;
          const int64_t qb = (static_cast<int64_t>(a.num_text_tokens) + static_cast<int64_t>(iy) * 128) / a.sparse_q_size;
          bit0 = qb * a.num_heads + a.head_begin;
          if (a.head_dim == 128 && nt <= 64) {  // one bit per column block: fetch the row's bits at once
            rowbits = load_bits64(seg, bit0, limit, nt);
            cnt = __popcll(rowbits);
            fast = true;
          } else {
            for (int ix = 0; ix < nt; ++ix) cnt += get_bit(seg, bit0 + (ix * 128) / a.head_dim, limit);
          }
        }
      }
      // x: two-block records, xt: single-block records (inclusive scans over the CTA)
      const int npair = cnt >> 1, nsingle = cnt & 1;
      if (!have) {
        x = npair; xt = nsingle;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          const int yt = __shfl_up_sync(0xffffffffu, xt, o);
          if (lane >= o) { x += y; xt += yt; }
        }
        if (lane == 31) { s_warp[warp] = x; s_warp_t[warp] = xt; }
        __syncthreads();
        if (warp == 0) {
          int w = lane < warps ? s_warp[lane] : 0, wt = lane < warps ? s_warp_t[lane] : 0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            const int yt = __shfl_up_sync(0xffffffffu, wt, o);
            if (lane >= o) { w += y; wt += yt; }
          }
          s_warp[lane] = w;
          s_warp_t[lane] = wt;
        }
        __syncthreads();
      }
      if (pass == 1 && r < rows && cnt > 0) {
        int pos = s_carry + (warp ? s_warp[warp - 1] : 0) + x - npair;
        const int spos = pairs_total + n_split + s_carry_t + (warp ? s_warp_t[warp - 1] : 0) + xt - nsingle;
        const int b = r / mt, iy = r % mt;
        int first = -1;
        for (int ix = 0; ix < nt; ++ix) {
          if (fast) {   // straight to the next active block
            if (rowbits == 0) break;
            ix = __ffsll(static_cast<long long>(rowbits)) - 1;
            rowbits &= rowbits - 1;
          } else if (!a.is_full && !get_bit(seg, bit0 + (ix * 128) / a.head_dim, limit)) {
            continue;
          }
          if (first < 0) {
            first = ix;
          } else {
            if (pos < pairs_kept) {
              if (pos < a.max_tiles) *reinterpret_cast<int4*>(a.tiles + 4 * pos) = make_int4(b, iy, first, ix);
            } else {
              const int sp = pairs_kept + 2 * (pos - pairs_kept);
              if (sp + 1 < a.max_tiles) {
                *reinterpret_cast<int4*>(a.tiles + 4 * sp) = make_int4(b, iy, first, -1);
                *reinterpret_cast<int4*>(a.tiles + 4 * sp + 4) = make_int4(b, iy, ix, -1);
              }
            }
            ++pos;
            first = -1;
          }
        }
        if (first >= 0 && spos < a.max_tiles) *reinterpret_cast<int4*>(a.tiles + 4 * spos) = make_int4(b, iy, first, -1);
      }
      __syncthreads();
      if (tid == 0) { s_carry += s_warp[31]; s_carry_t += s_warp_t[31]; }
      __syncthreads();
    }
    if (pass == 0) {
      if (tid == 0) { s_pairs_total = s_carry; s_best = 0x7fffffff; }
      __syncthreads();
      // thread k rates the list with its last k two-block records cut; the smallest (end time, k) wins
      const int P = s_carry, S = s_carry_t, n = a.n_ctas > 0 ? a.n_ctas : 1;
      if (tid <= P && tid <= n && P + S + tid <= a.max_tiles) {
        const int t = gemm_q_makespan(P - tid, S + 2 * tid, n);
        atomicMin(&s_best, ((t < 32767 ? t : 32767) << 16) | tid);
      }
      __syncthreads();
      if (tid == 0 && s_best == 0x7fffffff) s_best = 0;  // a list that does not fit is reported below, uncut
      __syncthreads();
    }
  }
  if (tid == 0) {
    const int n_split = s_best & 0xffff;
    const int n_rec = s_carry + s_carry_t + n_split;
    a.counters[0] = n_rec;
    a.counters[1] = 2 * s_carry + s_carry_t;
    a.counters[2] = n_rec > a.max_tiles ? kDevBadIndex : kDevOk;
    a.counters[3] = s_carry - n_split;
    a.counters[4] = kDevOk;  // status word of the GEMM kernel that follows
    a.counters[5] = 0;       // its tile cursor
    a.counters[6] = 0;       // and the count of CTAs that have finished
  }
}

__global__ void __launch_bounds__(1024) gemm_q_tiles_kernel(GemmListArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  gemm_q_tiles_body(a);
}

// GEMM-O: per 128-row block the ascending list of selected local heads, plus the row blocks sorted
// by descending list length (stable). counters[0] = number of row blocks, counters[1] = total heads.
__device__ __forceinline__ void gemm_o_rows_body(const GemmListArgs& a) {
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  extern __shared__ int s_hist[];  // local_heads + 2 buckets
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mt = a.m / 128;
  const int rows = a.batch * mt;
  const int warps = static_cast<int>(blockDim.x) >> 5;   // as in gemm_q_tiles_body
  const int local_heads = a.k / a.head_dim;
  const int want = a.is_for_cache ? 0 : 1;
  if (tid == 0) s_carry = 0;
  for (int i = tid; i <= local_heads; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  for (int base = 0; base < rows; base += blockDim.x) {
    const int r = base + tid;
    int cnt = 0;
    uint64_t rowbits = 0;
    if (r < rows) {
      const int b = r / mt, iy = r % mt;
      const int64_t ioff = a.info_indptr[b];
      const int64_t qb = (static_cast<int64_t>(a.num_text_tokens) + static_cast<int64_t>(iy) * 128) / a.sparse_q_size;
      const int64_t bit0 = qb * a.num_heads + a.head_begin;
      if (local_heads <= 64) {  // fetch the row's bits at once
        rowbits = load_bits64(a.sparse_info + ioff, bit0, a.info_bytes - ioff, local_heads);
        if (!want) rowbits = ~rowbits & (local_heads < 64 ? ((1ull << local_heads) - 1ull) : ~0ull);
        cnt = __popcll(rowbits);
      } else {
        for (int h = 0; h < local_heads; ++h)
          cnt += get_bit(a.sparse_info + ioff, bit0 + h, a.info_bytes - ioff) == want;
      }
    }
    int x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = lane < warps ? s_warp[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    const int off = s_carry + (warp ? s_warp[warp - 1] : 0) + x - cnt;
    if (r < rows) {
      a.row_indptr[r] = off;
      atomicAdd(&s_hist[cnt], 1);
      const int b = r / mt, iy = r % mt;
      const int64_t ioff = a.info_indptr[b];
      const int64_t qb = (static_cast<int64_t>(a.num_text_tokens) + static_cast<int64_t>(iy) * 128) / a.sparse_q_size;
      const int64_t bit0 = qb * a.num_heads + a.head_begin;
      int w = off;
      if (local_heads <= 64) {
        uint64_t bits = rowbits;
        while (bits) {
          a.row_heads[w++] = __ffsll(static_cast<long long>(bits)) - 1;
          bits &= bits - 1;
        }
      } else {
        for (int h = 0; h < local_heads; ++h)
          if (get_bit(a.sparse_info + ioff, bit0 + h, a.info_bytes - ioff) == want) a.row_heads[w++] = h;
      }
    }
    __syncthreads();
    if (tid == 0) s_carry += s_warp[31];
    __syncthreads();
  }
  if (tid == 0) {
    a.row_indptr[rows] = s_carry;
    a.counters[0] = rows;
    a.counters[1] = s_carry;
    a.counters[2] = kDevOk;
    a.counters[4] = kDevOk;  // status word of the GEMM kernel that follows
    a.counters[5] = 0;       // its tile cursor
    a.counters[6] = 0;       // and the count of CTAs that have finished
    // bucket starts, descending count
    int acc = 0;
    for (int k = local_heads; k >= 0; --k) { const int v = s_hist[k]; s_hist[k] = acc; acc += v; }
  }
  __syncthreads();
  if (warp == 0) {
    for (int base = 0; base < rows; base += 32) {
      const int r = base + lane;
      const bool ok = r < rows;
      const int cnt = ok ? (a.row_indptr[r + 1] - a.row_indptr[r]) : -1 - lane;
      const unsigned grp = __match_any_sync(0xffffffffu, cnt);
      const int rank = __popc(grp & ((1u << lane) - 1u));
      const int leader = __ffs(grp) - 1;
      int start = 0;
      if (ok && lane == leader) { start = s_hist[cnt]; s_hist[cnt] = start + __popc(grp); }
      start = __shfl_sync(0xffffffffu, start, leader);
      if (ok) a.row_order[start + rank] = r;
      __syncwarp();
    }
  }
}

__global__ void __launch_bounds__(1024) gemm_o_rows_kernel(GemmListArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  gemm_o_rows_body(a);
}

// The lists of a whole layer step (GEMM-Q tiles, GEMM-O rows, attention items and units) in one launch: they only share
// the masks, so each kind has CTAs of its own. In front of a small layer three launches in a row, each a few
// microseconds of latency, were as long as the projection they ran beside. With 512 threads the GEMM list bodies take a
// second pass past 512 row blocks, where 1024 would do with one.
__global__ void __launch_bounds__(kSmallThreads) layer_lists_kernel(CompactArgs a, UnitArgs u, int by_length, int heads_per_group,
                                                                    GemmListArgs q, GemmListArgs o) {
  if (blockIdx.x == 0) {
    gemm_q_tiles_body(q);
  } else if (blockIdx.x == 1) {
    gemm_o_rows_body(o);
  } else {
    ZeroArgs z;
    z.out = nullptr;
    z.token_bytes = 0;
    z.head_bytes = 16;
    ZeroLater later;
    later.rec = nullptr;
    later.count = nullptr;
    attn_lists_small_body(a, u, z, later, by_length, heads_per_group, static_cast<int>(blockIdx.x) - 2);
  }
}

cudaError_t launch_layer_lists(const CompactArgs& a, const UnitArgs& u, const GemmListArgs& q, const GemmListArgs& o,
                               cudaStream_t stream) {
  int by_length, hpg;
  order_rule(a, &by_length, &hpg);
  const int wpb = kSmallThreads / 32;
  const int blocks = static_cast<int>((a.n_cand + wpb - 1) / wpb) + 2;
  size_t smem = static_cast<size_t>(a.n_cand) * 8;
  const size_t hist = static_cast<size_t>(o.k / o.head_dim + 2) * sizeof(int);
  if (smem < hist) smem = hist;
  layer_lists_kernel<<<blocks, kSmallThreads, smem, stream>>>(a, u, by_length, hpg, q, o);
  return cudaGetLastError();
}

cudaError_t launch_gemm_q_tiles(const GemmListArgs& a, cudaStream_t stream) {
  gemm_q_tiles_kernel<<<1, 1024, 0, stream>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_gemm_o_rows(const GemmListArgs& a, cudaStream_t stream) {
  const int local_heads = a.k / a.head_dim;
  gemm_o_rows_kernel<<<1, 1024, (local_heads + 2) * sizeof(int), stream>>>(a);
  return cudaGetLastError();
}

}  // namespace fo
