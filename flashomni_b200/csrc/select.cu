// Block selection: from pooled attention scores [B, H, n, n] to the packed masks of the hot path
// (sparse_info bits [b][qb][h], sparse_kv_info bits [b][qb][h][kvb], little-endian, one byte segment per
// request). The reference does this with torch ops and Triton fill kernels on an unpacked [B, H, nq, nkv]
// layout that callers then transpose and bit-pack (benchmark/test_attn_score.py:93-133,
// benchmark/utils.py:83-84); here two launches write the packed form directly.
//
// Per row of scores: mass_j = floor(2^31 * exp(x_j - max)) with a fixed polynomial exponential whose
// multiplies and adds are rounded separately (the CPU statement of the same arithmetic is bit-identical),
// integer total, limit = floor(threshold * total) in fp64, and the blocks taken in ascending (mass, index)
// order while the cumulative mass stays <= limit are switched off.
//
// What bounds it: issue slots (the exponential's separately rounded steps and the sums over the row), then the read
// of the scores. A warp owns a row and keeps its masses in registers. No sort and no bit-by-bit search over 48-bit
// keys: the cut is bracketed by masses (lo, hi] with sum(mass <= lo) <= limit < sum(mass <= hi), pivots doubled or
// halved from the mean mass and then halved in float bits, one exact 64-bit sum and count per pivot; as soon as at
// most 32 entries lie in the bracket each lane takes one and ranks it against the others. Equal masses that never get
// below 32 are cut by index directly.
// Measured on a B200 at 40 heads x 604 blocks, thresholds 0.2 / 0.3 (the text-to-image scores switch most q-blocks off):
// whole call 82.4 us with four launches, a memset and threshold arrays, 25.5 us with these two launches; on the device
// 21.1 -> 19.1 us with the score values as asynchronous copies, a byte of sparse_info from at most two flags and the rows'
// flag addresses worked out before the first kernel ends (every row computed 87 -> 83, 24 heads x 2048 blocks 53.6 -> 49).
// Both kernels run their code once per thread, so length of code counts: four masses at a time and unrolled, the ranking of
// the image blocks took 4.0 us instead of 2.4. Rows computed ahead of their flags cost more than they saved (19 -> 28 us).
#include <cooperative_groups.h>

#include <utility>

#include "internal.h"

namespace fo {
namespace {
namespace cg = cooperative_groups;

constexpr int kSelWarps = 8;           // rows per CTA
constexpr int kSelMaxBlocks = 2048;    // longest row (64 entries per lane)

__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Masses of two entries. rint(t) through the 1.5 * 2^23 constant (round to nearest even for |t| < 2^22), whose low
// bits are also the integer n; 2^(n + 31) is added to the exponent field (p in [0.70, 1.42], n >= -64: never
// denormal). Entries with t < -64, and NaN, are 0.
__device__ __forceinline__ void det_exp2_mass2(float xa, float xb, float row_max, uint32_t& ma, uint32_t& mb) {
  constexpr float kMagic = 12582912.0f;
  auto two = [](float c) { return pack_f32x2(c, c); };
  const uint64_t t = mul_f32x2(fadd2(pack_f32x2(xa, xb), two(-row_max)), two(1.4426950408889634f));
  const uint64_t tm = fadd2(t, two(kMagic));
  const uint64_t n = fadd2(tm, two(-kMagic));
  float na, nb, ta, tb, pa, pb, tma, tmb;
  unpack_f32x2(n, na, nb);
  unpack_f32x2(t, ta, tb);
  unpack_f32x2(tm, tma, tmb);
  const uint64_t f = fadd2(t, pack_f32x2(-na, -nb));
  uint64_t p = two(0.0013333558f);
  p = fadd2(mul_f32x2(p, f), two(0.0096181291f));
  p = fadd2(mul_f32x2(p, f), two(0.0555041087f));
  p = fadd2(mul_f32x2(p, f), two(0.2402265070f));
  p = fadd2(mul_f32x2(p, f), two(0.6931471806f));
  p = fadd2(mul_f32x2(p, f), two(1.0f));
  unpack_f32x2(p, pa, pb);
  const int ia = (__float_as_int(tma) - __float_as_int(kMagic) + 31) << 23;
  const int ib = (__float_as_int(tmb) - __float_as_int(kMagic) + 31) << 23;
  ma = __float2uint_rz(__int_as_float(__float_as_int(pa) + ia));
  mb = __float2uint_rz(__int_as_float(__float_as_int(pb) + ib));
  ma = !(ta >= -64.0f) ? 0u : (ma > 0x80000000u ? 0x80000000u : ma);
  mb = !(tb >= -64.0f) ? 0u : (mb > 0x80000000u ? 0x80000000u : mb);
}

// Sum over the warp of values below 2^48 whose bits 48.. hold a count (count sum below 2^16 per lane, mass below 2^37).
__device__ __forceinline__ void warp_sum_count(uint64_t v, uint64_t& sum, int& count) {
  const uint32_t a = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(v & 0x7ffffffu));          // 27 bits
  const uint32_t b = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>((v >> 27) & 0x1fffffu));   // 21 bits
  count = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<uint32_t>(v >> 48)));
  sum = static_cast<uint64_t>(a) + (static_cast<uint64_t>(b) << 27);
}

struct SelScratch {   // per warp
  uint32_t m[32];
  uint32_t j[32];
};

// Keep flags of one row of `len` <= 32 * kPer entries (entry 32 k + i in bit i of words[k]; bits past `len` are 0).
// All 32 lanes call; `words` and `sc` are this warp's shared memory.
template <int kPer>
__device__ __forceinline__ void select_row(const float* __restrict__ x, int len, float threshold, uint32_t* words,
                                           SelScratch* sc) {
  static_assert(kPer % 2 == 0, "entries are handled in pairs");
  const int lane = threadIdx.x & 31;
  uint32_t m[kPer];
  float mx = -INFINITY;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int j = 32 * k + lane;
    const float v = j < len ? x[j] : -INFINITY;
    m[k] = __float_as_uint(v);
    mx = fmaxf(mx, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  uint64_t mine = 0;
#pragma unroll
  for (int k = 0; k < kPer; k += 2) {
    det_exp2_mass2(__uint_as_float(m[k]), __uint_as_float(m[k + 1]), mx, m[k], m[k + 1]);
    if (32 * k + lane >= len) m[k] = 0u;
    if (32 * (k + 1) + lane >= len) m[k + 1] = 0u;
    mine += m[k];
    mine += m[k + 1];
  }
  uint64_t total;
  int cnt;
  warp_sum_count(mine, total, cnt);
  // off: key (mass, index) <= (Km, Kj)
  bool any_off = threshold >= 0.f;
  uint32_t Km = 0xffffffffu;
  int Kj = 0;
  if (any_off) {
    const unsigned long long limit = __double2ull_rd(__dmul_rn(static_cast<double>(threshold), static_cast<double>(total)));
    if (limit < total) {
      uint32_t lo = 0u, hi = 0x80000000u;
      uint64_t sum_lo = 0;
      int cnt_lo = 0, cnt_hi = 32 * kPer;       // entries at or below; not counted yet: the widest bracket
      bool lo_seen = false, hi_seen = false;
      uint32_t piv = static_cast<uint32_t>(total / static_cast<unsigned>(len));
      while (hi - lo > 1u) {
        uint32_t mid = piv;
        if (lo_seen && hi_seen) {   // halve the octaves, then the integers
          mid = (hi >> 1) <= lo ? lo + ((hi - lo) >> 1)
                                : static_cast<uint32_t>(__uint_as_float((__float_as_uint(static_cast<float>(lo)) +
                                                                         __float_as_uint(static_cast<float>(hi))) >> 1));
        }
        if (mid <= lo) mid = lo + 1u;
        if (mid >= hi) mid = hi - 1u;
        uint64_t acc = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
          if (m[k] <= mid) acc += (1ull << 48) + m[k];
        uint64_t s;
        warp_sum_count(acc, s, cnt);
        if (s <= limit) {
          lo = mid; sum_lo = s; cnt_lo = cnt; lo_seen = true;
          piv = mid < 0x40000000u ? mid * 2u : 0x80000000u;
        } else {
          hi = mid; cnt_hi = cnt; hi_seen = true;
          piv = mid >> 1;
        }
        if (cnt_hi - cnt_lo <= 32 && lo_seen && hi_seen) break;
      }
      if (hi - lo <= 1u) {
        // every entry of the bracket has mass `hi`: the first `n_off` of them by index go
        const uint64_t n_off = (limit - sum_lo) / hi;
        Km = lo; Kj = 0x7fffffff;
        uint64_t seen = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          const unsigned eq = __ballot_sync(0xffffffffu, m[k] == hi && 32 * k + lane < len);
          const uint64_t here = static_cast<uint64_t>(__popc(eq));
          if (seen < n_off && n_off <= seen + here) {
            Km = hi;
            Kj = 32 * k + static_cast<int>(__fns(eq, 0, static_cast<int>(n_off - seen)));
          }
          seen += here;
        }
      } else {
        int filled = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          const bool in = m[k] > lo && m[k] <= hi;
          const unsigned b = __ballot_sync(0xffffffffu, in);
          if (in) {
            const int at = filled + __popc(b & ((1u << lane) - 1u));
            if (at < 32) { sc->m[at] = m[k]; sc->j[at] = static_cast<uint32_t>(32 * k + lane); }
          }
          filled += __popc(b);
        }
        __syncwarp();
        const bool have = lane < filled;
        const uint32_t cm = have ? sc->m[lane] : 0xffffffffu;
        const uint32_t cj = have ? sc->j[lane] : 0u;
        uint64_t prefix = sum_lo;
        int rank = 0;
        for (int e = 0; e < filled; ++e) {   // entries are in index order: equal masses rank by lane
          const uint32_t om = sc->m[e];
          const bool before = om < cm || (om == cm && e <= lane);
          prefix += before ? om : 0u;
          rank += before ? 1 : 0;
        }
        const unsigned off = __ballot_sync(0xffffffffu, have && prefix <= limit);
        const int n_off = __popc(off);
        const unsigned last = __ballot_sync(0xffffffffu, have && rank == n_off);
        if (n_off > 0) {
          const int src = __ffs(last) - 1;
          Km = __shfl_sync(0xffffffffu, cm, src);
          Kj = static_cast<int>(__shfl_sync(0xffffffffu, cj, src));
        } else {
          Km = lo; Kj = 0x7fffffff;
        }
        __syncwarp();
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int j = 32 * k + lane;
    const bool off = any_off && (m[k] < Km || (m[k] == Km && j <= Kj));
    const unsigned w = __ballot_sync(0xffffffffu, j < len && !off);
    if (lane == (k & 31)) words[k] = w;
  }
  __syncwarp();
}

// First launch. Cluster b < batch (eight CTAs): which image q-blocks of request b stay on, sparse_info and the indptrs;
// the other clusters zero the kv bit stream, into which the rows of the second launch are written.
// The text-to-image score of a block is sum over heads (outer) and text rows (inner) of score[b][h][q][t2t + j] in
// sequential fp32: a CTA fetches the values of its eighth of the blocks with every thread into shared memory (asynchronous
// copies, a warp per score row, so that no thread holds values or divides per value), one thread
// per block adds them up. The scores then go to all eight CTAs (distributed shared memory), which compute the masses
// redundantly and rank an eighth of the blocks each, eight lanes per block, against all of them: no sort, no search.
// Shared memory of another CTA may only be touched once that CTA runs: each announces itself at the cluster barrier on
// entry and waits there just in front of its first remote store, so that the barrier's latency lies under the score loads.
constexpr int kSelQThreads = 1024, kSelCluster = 8;
constexpr int kT2iFloats = 16384;      // values in flight per pass and CTA (64 KB)
__global__ void __cluster_dims__(kSelCluster, 1, 1) __launch_bounds__(kSelQThreads) select_q_kernel(SelectArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ float s_val[];
  __shared__ float s_t2i[kSelMaxBlocks];
  __shared__ uint32_t s_mass[kSelMaxBlocks];
  __shared__ uint8_t s_keep[kSelMaxBlocks];
  __shared__ float s_max[kSelQThreads / 32];
  __shared__ unsigned long long s_sum[kSelQThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = static_cast<int>(blockIdx.x) / kSelCluster, rank = static_cast<int>(blockIdx.x) % kSelCluster;
  if (b >= a.batch) {
    const int first = a.batch * kSelCluster;
    uint32_t* words = reinterpret_cast<uint32_t*>(a.sparse_kv_info);
    const int64_t step = static_cast<int64_t>(gridDim.x - first) * kSelQThreads;
    for (int64_t i = static_cast<int64_t>(blockIdx.x - first) * kSelQThreads + tid; i < a.kv_words; i += step) words[i] = 0u;
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  const int n_img = a.n - a.t2t;
  if (n_img > 0 && a.t2t > 0) {
    auto running = cluster.barrier_arrive();
    const int share = (n_img + kSelCluster - 1) / kSelCluster, j0 = rank * share;
    const int cols = n_img - j0 < share ? (n_img - j0 > 0 ? n_img - j0 : 0) : share;
    const int pairs = a.heads * a.t2t, per_pass = kT2iFloats / share;
    const float* score = a.score + static_cast<int64_t>(b) * a.heads * a.n * a.n + a.t2t + j0;
    float acc = 0.f;
    for (int p0 = 0; p0 < pairs; p0 += per_pass) {
      const int np = pairs - p0 < per_pass ? pairs - p0 : per_pass;
      for (int p = warp; p < np; p += kSelQThreads / 32) {   // all of them in flight at once
        const int pair = p0 + p, h = pair / a.t2t, q = pair - h * a.t2t;
        const float* src = score + (static_cast<int64_t>(h) * a.n + q) * a.n;
        for (int c = lane; c < cols; c += 32) cp_async_4(s_val + p * cols + c, src + c);
      }
      cp_async_wait_all();
      __syncthreads();
      if (tid < cols) {
#pragma unroll 8
        for (int p = 0; p < np; ++p) acc = __fadd_rn(acc, s_val[p * cols + tid]);
      }
      __syncthreads();
    }
    cluster.barrier_wait(std::move(running));
    if (tid < cols) {
#pragma unroll
      for (int r = 0; r < kSelCluster; ++r) cluster.map_shared_rank(s_t2i, r)[j0 + tid] = acc;
    }
    cluster.sync();
    float mx = -INFINITY;
    for (int j = tid; j < n_img; j += kSelQThreads) mx = fmaxf(mx, s_t2i[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) s_max[warp] = mx;
    __syncthreads();
    mx = s_max[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    unsigned long long mine = 0;
    for (int j = tid; j < n_img; j += kSelQThreads) {
      uint32_t m, unused;
      det_exp2_mass2(s_t2i[j], s_t2i[j], mx, m, unused);
      s_mass[j] = m;
      mine += m;
    }
    uint64_t part;
    int none;
    warp_sum_count(mine, part, none);
    if (lane == 0) s_sum[warp] = part;
    __syncthreads();
    unsigned long long total = s_sum[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const float threshold = a.q_thr != nullptr ? a.q_thr[b] : a.q_thr_all;
    const bool any_off = threshold >= 0.f;
    const unsigned long long limit =
        any_off ? __double2ull_rd(__dmul_rn(static_cast<double>(threshold), static_cast<double>(total))) : 0ull;
    const int sub = lane & 7;
    for (int e = j0 + (tid >> 3); e < j0 + cols; e += kSelQThreads / 8) {
      const uint32_t em = s_mass[e];
      unsigned long long prefix = 0;
      for (int i = sub; i < n_img; i += 8) {
        const uint32_t m = s_mass[i];
        if (m < em || (m == em && i <= e)) prefix += m;
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) prefix += __shfl_xor_sync(0xffu << (lane & 24), prefix, o);
      cluster.map_shared_rank(s_keep, sub)[e] = (any_off && prefix <= limit) ? 0 : 1;
    }
    cluster.sync();
  } else {  // no text rows to score the image blocks with: everything stays on
    for (int j = tid; j < n_img; j += kSelQThreads) s_keep[j] = 1;
    __syncthreads();
  }
  auto kept = [&](int qb) -> uint32_t { return qb < a.t2t ? 1u : s_keep[qb - a.t2t]; };   // text blocks always
  const int t0 = rank * kSelQThreads + tid;
  for (int qb = t0; qb < a.n; qb += kSelCluster * kSelQThreads)
    a.q_keep[static_cast<int64_t>(b) * a.n + qb] = static_cast<uint8_t>(kept(qb));
  const int64_t nbits = static_cast<int64_t>(a.n) * a.heads;
  for (int64_t i = t0; i < a.info_seg_bytes; i += kSelCluster * kSelQThreads) {
    uint32_t v = 0;
    int qb = i < (1 << 28) ? static_cast<int>(i) * 8 / a.heads : static_cast<int>(i * 8 / a.heads);
    int h = static_cast<int>(i * 8 - static_cast<int64_t>(qb) * a.heads);
    if (a.heads >= 8) {   // one or two q-blocks in the byte
      const int left = a.heads - h, own = left < 8 ? left : 8;
      if (kept(qb)) v = (1u << own) - 1u;
      if (own < 8 && qb + 1 < a.n && kept(qb + 1)) v |= 0xffu << own & 0xffu;
    } else {
      for (int t = 0; t < 8; ++t) {
        if (i * 8 + t < nbits && kept(qb)) v |= 1u << t;
        if (++h == a.heads) { h = 0; ++qb; }
      }
    }
    a.sparse_info[b * a.info_seg_bytes + i] = static_cast<uint8_t>(v);
  }
  if (t0 == 0) {
    if (b == 0) a.info_indptr[0] = a.kv_info_indptr[0] = 0;
    a.info_indptr[b + 1] = static_cast<int32_t>((b + 1) * a.info_seg_bytes);
    a.kv_info_indptr[b + 1] = static_cast<int32_t>((b + 1) * a.kv_seg_bytes);
  }
}

// Second launch: a warp per (b, h, qb) row writes its keep flags into the zeroed stream, rows dealt round-robin over the
// resident warps; a warp looks up the q-block flags of 32 of its rows at once, so rows of blocks that are off (most of
// them, when the text-to-image scores are peaked) cost nothing. Launched while the first one runs (programmatic
// dependent launch), which it waits for before anything else. The words that a row shares with its neighbours are
// OR-ed, the others stored.
template <int kPer>
__global__ void __launch_bounds__(kSelWarps * 32) select_kv_kernel(SelectArgs a) {
  __shared__ uint32_t s_words[kSelWarps][kPer];
  __shared__ SelScratch s_sc[kSelWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t rows = static_cast<int64_t>(a.batch) * a.heads * a.n;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kSelWarps + warp, step = static_cast<int64_t>(gridDim.x) * kSelWarps;
  uint32_t* words = s_words[warp];
  auto keep_of = [&](int64_t row) { return a.q_keep + row / (static_cast<int64_t>(a.n) * a.heads) * a.n + row % a.n; };
  const uint8_t* keep = keep_of(first + lane * step < rows ? first + lane * step : 0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int64_t base = first; base < rows; base += 32 * step) {
    const int64_t mine = base + lane * step;
    bool on = mine < rows;
    if (base != first && on) keep = keep_of(mine);
    if (on && a.zero_inactive) on = __ldcg(keep) != 0;
    for (unsigned left = __ballot_sync(0xffffffffu, on); left != 0u; left &= left - 1u) {
      const int64_t row = base + (__ffs(left) - 1) * step;
      const int q = static_cast<int>(row % a.n);
      const int h = static_cast<int>((row / a.n) % a.heads);
      const int b = static_cast<int>(row / (static_cast<int64_t>(a.n) * a.heads));
      if (q < a.t2t) {  // text rows keep every kv-block
        for (int k = lane; k < kPer; k += 32) {
          const int rem = a.n - 32 * k;
          words[k] = rem >= 32 ? 0xffffffffu : (rem > 0 ? (1u << rem) - 1u : 0u);
        }
        __syncwarp();
      } else {
        const float* x = a.score + ((static_cast<int64_t>(b) * a.heads + h) * a.n + q) * a.n;
        select_row<kPer>(x, a.n, a.kv_thr != nullptr ? a.kv_thr[h] : a.kv_thr_all, words, &s_sc[warp]);
      }
      const int64_t bit0 = static_cast<int64_t>(b) * a.kv_seg_bytes * 8 + (static_cast<int64_t>(q) * a.heads + h) * a.n;
      uint32_t* out = reinterpret_cast<uint32_t*>(a.sparse_kv_info) + (bit0 >> 5);
      const int sh = static_cast<int>(bit0 & 31);
      const int n_in = (a.n + 31) >> 5, n_out = (sh + a.n + 31) >> 5;
      for (int i = lane; i < n_out; i += 32) {
        const uint32_t cur = i < n_in ? words[i] : 0u, prev = i > 0 ? words[i - 1] : 0u;
        const uint32_t w = sh != 0 ? (cur << sh) | (prev >> (32 - sh)) : cur;
        if (i * 32 >= sh && (i + 1) * 32 <= sh + a.n) out[i] = w;
        else if (w != 0u) atomicOr(out + i, w);
      }
      __syncwarp();
    }
  }
}

}  // namespace

template <int kPer>
static cudaError_t launch_kv(const SelectArgs& a, cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(a.batch) * a.heads * a.n;
  int64_t ctas = (rows + kSelWarps - 1) / kSelWarps;
  if (ctas > 148 * 3) ctas = 148 * 3;
  return launch_dependent(select_kv_kernel<kPer>, static_cast<int>(ctas), kSelWarps * 32, 0, stream, true, a);
}

cudaError_t launch_select_blocks(const SelectArgs& a, cudaStream_t stream) {
  if (a.n > kSelMaxBlocks) return cudaErrorInvalidValue;
  int64_t zero_clusters = (a.kv_words + 4 * kSelCluster * kSelQThreads - 1) / (4 * kSelCluster * kSelQThreads);
  if (zero_clusters > 16) zero_clusters = 16;
  if (zero_clusters < 1) zero_clusters = 1;
  cudaError_t e = cudaFuncSetAttribute(select_q_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kT2iFloats * 4);
  if (e != cudaSuccess) return e;
  select_q_kernel<<<static_cast<int>((a.batch + zero_clusters) * kSelCluster), kSelQThreads, kT2iFloats * 4, stream>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // Entries per lane: image layers, video layers, and whatever else is allowed. The masses of a row live in registers, so a
  // wider instantiation costs occupancy and idle lanes: every row computed, whole call on a B200, 40 heads x 604 / 640 blocks
  // 94 / 102 us (522 / 546 with the search in shared memory that this replaced), 641 blocks 301 (584), 24 heads x 2048
  // 661 (2878). A step between 640 and 2048 would help the sizes just past 640; none is built.
  if (a.n <= 128) return launch_kv<4>(a, stream);
  if (a.n <= 640) return launch_kv<20>(a, stream);
  return launch_kv<64>(a, stream);
}

}  // namespace fo
