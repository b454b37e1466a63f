// GEMM-Q / GEMM-O on tcgen05: one persistent, warp-specialised kernel.
//
//   Y[b, rows(iy), cols(ix)] = init + sum_{k-blocks of the tile} X[b, rows, kblk] * W[cols, kblk]^T
//
// GEMM-Q (reference: include/flashomni/gemm/w16a16/gemm.cuh:27-228): the tile list holds only the
// active 128x128 output tiles; every tile runs the whole K range; init = bias[cols] or 0; tiles
// that are not listed are never touched.
// GEMM-O (reference: include/flashomni/gemm/w16a16/gemm_reduction.cuh:27-276): every output tile is
// produced; its K loop visits only the K-slices of the heads selected for its row block (compacted
// list, ascending); init = cache[b, rows, cols] or bias[cols] or 0.
//
// A CTA works on "pair tiles": one 128-row A tile against TWO 128-column blocks of W (any two: for
// GEMM-Q they are two active heads of the same row block), issued as one UMMA of N = 256 so that
// the A operand is read from shared memory once per 256 output columns. A leftover single block
// runs as N = 128.
//
// CTA = 192 threads: warps 0-3 epilogue, warp 4 TMA producer, warp 5 MMA issuer (with a full init tensor warp 6 loads its
// slabs). K step 64 (one 128-byte swizzle atom), 4-stage ring of (A 16 KB + B 32 KB), two 256-column TMEM accumulators so
// the epilogue of tile i overlaps the main loop of tile i+1. The epilogue converts slabs of 64 columns, or 32 with a full init
// tensor (TMEM -> registers -> +init -> 16-bit) into a swizzled shared-memory slab and hands each slab to a
// TMA store, so global writes are full 128-byte lines and asynchronous. The tiles of the sparse modes
// (unequal lengths) are handed to the persistent CTAs through a device-wide cursor, in list order; the
// equal tiles of a dense launch keep fixed round-robin shares.
#include <cuda_fp16.h>

#include "internal.h"
#include "mask_bits.cuh"

namespace fo {
namespace {

constexpr int kBM = 128, kBNH = 128, kBK = 64;
constexpr int kABytes = kBM * kBK * 2;        // 16 KB
constexpr int kBHalfBytes = kBNH * kBK * 2;   // 16 KB per 128-column block of W
constexpr int kStageBytes = kABytes + 2 * kBHalfBytes;
constexpr int kStages = 4;
constexpr int kSlabsBytes = 2 * kBM * 64 * 2;    // staging of the epilogue: two slabs of 64 columns, or four of 32
constexpr int kMaxSlabBufs = 4;
// With a full init tensor (GEMM-O and the cached contribution) the init values of a slab are loaded by TMA into the staging
// slab that the result leaves from, up to three slabs ahead, by a warp of their own. Loaded by the epilogue threads instead, one
// slab ahead and a row per thread, they made the epilogue wait for HBM on every slab. GEMM-O with its list, inputs that change
// from call to call, us on a B200, threads -> TMA: 9216 rows x 3072 with 3 / 6 / 12 / 24 heads 54.7 / 57.0 / 63.9 / 90.7 -> 41.7 /
// 45.0 / 55.6 / 87.1, 4608 rows 31.5 / 34.5 / 40.6 / 56.5 -> 26.4 / 29.2 / 36.9 / 54.1, 1024 rows with 24 heads 33.3 -> 32.1, 4608 x 5120
// with 40 heads 125.8 -> 121.6. Slabs of 64 columns would leave three operand stages: 38.0 us with 3 heads of 9216
// rows, but 91.3 with 24 and 239 against 230 with 40 of 9216 x 5120.
constexpr int threads_of(bool cache) { return cache ? 224 : 192; }
constexpr int slabs_of(bool cache) { return cache ? 4 : 2; }
constexpr int kTmemCols = 512;
constexpr int kMaxHeadsSmem = 128;
constexpr int kTileQ = 8;   // entries of the tile queue (the producer runs at most a few tiles ahead of the epilogue)
constexpr int kFirstRows = 192;   // own_first: row blocks, one per thread of the smaller CTA

struct alignas(16) Tail {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t slab_full[kMaxSlabBufs];    // init values of a slab have landed
  uint64_t slab_empty[kMaxSlabBufs];   // the store of the slab has read it
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t tq_full[kTileQ];   // tile queue: the producer warp draws tiles, looks them up and hands them to the other roles
  uint64_t tq_empty[kTileQ];
  int4 tile_q[kTileQ];        // (a_row, w_row0, w_row1, nkb); a_row -1 ends the sequence
  uint32_t tmem_base;
  int abort_flag;
  int epi_go;                   // outcome of the epilogue warps' vote of the current round
  int heads[2][kMaxHeadsSmem];  // GEMM-O: head lists of the current and the next tile, staged for the producer
};
constexpr int kSmemBytes = kStages * kStageBytes + kSlabsBytes + 1024 + static_cast<int>(sizeof(Tail));
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");


struct TileInfo {
  int a_row;             // first row of the A tile in [batch*m]
  int w_row0, w_row1;    // first rows of the two W blocks (= first output columns); w_row1 < 0: single
  int nkb;               // number of 64-wide K blocks
  const int32_t* heads;  // GEMM-O: selected heads of the row block (null for GEMM-Q)
};

// tiles per row block where the launch has no tile list: pairs of column blocks, or single blocks (launch_gemm)
__device__ __forceinline__ int tiles_per_row(const GemmArgs& a) { return a.single ? a.n / kBNH : (a.n / kBNH + 1) / 2; }

__device__ __forceinline__ int num_tiles(const GemmArgs& a) {
  if (a.mode == kGemmQ && a.tiles != nullptr) {
    const int cap = a.batch * (a.m / kBM) * (a.n / kBNH);  // a list holds at most one record per 128x128 tile
    const int n = *a.n_tiles_ptr;
    return n < cap ? (n < 0 ? 0 : n) : cap;
  }
  return a.batch * (a.m / kBM) * tiles_per_row(a);
}

__device__ __forceinline__ TileInfo get_tile(const GemmArgs& a, int t) {
  TileInfo ti;
  const int nct = a.n / kBNH;
  if (a.mode == kGemmQ && a.tiles != nullptr) {
    const int4 rec = *reinterpret_cast<const int4*>(a.tiles + 4 * t);  // (b, iy, ix0, ix1)
    ti.a_row = rec.x * a.m + rec.y * kBM;
    ti.w_row0 = rec.z * kBNH;
    ti.w_row1 = rec.w >= 0 ? rec.w * kBNH : -1;
    ti.nkb = (a.k + kBK - 1) / kBK;  // a last partial K block reads zeros past k (TMA fill)
    ti.heads = nullptr;
    return ti;
  }
  const int npr = tiles_per_row(a);
  const int j = t % npr;
  const int rr = t / npr;
  ti.w_row0 = (a.single ? j : 2 * j) * kBNH;
  ti.w_row1 = (!a.single && 2 * j + 1 < nct) ? (2 * j + 1) * kBNH : -1;
  if (a.mode == kGemmQ) {  // dense: row blocks in natural order
    ti.a_row = rr * kBM;
    ti.nkb = (a.k + kBK - 1) / kBK;  // a last partial K block reads zeros past k (TMA fill)
    ti.heads = nullptr;
  } else {
    const int r = a.row_order[rr];
    ti.a_row = r * kBM;
    const int h0 = a.row_indptr[r], h1 = a.row_indptr[r + 1];
    ti.heads = a.row_heads + h0;
    ti.nkb = (h1 - h0) * a.kb_per_head;
  }
  return ti;
}

// What the list kernel in front of this one writes for tile blockIdx.x, worked out from the mask by the whole CTA: one row block
// per thread, at most kFirstRows of them and 64 column blocks (GEMM-Q, heads of 128) or heads (GEMM-O). With the list the first
// operands of a 4608 x 24 heads GEMM-Q arrive 9.6 us after its launch, with the mask after 4.4; what is left of that in the
// whole call is less, since the operands of the first round come from HBM in either case. GEMM-Q / GEMM-O with list kernel,
// inputs that change from call to call, us on a B200: 512 rows x 6 heads 12.5 / 13.6 -> 12.0 / 12.5, 1024 x 8 14.3 / 15.4 -> 13.6 /
// 14.3, 1280 x 24 32.8 / 31.0 -> 30.7 / 28.9, 2560 x 12 21.5 / 22.3 -> 20.0 / 20.2, 4608 x 24 51.6 / 52.2 -> 50.2 / 51.0, 9216 x 24
// 84.2 / 84.7 -> 83.2 / 84.0. More row blocks than that take 150 us and more, of which the list is a few percent.
struct FirstScratch {   // in the staging slabs, which nothing uses yet
  int sums[8];
  int hist[65];
  int best;
  int2 tile;            // GEMM-Q: (row block, column blocks ix0 | ix1 << 8, ix1 255 for a single one); GEMM-O: (row block, -)
  unsigned long long bits;
};
__device__ __forceinline__ TileInfo first_tile(const GemmArgs& a, FirstScratch& s, int* heads) {
  const GemmListArgs& l = a.list;
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, warp = tid >> 5, warps = static_cast<int>(blockDim.x) >> 5;
  const int mt = a.m / kBM, rows = a.batch * mt, t = static_cast<int>(blockIdx.x);
  const bool q = a.mode == kGemmQ;
  const int nbits = q ? a.n / kBNH : l.k / l.head_dim;
  TileInfo ti;
  ti.a_row = -1; ti.w_row0 = ti.nkb = 0; ti.w_row1 = -1; ti.heads = nullptr;

  for (int i = tid; i <= 64; i += static_cast<int>(blockDim.x)) s.hist[i] = 0;
  if (tid == 0) { s.best = 0x7fffffff; s.tile = make_int2(-1, 0); }
  uint64_t bits = 0;
  if (tid < rows) {
    const int b = tid / mt, iy = tid % mt;
    const int64_t ioff = l.info_indptr[b];
    const uint32_t qb = (static_cast<uint32_t>(l.num_text_tokens) + static_cast<uint32_t>(iy) * 128u) / static_cast<uint32_t>(l.sparse_q_size);
    bits = load_bits64(l.sparse_info + ioff, static_cast<int64_t>(qb) * l.num_heads + l.head_begin, l.info_bytes - ioff, nbits);
    if (!q && l.is_for_cache) bits = ~bits & (nbits < 64 ? (1ull << nbits) - 1ull : ~0ull);
  }
  const int cnt = __popcll(bits);
  if (q) {
    const int npair = cnt >> 1, nsingle = cnt & 1;
    int x = npair << 16 | nsingle;   // inclusive scans of both kinds of record in one word: at most 192 * 32 and 192
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s.sums[warp] = x;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < warps; ++w) {
      if (w == warp) before = total;
      total += s.sums[w];
    }
    x += before;
    const int P = total >> 16, S = total & 0xffff, n = l.n_ctas > 0 ? l.n_ctas : 1;
    for (int k = tid; k <= P && k <= n && k < 1024 && P + S + k <= l.max_tiles; k += static_cast<int>(blockDim.x)) {
      const int e = gemm_q_makespan(P - k, S + 2 * k, n);
      atomicMin(&s.best, ((e < 32767 ? e : 32767) << 16) | k);
    }
    __syncthreads();
    const int n_split = s.best == 0x7fffffff ? 0 : s.best & 0xffff, kept = P - n_split;
    const int p0 = (x >> 16) - npair, s0 = (x & 0xffff) - nsingle;   // numbers of this row's first records
    const int cut = t - kept, single = t - P - n_split;
    int skip = -1, take = 0;   // active column blocks of this row in front of the tile, and its own
    if (t < kept) {
      if (t >= p0 && t < p0 + npair) { skip = 2 * (t - p0); take = 2; }
    } else if (cut < 2 * n_split) {
      const int p = kept + (cut >> 1);
      if (p >= p0 && p < p0 + npair) { skip = 2 * (p - p0) + (cut & 1); take = 1; }
    } else if (nsingle && single == s0) {
      skip = cnt - 1; take = 1;
    }
    if (take) {
      uint64_t rest = bits;
      for (int i = 0; i < skip; ++i) rest &= rest - 1;
      const int ix0 = __ffsll(static_cast<long long>(rest)) - 1;
      rest &= rest - 1;
      s.tile = make_int2(tid, ix0 | (take == 2 ? __ffsll(static_cast<long long>(rest)) - 1 : 255) << 8);
    }
    __syncthreads();
    const int2 rec = s.tile;
    if (rec.x < 0) return ti;
    ti.a_row = rec.x * kBM;
    ti.w_row0 = (rec.y & 255) * kBNH;
    ti.w_row1 = (rec.y >> 8) == 255 ? -1 : (rec.y >> 8) * kBNH;
    ti.nkb = (a.k + kBK - 1) / kBK;
    return ti;
  }
  // GEMM-O: the row block that comes (t / tiles of a row)-th when they are sorted by falling head count, stable
  __syncthreads();
  if (tid < rows) atomicAdd(&s.hist[cnt], 1);
  __syncthreads();
  const int npr = tiles_per_row(a), want = t / npr, j = t % npr;
  // counts from 64 down, two a lane: the bucket that holds the row and how many rows of that count come before it
  const int h1 = s.hist[64 - 2 * lane], h2 = s.hist[63 - 2 * lane];
  int x = h1 + h2;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const unsigned past = __ballot_sync(0xffffffffu, x > want);
  int bucket = 0, nth = want - __shfl_sync(0xffffffffu, x, 31);   // no lane: the rows without a head
  if (past != 0u) {
    const int src = __ffs(past) - 1;
    const int start = __shfl_sync(0xffffffffu, x - h1 - h2, src), first = __shfl_sync(0xffffffffu, h1, src);
    const bool lower = want >= start + first;
    bucket = 64 - 2 * src - (lower ? 1 : 0);
    nth = want - start - (lower ? first : 0);
  }
  const unsigned mine = __ballot_sync(0xffffffffu, tid < rows && cnt == bucket);
  if (lane == 0) s.sums[warp] = __popc(mine);
  __syncthreads();
  int before = __popc(mine & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) before += s.sums[w];
  if (tid < rows && cnt == bucket && before == nth) {
    s.tile = make_int2(tid, 0);
    s.bits = bits;
  }
  __syncthreads();
  const int row = s.tile.x;
  if (row < 0) return ti;
  const uint64_t hb = s.bits;
  if (tid < 64 && (hb >> tid & 1ull)) heads[__popcll(hb & ((1ull << tid) - 1ull))] = tid;
  fence_proxy_async_smem();   // the first init slabs land on the scratch
  __syncthreads();
  ti.a_row = row * kBM;
  ti.w_row0 = (a.single ? j : 2 * j) * kBNH;
  ti.w_row1 = (!a.single && 2 * j + 1 < a.n / kBNH) ? (2 * j + 1) * kBNH : -1;
  ti.nkb = __popcll(hb) * a.kb_per_head;
  ti.heads = heads;
  return ti;
}

__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <bool kBf16, bool kCache>
__global__ void __launch_bounds__(threads_of(kCache), 1) gemm_kernel(const __grid_constant__ GemmArgs a) {
  constexpr int kSlabBufs = slabs_of(kCache), kSlabCols = kCache ? 32 : 64, kSlabBytes = kBM * kSlabCols * 2;
  constexpr int kSlabsPerBlock = kBNH / kSlabCols;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* smem_slab = smem + kStages * kStageBytes;
  Tail* tail = reinterpret_cast<Tail*>(smem_slab + kSlabsBytes);
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tail->acc_full[i], 1);
      mbar_init(&tail->acc_empty[i], 4);
    }
    for (int i = 0; i < kTileQ; ++i) {
      mbar_init(&tail->tq_full[i], 1);
      mbar_init(&tail->tq_empty[i], kCache ? 6 : 5);  // the MMA thread, the four epilogue warps, the loader of init slabs
    }
    for (int i = 0; i < kSlabBufs; ++i) {
      mbar_init(&tail->slab_full[i], 1);
      mbar_init(&tail->slab_empty[i], 1);
    }
    tail->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&a.tmap_a);
    tma_prefetch_desc(&a.tmap_b);
    tma_prefetch_desc(&a.tmap_y);
    if (kCache) tma_prefetch_desc(&a.tmap_c);
  }
  if (warp == 5) {
    tmem_alloc(&tail->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tail->tmem_base;
  // launched while the list in front of it was built: waits for it now, or before the second tile (every CTA, also one without)
  if (a.after_list && !a.own_first) asm volatile("griddepcontrol.wait;" ::: "memory");
  TileInfo first;
  if (a.own_first) first = first_tile(a, *reinterpret_cast<FirstScratch*>(smem_slab), tail->heads[0]);

  // Tiles are handed out in list order through a device-wide cursor (the GEMM-O rows are sorted
  // longest first, the GEMM-Q list ends with its half-size tiles), so that a CTA that finishes early
  // takes the next tile instead of idling at the end of a fixed share. Tile i < gridDim.x goes to CTA i; the cursor counts the tiles after those.
  // Entry k of a CTA's sequence travels through slot k % kTileQ.
  auto read_slot = [&](int k) -> TileInfo {  // one thread of a consumer role; a_row -1 ends the sequence, -2 when the wait gave up
    const int slot = k % kTileQ;
    TileInfo ti;
    ti.a_row = -2; ti.w_row0 = ti.nkb = 0; ti.w_row1 = -1; ti.heads = nullptr;
    if (!mbar_wait(&tail->tq_full[slot], static_cast<uint32_t>(k / kTileQ) & 1u, abort_flag)) return ti;
    const int4 rec = tail->tile_q[slot];
    mbar_arrive(&tail->tq_empty[slot]);
    ti.a_row = rec.x; ti.w_row0 = rec.y; ti.w_row1 = rec.z; ti.nkb = rec.w;
    return ti;
  };

  if (warp == 4) {
    // ------------------------------------------------------------- TMA producer
    // All lanes stage the tile's head list in shared memory (one coalesced read instead of one
    // dependent global load per K block); lane 0 then issues the copies.
    // The head list of tile i+1 is fetched into registers while lane 0 feeds tile i, so that the
    // dependent global loads (row order -> row indptr -> heads) never sit between two tiles.
    int stage = 0;
    uint32_t phase = 0;
    int ok = 1;
    int hreg[kMaxHeadsSmem / 32];
    auto fetch_heads = [&](const TileInfo& ti) {
      if (ti.heads == nullptr) return;
      const int nh = ti.nkb / a.kb_per_head;
#pragma unroll
      for (int i = 0; i < kMaxHeadsSmem / 32; ++i) hreg[i] = (lane + 32 * i < nh && nh <= kMaxHeadsSmem) ? ti.heads[lane + 32 * i] : 0;
    };
    auto stash_heads = [&](int par) {
#pragma unroll
      for (int i = 0; i < kMaxHeadsSmem / 32; ++i) tail->heads[par][lane + 32 * i] = hreg[i];
    };
    int n_pub = 0;  // entries published so far (lane 0)
    auto publish = [&](const TileInfo& ti) -> bool {  // lane 0
      const int slot = n_pub % kTileQ;
      if (!mbar_wait(&tail->tq_empty[slot], (static_cast<uint32_t>(n_pub / kTileQ) & 1u) ^ 1u, abort_flag)) return false;
      tail->tile_q[slot] = make_int4(ti.a_row, ti.w_row0, ti.w_row1, ti.nkb);
      mbar_arrive(&tail->tq_full[slot]);
      ++n_pub;
      return true;
    };
    int n_tiles = 0, n_drawn = 0;
    auto draw = [&]() -> int {  // lane 0: the next tile of the device-wide sequence
      // equal tiles (dense: no cursor) keep the fixed round-robin share and skip the atomic
      ++n_drawn;
      const int t = a.cursor != nullptr ? atomicAdd(a.cursor, 1) + static_cast<int>(gridDim.x)
                                        : static_cast<int>(blockIdx.x) + n_drawn * static_cast<int>(gridDim.x);
      return t < n_tiles ? t : -1;
    };
    TileInfo none;
    none.a_row = -1; none.w_row0 = none.nkb = 0; none.w_row1 = -1; none.heads = nullptr;
    // `cur` is being loaded, t_n1 is known, t_n2 is drawn while `cur` runs, so that the atomic's round trip never sits
    // between two tiles. The next tile's record goes to the other roles before the rest of `cur` is loaded.
    TileInfo cur = none;
    int t_n1 = -1;
    if (a.own_first) {
      cur = first;
    } else {
      n_tiles = num_tiles(a);
      if (static_cast<int>(blockIdx.x) < n_tiles) cur = get_tile(a, static_cast<int>(blockIdx.x));
    }
    if (lane == 0) ok = publish(cur) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!a.own_first && cur.a_row >= 0) {
      fetch_heads(cur);
      stash_heads(0);
    }
    __syncwarp();
    bool is_first = true;
    bool list_due = a.own_first != 0;   // the list is still to be waited for
    int par = 0;
    while (cur.a_row >= 0 && ok) {
      TileInfo ti = cur;
      if (ti.heads != nullptr && ti.nkb / a.kb_per_head <= kMaxHeadsSmem) ti.heads = tail->heads[par];
      // K columns are generated without divisions: (head list entry, K block inside the head)
      int hh = 0, sub = 0;
      int kcol = (ti.heads != nullptr && ti.nkb > 0) ? ti.heads[0] * a.kb_per_head * kBK : 0;
      auto load = [&](int j0, int j1) {   // lane 0
        const uint32_t bytes = ti.w_row1 >= 0 ? kStageBytes : (kABytes + kBHalfBytes);
        for (int j = j0; j < j1; ++j) {
          if (!mbar_wait(&tail->empty[stage], phase ^ 1u, abort_flag)) { ok = 0; break; }
          uint8_t* sa = smem + stage * kStageBytes;
          mbar_expect_tx(&tail->full[stage], bytes);
          tma_load_2d(sa, &a.tmap_a, &tail->full[stage], kcol, ti.a_row);
          tma_load_2d(sa + kABytes, &a.tmap_b, &tail->full[stage], kcol, ti.w_row0);
          if (ti.w_row1 >= 0)
            tma_load_2d(sa + kABytes + kBHalfBytes, &a.tmap_b, &tail->full[stage], kcol, ti.w_row1);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
          // next K block
          if (ti.heads == nullptr) {
            kcol += kBK;
          } else if (++sub < a.kb_per_head) {
            kcol += kBK;
          } else {
            sub = 0;
            ++hh;
            if (j + 1 < ti.nkb) kcol = ti.heads[hh] * a.kb_per_head * kBK;
          }
        }
      };
      int head = 0;   // K blocks loaded before the next tile is looked up
      if (is_first) {
        head = ti.nkb < kStages ? ti.nkb : kStages;
        if (lane == 0) load(0, head);
        __syncwarp();
        is_first = false;
        if (list_due) {
          asm volatile("griddepcontrol.wait;" ::: "memory");
          list_due = false;
          n_tiles = num_tiles(a);
        }
        if (lane == 0) t_n1 = draw();
      }
      t_n1 = __shfl_sync(0xffffffffu, t_n1, 0);
      int t_n2 = -1;
      if (lane == 0 && t_n1 >= 0) t_n2 = draw();
      TileInfo nxt = none;
      if (t_n1 >= 0) {
        nxt = get_tile(a, t_n1);
        fetch_heads(nxt);
      }
      if (lane == 0) {
        if (ok && !publish(nxt)) ok = 0;
        if (ok) load(head, ti.nkb);
      }
      __syncwarp();
      if (t_n1 >= 0) stash_heads(par ^ 1);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      stage = __shfl_sync(0xffffffffu, stage, 0);
      phase = __shfl_sync(0xffffffffu, phase, 0);
      t_n1 = t_n2;
      cur = nxt;
      par ^= 1;
      __syncwarp();
    }
    if (list_due) asm volatile("griddepcontrol.wait;" ::: "memory");
  } else if (warp == 5) {
    // ------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc256 = make_idesc_f16(kBM, 2 * kBNH, kBf16, 0, 0);
      constexpr uint32_t idesc128 = make_idesc_f16(kBM, kBNH, kBf16, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      // every operand tile is K-major with 128-byte swizzle: same descriptor high word, low word = address
      const uint64_t desc0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint32_t desc_hi = static_cast<uint32_t>(desc0 >> 32), desc_lo0 = static_cast<uint32_t>(desc0);
      for (int k_seq = 0; ok; ++k_seq) {
        const TileInfo ti = read_slot(k_seq);
        if (ti.a_row < 0) break;
        const uint32_t idesc = ti.w_row1 >= 0 ? idesc256 : idesc128;
        if (!mbar_wait(&tail->acc_empty[acc], acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * 2 * kBNH);
        for (int j = 0; j < ti.nkb; ++j) {
          if (!mbar_wait(&tail->full[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          // descriptor low words of the 4 K = 16 steps (advancing 32 bytes inside the swizzle atom = +2)
          const uint32_t a_lo = desc_lo0 + static_cast<uint32_t>((stage * kStageBytes) >> 4);
          const uint32_t b_lo = a_lo + static_cast<uint32_t>(kABytes >> 4);
          const uint32_t la[4] = {a_lo, a_lo + 2u, a_lo + 4u, a_lo + 6u};
          const uint32_t lb[4] = {b_lo, b_lo + 2u, b_lo + 4u, b_lo + 6u};
          umma_ss_x4(d_tmem, desc_hi, desc_hi, idesc, j != 0 ? 1u : 0u, la, lb);
          umma_commit(&tail->empty[stage]);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(&tail->acc_full[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (kCache && warp == 6) {
    // ------------------------------------------------------------- loader of init slabs, in the epilogue's order
    if (lane == 0) {
      uint32_t count = 0;
      for (int k_seq = 0;; ++k_seq) {
        const TileInfo ti = read_slot(k_seq);
        if (ti.a_row < 0) break;
        const int nslab = ti.w_row1 >= 0 ? 2 * kSlabsPerBlock : kSlabsPerBlock;
        bool ok = true;
        for (int s = 0; s < nslab && ok; ++s, ++count) {
          const uint32_t buf = count % kSlabBufs;
          ok = mbar_wait(&tail->slab_empty[buf], ((count / kSlabBufs) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&tail->slab_full[buf], kSlabBytes);
          tma_load_2d(smem_slab + buf * kSlabBytes, &a.tmap_c, &tail->slab_full[buf],
                      (s < kSlabsPerBlock ? ti.w_row0 : ti.w_row1) + (s % kSlabsPerBlock) * kSlabCols, ti.a_row);
        }
        if (!ok) break;
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue warps 0..3
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t slab_count = 0;  // slabs handed to TMA stores so far (selects the staging buffer)
    const uint16_t* init16 = reinterpret_cast<const uint16_t*>(a.init);
    const int r_in_tile = warp * 32 + lane;
    // 16-byte pieces of a row of the slab: the 128-byte swizzle of 64 columns, the 64-byte one of 32
    constexpr int kPieces = kSlabCols / 8;
    const uint32_t swz = static_cast<uint32_t>(kCache ? (r_in_tile >> 1) & 3 : r_in_tile & 7);
    auto read_slot_warp = [&](int k) -> TileInfo {  // lane 0 reads, the warp shares the record
      TileInfo ti;
      ti.a_row = ti.w_row0 = ti.w_row1 = ti.nkb = 0; ti.heads = nullptr;
      if (lane == 0) ti = read_slot(k);
      ti.a_row = __shfl_sync(0xffffffffu, ti.a_row, 0);
      ti.w_row0 = __shfl_sync(0xffffffffu, ti.w_row0, 0);
      ti.w_row1 = __shfl_sync(0xffffffffu, ti.w_row1, 0);
      ti.nkb = __shfl_sync(0xffffffffu, ti.nkb, 0);
      return ti;
    };
    // The four warps leave this loop together: every round ends in a vote (two CTA-local barriers around one
    // shared word), so a wait that ran out in one warp can never leave the others behind at `epi_bar`.
    for (int k_seq = 0;; ++k_seq) {
      const TileInfo ti = read_slot_warp(k_seq);
      const int t_this = ti.a_row;
      bool fail = t_this == -2;
      const int nslab = ti.w_row1 >= 0 ? 2 * kSlabsPerBlock : kSlabsPerBlock;
      // init values of slab 0 are fetched before the accumulator is waited for
      uint4 initv[kPieces];
      auto load_init = [&](int s) {
        const int col0 = (s < kSlabsPerBlock ? ti.w_row0 : ti.w_row1) + (s % kSlabsPerBlock) * kSlabCols;
        if constexpr (!kCache) {
          if (a.init_mode == kInitBias1D) {
            const uint4* p = reinterpret_cast<const uint4*>(init16 + col0);
#pragma unroll
            for (int i = 0; i < kPieces; ++i) initv[i] = __ldg(p + i);
          }
        }
      };
      if (t_this >= 0) {
        load_init(0);
        if (!mbar_wait_warp(&tail->acc_full[acc], acc_phase, abort_flag)) fail = true;
      }
      if (fail && lane == 0) *abort_flag = 1;
      epi_bar();
      if (threadIdx.x == 0) tail->epi_go = (*abort_flag == 0) ? 1 : 0;
      epi_bar();
      if (tail->epi_go == 0 || t_this < 0) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(acc * 2 * kBNH);
#pragma unroll 1
      for (int s = 0; s < nslab; ++s) {
        const int col0 = (s < kSlabsPerBlock ? ti.w_row0 : ti.w_row1) + (s % kSlabsPerBlock) * kSlabCols;
        uint32_t v[kSlabCols];
        if (ti.nkb > 0) {
          tmem_ld_x32(taddr + static_cast<uint32_t>(s * kSlabCols), v);
          if constexpr (kSlabCols == 64) tmem_ld_x32(taddr + static_cast<uint32_t>(s * kSlabCols + 32), v + 32);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < kSlabCols; ++i) v[i] = 0u;
        }
        if (s == nslab - 1) {  // accumulator fully read: hand it back to the MMA warp
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tail->acc_empty[acc]);
        }
        uint8_t* buf = smem_slab + (slab_count % kSlabBufs) * kSlabBytes;
        uint8_t* rowp = buf + r_in_tile * kSlabCols * 2;
        bool ok = true;
        if constexpr (kCache) {  // this thread's row of the slab
          ok = mbar_wait_all(&tail->slab_full[slab_count % kSlabBufs], (slab_count / kSlabBufs) & 1u, abort_flag);
#pragma unroll
          for (int c = 0; c < kPieces; ++c) initv[c] = *reinterpret_cast<const uint4*>(rowp + ((static_cast<uint32_t>(c) ^ swz) << 4));
        }
        uint4 outv[kPieces];
        uint32_t* o32 = reinterpret_cast<uint32_t*>(outv);
        const uint32_t* a32 = reinterpret_cast<const uint32_t*>(initv);
#pragma unroll
        for (int i = 0; i < kSlabCols / 2; ++i) {
          float lo = __uint_as_float(v[2 * i]);
          float hi = __uint_as_float(v[2 * i + 1]);
          if (kCache || a.init_mode != kInitNone) {
            if (kBf16) {
              lo += __uint_as_float(a32[i] << 16);
              hi += __uint_as_float(a32[i] & 0xFFFF0000u);
            } else {
              const __half2 h2 = *reinterpret_cast<const __half2*>(&a32[i]);
              lo += __low2float(h2);
              hi += __high2float(h2);
            }
          }
          o32[i] = kBf16 ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
        }
        if constexpr (!kCache) {
          if (s + 1 < nslab) load_init(s + 1);  // next slab's init loads fly during the store hand-off
          // staging buffer of this slab must no longer be read by the store issued two slabs ago
          if (threadIdx.x == 0) tma_store_wait_read<1>();
          epi_bar();
        }
#pragma unroll
        for (int c = 0; c < kPieces; ++c)
          *reinterpret_cast<uint4*>(rowp + ((static_cast<uint32_t>(c) ^ swz) << 4)) = outv[c];
        fence_proxy_async_smem();
        epi_bar();
        if (threadIdx.x == 0) {
          if (ok) tma_store_2d(&a.tmap_y, buf, col0, ti.a_row);
          tma_store_commit();
          if constexpr (kCache) {  // the slab before this one has been read: its buffer takes the next init values
            tma_store_wait_read<1>();
            if (slab_count > 0u) mbar_arrive(&tail->slab_empty[(slab_count - 1u) % kSlabBufs]);
          }
        }
        ++slab_count;
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (threadIdx.x == 0) tma_store_wait_all<0>();
  }

  // ------------------------------------------------------------- common exit
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    // give copies that may still be in flight time to land before the CTA's smem is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    if (threadIdx.x == 0) atomicExch(a.status, kDevWaitTimeout);
    __syncthreads();
  }
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  // the last CTA to get here puts the tile cursor (and its own arrival count, the word after it) back to zero,
  // so the next launch over the same workspace needs no reset in between
  if (threadIdx.x == 0 && a.cursor != nullptr) {
    __threadfence();
    if (atomicAdd(a.cursor + 1, 1) == static_cast<int>(gridDim.x) - 1) {
      atomicExch(a.cursor, 0);
      atomicExch(a.cursor + 1, 0);
    }
  }
}

}  // namespace


cudaError_t launch_gemm(const GemmArgs& a, int max_ctas, cudaStream_t stream) {
  // Without a tile list (GEMM-O, dense): when even the single 128 x 128 tiles fit the CTAs in one round, they are the
  // tiles. A pair tile moves 25 % fewer operand bytes per FLOP, which is what counts once the SMs are full, but here it
  // would leave half of them idle and take twice the MMAs and the epilogue on the others. GEMM-O kernel
  // on a B200, 24 heads of 128: 24, 96 and 144 single tiles 24.3, 22.9 and 23.3 us, as 12, 48 and 72 pairs 29.3, 27.8 and 28.2
  // us; dense with K = 1024: 10.9-11.8 against 12.8-13.3 us. With one tile more than CTAs a second round would cost
  // more than that.
  GemmArgs g = a;
  const bool listed = a.mode == kGemmQ && a.tiles != nullptr;
  const int blocks = a.batch * (a.m / kBM) * (a.n / kBNH);
  g.single = !listed && blocks <= max_ctas ? 1 : 0;
  const int cap = listed || g.single ? blocks : a.batch * (a.m / kBM) * ((a.n / kBNH + 1) / 2);
  if (cap <= 0) return cudaSuccess;
  const int grid = cap < max_ctas ? cap : max_ctas;
  const bool cache = a.init_mode == kInitFull;
  const int rows = a.batch * (a.m / kBM);
  g.own_first = a.after_list && rows <= kFirstRows &&
                (listed ? a.list.head_dim == kBNH && a.n / kBNH <= 64 && a.list.is_full == 0 : a.list.k / a.list.head_dim <= 64);
  const auto kernel = a.is_bf16 ? (cache ? gemm_kernel<true, true> : gemm_kernel<true, false>)
                                : (cache ? gemm_kernel<false, true> : gemm_kernel<false, false>);
  static std::atomic<uint64_t> done[4] = {{0}, {0}, {0}, {0}};
  const cudaError_t e = allow_smem(kernel, kSmemBytes, done[(a.is_bf16 ? 1 : 0) + (cache ? 2 : 0)]);
  if (e != cudaSuccess) return e;
  return launch_dependent(kernel, grid, threads_of(cache), kSmemBytes, stream, g.after_list != 0, g);
}

}  // namespace fo
