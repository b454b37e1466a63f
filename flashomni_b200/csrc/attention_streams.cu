// Block-sparse prefill attention, two independent streams of kv blocks per SM (tcgen05 / TMEM / TMA).
//
// Same result and same work lists as attention.cu (reference: include/flashomni/attention/prefill.cuh:1203-1531); this is
// the kernel of every launch of whole items without a causal or custom mask at head dimension 64 and 128. Every CTA walks
// its units as one sequence of kv blocks g = 0, 1, 2, ...; block g belongs to stream g & 1, and each stream has its own S
// (fp32, 128 TMEM columns, its P is written over it), its own O (fp32, 128 columns), its own running maximum and row sum.
// Nothing passes between the two streams until the end of a unit, where the epilogue adds the two O, each scaled to the
// common maximum.
//
//   issuer of a stream    QK(0) | PV(0) QK(1) | PV(1) QK(2) | ...      one batch of 16 MMAs, one commit
//   softmax of a stream   S -> registers (one q row per thread) -> maximum -> P = exp2 -> TMEM
//
// The MMAs of one thread execute in order: QK(i) may write over the P that PV(i - 1) reads, and the commit behind QK(i) also
// says that PV(i - 1) is done and that the stream's K and V slots are free.
//
// What bounds it: the chain of one stream, S visible -> P complete -> PV and QK -> next S visible, during which the other
// stream has the tensor pipe; on long launches the power cap (1.44 GHz instead of 1.77). By a clock trace of a step (one
// block on each stream, 3 300 clocks): loads and maximum 450, exponentials 1 300 (1 160 in a loop of their own, 1 024 at the
// MUFU's rate), P handed over to MMAs issued 150, sixteen MMAs 1 040, their completion seen by the softmax 250-300. What the
// structure was tuned by, us of a call on a B200, 4608 tokens, 24 heads of 128, density 0.5 / all blocks, back to back:
//   attention.cu (two groups of eight softmax warps on alternate blocks of one O, running maximum passed on)     111 / 266
//   one issuer thread for both streams (its waits and commits fall between the batches)                          117 / 300
//   an issuer per stream, batches as they come (both streams end up in phase)                                    122 / 313
//   batches in turns                                                                                             111 / 264
//   + half of P handed over early, conversions and sums some pairs behind the exponentials                       108 / 258
//   + next unit's record and Q fetched ahead, O read out in full before it is stored (this kernel)               107 / 256
//   a quarter (an eighth) of the exponentials as polynomials on the FMA pipe                                     112 / 275 (- / 265)
//   P handed over after three quarters (a quarter) instead of half                                               109 / 263 (109 / 258)
//   each stream with units of its own instead of alternate blocks of one unit                                    125 / 261
// Other shapes, device time of a call from a graph, attention.cu -> here: one request of 4608 tokens with 12 heads 76 -> 68, at
// density 0.2 67 -> 59; 32 requests of 256 tokens 60 -> 50, 8 of 1024 118 -> 108; 64 requests of 128 tokens 59.5 -> 50.8, of 100
// 55.4 -> 46.8, of 77 50.8 -> 45.6, of 33 46.6 -> 43.1, of 20 46.0 -> 43.9. Rows of a slab that is not whole leave from the thread
// that has them: staged like the others, four rows an instruction, 64 requests of 77 / 33 / 20 tokens took 55.8 / 53.8 / 50.5.
//
// Warps: 0-3 softmax stream 0, 4-7 softmax stream 1 (TMEM lane = q row), 8-11 epilogue, 12 TMA producer and drawer of
// work-list positions, 13 and 14 MMA issuers, 15 writes the q-blocks without work.
// Every mbarrier wait is bounded. A wait that runs out may do so for some lanes of a warp only: the softmax and epilogue warps go
// on together to a vote and leave there, the former behind the block, the latter before anything is stored.
#include <cuda_fp16.h>

#include "internal.h"

namespace fo {
namespace {

constexpr int kBQ = 128, kBKV = 128;
constexpr int kTileBytes = 128 * 128 * 2;   // slot of a 128-row tile of Q, K or V (head dimension 64 fills half of it)
constexpr int kHalfBytes = kTileBytes / 2;  // one 64-column half (one swizzle-atom column)
constexpr int kQBufs = 2;
constexpr int kRing = 4;
constexpr int kStreamWarps = 4;
constexpr int kSoftmaxWarps = 2 * kStreamWarps;
constexpr int kWarpEpilogue = kSoftmaxWarps;      // first of four (TMEM lane quadrant = warp % 4)
constexpr int kEpilogueWarps = 4;
constexpr int kWarpProducer = kWarpEpilogue + kEpilogueWarps;
constexpr int kWarpMma = kWarpProducer + 1;
constexpr int kWarpZero = kWarpMma + 2;
constexpr int kThreads = (kWarpZero + 1) * 32;   // 512
// setmaxnreg split. The 60 bytes that are spilled at head dimension 128 are descriptor words of the issuers (14.6 local loads of one
// warp per kv block); 184 / 88 / 56 gave the epilogue too few: image layer 95.2 us instead of 94.5, 64 requests of 90 / 20 tokens 51.5 /
// 47.8 instead of 47.5 / 43.9 (device time of a call from a graph).
constexpr int kRegsSoftmax = 168, kRegsEpilogue = 120, kRegsOther = 56;
// setmaxnreg.inc waits until the registers are free in the pool the CTA was launched with: a split that asks for more
// never returns.
constexpr int kRegsAtLaunch = (65536 / kThreads) / 8 * 8;
static_assert(kSoftmaxWarps * 32 * kRegsSoftmax + kEpilogueWarps * 32 * kRegsEpilogue + 4 * 32 * kRegsOther <= kThreads * kRegsAtLaunch,
              "register split exceeds the CTA's register pool");
constexpr int kTmemCols = 512;
constexpr uint32_t kColS = 0, kColO = 256;  // stream s: + 128 s
constexpr int kRotStep = 5;                 // q-block qb starts its kv list at entry (qb * kRotStep) mod length
constexpr int kItemQ = 8;
constexpr int kItemReaders = kSoftmaxWarps + kEpilogueWarps + 2;  // softmax and epilogue warps, the two issuers
constexpr int kEarly = 4;                   // MMAs of a PV (16 kv rows each) that may start before the whole P is there
constexpr int kLag = 4;                     // pairs of columns between an exponential and its use
constexpr float kRescaleThreshold = 8.0f;   // lazy rescale: keep the old maximum while exp2 stays <= 2^8

struct Tail {
  uint64_t q_full[kQBufs], q_empty[kQBufs];
  uint64_t full[kRing];            // K of stream 0, K of stream 1, V of stream 0, V of stream 1
  uint64_t batch[2];               // a stream's batch of MMAs (PV of block i - 1, QK of block i) is done
  uint64_t p_most[2], p_full[2];   // the first kEarly * 16 columns of a stream's P are in TMEM (and O is rescaled); all of them
  uint64_t turn[2];                // a stream's issuer may issue its next batch
  uint64_t stats_ready[2];         // indexed by unit parity: both streams have published (m, l)
  uint64_t stats_free[2];          // the epilogue has read them
  uint64_t o_full[2];              // the last PV of a unit on a stream is done
  uint64_t o_free[2];              // the epilogue has read a stream's O
  uint64_t iq_full[kItemQ], iq_empty[kItemQ];  // unit queue: the producer draws work-list positions for the CTA
  int4 item_q[kItemQ][2];          // the units' records; no kv blocks: the end
  uint32_t tmem_base;
  int abort_flag;
  float stats_m[2][2][128];        // [unit parity][stream][row]: the maximum the sum refers to
  float stats_l[2][2][128];
};

constexpr int kOutSlabBytes = 32 * 128;            // 32 rows x 64 output columns: staging of an epilogue warp
constexpr int kSmemBytes = (kQBufs + kRing) * kTileBytes + kEpilogueWarps * kOutSlabBytes + 1024 + static_cast<int>(sizeof(Tail));
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ int rot_of(int qb, int n) {
  return static_cast<int>(static_cast<unsigned>(qb * kRotStep) % static_cast<unsigned>(n));
}

// Work-list positions: position i < gridDim.x goes to CTA i, the following ones are drawn from a device-wide cursor by
// the producer. It passes the records of the units that have kv blocks on to the other roles through a small shared-memory
// queue; units without any never enter it, so that no role ever walks past several entries in one go. The producer
// publishes unit u + 1 when the first blocks of unit u are on their way, at most seven units ahead of the epilogue, and a
// reader asks for a unit only when it is done with the one before: asked for a unit ahead, the issuers stood still for 4 000
// clocks at the start of every unit (32 requests of 256 tokens 54 us instead of 51, 16 of 512 tokens 72.7 instead of 67.7).
struct ItemDraw {
  Tail* tail;
  int32_t* cursor;
  volatile int* abort_flag;
  int n_items, n_pub, ahead;  // `ahead` is drawn (and in flight) while the position in front of it is looked at
  __device__ __forceinline__ int draw() {
    const int p = atomicAdd(cursor, 1) + static_cast<int>(gridDim.x);
    return p < n_items ? p : -1;
  }
  __device__ __forceinline__ void init(Tail* t, int32_t* cur, volatile int* ab, int n) {
    tail = t; cursor = cur; abort_flag = ab; n_items = n; n_pub = 0;
    ahead = static_cast<int>(blockIdx.x) < n ? static_cast<int>(blockIdx.x) : -1;
  }
  __device__ __forceinline__ int next() {  // the next position, published or not
    const int p = ahead;
    if (p >= 0) ahead = draw();
    return p;
  }
  __device__ __forceinline__ bool publish(const int4& u0, const int4& u1) {
    const int slot = n_pub % kItemQ;
    if (!mbar_wait(&tail->iq_empty[slot], (static_cast<uint32_t>(n_pub / kItemQ) & 1u) ^ 1u, abort_flag)) return false;
    tail->item_q[slot][0] = u0;
    tail->item_q[slot][1] = u1;
    mbar_arrive(&tail->iq_full[slot]);
    ++n_pub;
    return true;
  }
};

template <bool kWholeWarp>
struct ItemRead {  // the reading roles: one thread, or all lanes of a warp
  Tail* tail;
  volatile int* abort_flag;
  int k;
  __device__ __forceinline__ void init(Tail* t, volatile int* ab) { tail = t; abort_flag = ab; k = 0; }
  __device__ __forceinline__ bool next(int4& u0, int4& u1) {  // false at the end
    const int slot = k % kItemQ;
    const uint32_t phase = static_cast<uint32_t>(k / kItemQ) & 1u;
    if (!(kWholeWarp ? mbar_wait_all(&tail->iq_full[slot], phase, abort_flag) : mbar_wait(&tail->iq_full[slot], phase, abort_flag))) return false;
    u0 = tail->item_q[slot][0];
    u1 = tail->item_q[slot][1];
    if (kWholeWarp) {
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(&tail->iq_empty[slot]);
    } else {
      mbar_arrive(&tail->iq_empty[slot]);
    }
    ++k;
    return u0.x > 0;
  }
};

// Waits for the TMEM loads issued so far; naming the 32 registers keeps their uses behind the wait.
__device__ __forceinline__ void tmem_wait_ld_32(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
template <bool kBf16, bool kSoftCap, int kD>
__global__ void __launch_bounds__(kThreads, 1) attention_streams_kernel(const __grid_constant__ AttnArgs a) {
  static_assert(kD == 128 || kD == 64, "head dimension");
  constexpr int kLoadBytes = 128 * kD * 2;   // bytes of one tile load
  constexpr int kHalves = kD / 64;           // 64-column boxes per tile
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* smem_q = smem;
  uint8_t* smem_ring = smem + kQBufs * kTileBytes;
  uint8_t* smem_stage = smem_ring + kRing * kTileBytes;
  Tail* tail = reinterpret_cast<Tail*>(smem_stage + kEpilogueWarps * kOutSlabBytes);
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // uniform: role state in uniform registers
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kQBufs; ++i) { mbar_init(&tail->q_full[i], 1); mbar_init(&tail->q_empty[i], 2); }
    for (int i = 0; i < kRing; ++i) mbar_init(&tail->full[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tail->batch[i], 1);
      mbar_init(&tail->o_full[i], 1);
      mbar_init(&tail->o_free[i], kEpilogueWarps);
      mbar_init(&tail->p_most[i], kStreamWarps);
      mbar_init(&tail->p_full[i], kStreamWarps);
      mbar_init(&tail->turn[i], 1);
      mbar_init(&tail->stats_ready[i], kSoftmaxWarps);
      mbar_init(&tail->stats_free[i], kEpilogueWarps);
    }
    for (int i = 0; i < kItemQ; ++i) { mbar_init(&tail->iq_full[i], 1); mbar_init(&tail->iq_empty[i], kItemReaders); }
    tail->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kWarpProducer && lane == 0) {
    tma_prefetch_desc(&a.tmap_q);
    tma_prefetch_desc(&a.tmap_k);
    tma_prefetch_desc(&a.tmap_v);
    tma_prefetch_desc(&a.tmap_o);
  }
  if (warp == kWarpMma) {
    tmem_alloc(&tail->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tail->tmem_base;
  if (a.after_lists) asm volatile("griddepcontrol.wait;" ::: "memory");  // launched while the lists in front of it were built

  // A list that ran out of room is not dereferenced; the launch only reports it. Parts of split lists are not for this kernel.
  const bool list_bad = a.unit_counters[3] != kDevOk || a.unit_counters[1] > 0;
  int n_items = a.unit_counters[0];
  if (list_bad || n_items < 0) n_items = 0;
  if (n_items > a.max_units) n_items = a.max_units;

  if (warp >= kWarpProducer) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
  if (warp == kWarpProducer) {
    // ------------------------------------------------------------------ TMA producer, in the order the issuers read
    if (lane == 0) {
      ItemDraw src;
      src.init(tail, a.status + 1, abort_flag, n_items);
      uint32_t g = 0;
      int unit_no = 0;
      int vh0 = 0, vrow0 = -1, vh1 = 0, vrow1 = -1;   // V tiles still to be loaded: of block g - 2 and of block g - 1
      bool ok = true;
      auto load = [&](uint32_t slot, const CUtensorMap* map, int h, int row) {
        uint8_t* dst = smem_ring + slot * kTileBytes;
        mbar_expect_tx(&tail->full[slot], kLoadBytes);
#pragma unroll
        for (int i = 0; i < kHalves; ++i) tma_load_3d(dst + i * kHalfBytes, map, &tail->full[slot], 64 * i, h, row);
      };
      // V of block b goes to slot 2 + (b & 1) once batch b >> 1 of its stream, which read the V before it, is done
      auto push_v = [&](uint32_t b, int h, int row) -> bool {
        if (!mbar_wait(&tail->batch[b & 1u], (b >> 1) & 1u, abort_flag)) return false;
        load(2u + (b & 1u), &a.tmap_v, h, row);
        return true;
      };
      // the record of the next unit, and the head of its kv list, are fetched while the current one is loaded: the chain
      // position -> record -> list entry would otherwise sit in front of every unit's first tiles
      bool q_pending = false;
      int n_next = 0, t_next = 0, kvb_first = 0, hk_next = 0, q_row_next = 0, kv_row_next = 0, kv_off_next = 0;
      auto take = [&](const int4& u0, const int4& u1) {   // a unit with kv blocks: the next one
        ok = src.publish(u0, u1);
        if (!ok) return;
        n_next = u0.x;
        kv_off_next = u0.y;
        hk_next = (u0.z & 0xffff) - a.head_begin;   // a unit's head is the kv head; its q tile holds the group's q heads
        q_row_next = u0.w;                          // of 128 / group tokens, token-major
        kv_row_next = u1.y;
        t_next = rot_of(q_row_next >> 7, n_next);
        kvb_first = a.kv_idx[kv_off_next + t_next];
        q_pending = true;
      };
      auto fetch = [&]() {
        n_next = 0;
        while (true) {
          const int pos = src.next();
          if (pos < 0) { ok = src.publish(make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)); return; }
          const int4* up = reinterpret_cast<const int4*>(a.units + 8 * static_cast<int64_t>(pos));
          const int4 u0 = up[0], u1 = up[1];
          if (u0.x <= 0) continue;   // (warp 15 writes its zeros)
          take(u0, u1);
          return;
        }
      };
      auto load_q = [&]() -> bool {  // of the unit fetched last
        const int qb = unit_no & 1;
        if (!mbar_wait(&tail->q_empty[qb], (static_cast<uint32_t>(unit_no >> 1) & 1u) ^ 1u, abort_flag)) return false;
        ++unit_no;
        uint8_t* dst = smem_q + qb * kTileBytes;
        mbar_expect_tx(&tail->q_full[qb], kLoadBytes);
#pragma unroll
        for (int i = 0; i < kHalves; ++i)
          tma_load_3d(dst + i * kHalfBytes, &a.tmap_q, &tail->q_full[qb], 64 * i, hk_next * a.group_size, q_row_next);
        q_pending = false;
        return true;
      };
      fetch();
      while (ok && n_next > 0) {
        const int n = n_next, hk = hk_next, kv_row0 = kv_row_next;
        const int32_t* kv = a.kv_idx + kv_off_next;
        int t = t_next;
        int kvb_next = kvb_first;
        for (int j = 0; j < n && ok; ++j) {
          const int kvb = kvb_next;
          if (j + 1 < n) {
            if (++t == n) t = 0;
            kvb_next = kv[t];
          }
          // (the wait of this V also frees the slot of the K below: both were read by batch (g - 2) >> 1 or before)
          if (vrow0 >= 0) ok = push_v(g - 2u, vh0, vrow0);
          vh0 = vh1; vrow0 = vrow1;
          if (ok && j == 0 && q_pending) ok = load_q();
          vh1 = hk; vrow1 = kv_row0 + kvb * kBKV;
          if (ok) load(g & 1u, &a.tmap_k, vh1, vrow1);
          ++g;
          // The next unit's Q comes from HBM: it is requested early, to the buffer of the unit before this one, whose last
          // QK has been issued by now (it is in front of this unit's second K, which is on its way).
          if (ok && j == (n > 1 ? 1 : 0)) {
            fetch();
            if (n > 1 && n_next > 0) ok = load_q();
          }
        }
      }
      if (ok && vrow0 >= 0) ok = push_v(g - 2u, vh0, vrow0);
      if (ok && vrow1 >= 0) push_v(g - 1u, vh1, vrow1);
    }
  } else if (warp == kWarpMma || warp == kWarpMma + 1) {
    // ------------------------------------------------------------------ MMA issuers, one per stream
    // Batch i of a stream is PV of its block i - 1 and QK of its block i, sixteen MMAs behind one set of waits and in front
    // of ONE commit: its completion says that S of block i is written, that the PV of block i - 1 is done (O may be
    // rescaled or read), and that the stream's K and V slots are free.
    if (lane == 0) {
      constexpr uint32_t idesc_qk = make_idesc_f16(kBQ, kBKV, kBf16, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_f16(kBQ, kD, kBf16, 0, 1);
      const uint32_t X = static_cast<uint32_t>(warp - kWarpMma);
      // descriptors: constant high words (128-byte swizzle; Q and K K-major, V MN-major with its two 64-column halves
      // 16 KB apart), low words hold the address
      const uint64_t dk = make_smem_desc_sw128(smem_u32(smem_ring + X * kTileBytes), 16, 1024);
      const uint64_t dv = make_smem_desc_sw128(smem_u32(smem_ring + (2u + X) * kTileBytes), kHalfBytes, 1024);
      const uint32_t hi_k = static_cast<uint32_t>(dk >> 32), hi_v = static_cast<uint32_t>(dv >> 32);
      const uint32_t q_lo0 = static_cast<uint32_t>(make_smem_desc_sw128(smem_u32(smem_q), 16, 1024));
      uint32_t lk[8], lv[8], tp[8];
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        // 16 elements further along K: +32 B inside a 64-column half, +16 KB for the second half; 16 kv rows further =
        // 16 * 128 B in the V tile, 8 columns further in the 16-bit P tile
        lk[kk] = static_cast<uint32_t>(dk) + static_cast<uint32_t>(((kk >> 2) * kHalfBytes + (kk & 3) * 32) >> 4);
        lv[kk] = static_cast<uint32_t>(dv) + static_cast<uint32_t>((kk * 2048) >> 4);
        tp[kk] = tmem_base + kColS + X * 128u + static_cast<uint32_t>(kk * 8);
      }
      const uint32_t tmem_s = tmem_base + kColS + X * 128u, tmem_o = tmem_base + kColO + X * 128u;
      ItemRead<false> src;
      src.init(tail, abort_flag);
      bool ok = true;
      int n = 0, j = 0, unit_no = -1;
      bool ended = false;
      uint32_t g0 = 0;      // blocks in front of the current unit
      uint32_t i = 0;       // this stream's batches so far
      uint32_t units_started = 0;
      uint32_t q_lo = 0;
      bool pv = false, pv_first = false;   // a PV is pending, and it is its unit's first one
      while (true) {
        // ---- the next block of this stream, if there is one
        j += 2;
        bool qk = true;
        bool new_unit = false;
        while (j >= n) {
          g0 += static_cast<uint32_t>(n);
          int4 u0, u1;   // (published while the unit before was loaded: no wait)
          n = ended || !src.next(u0, u1) ? 0 : u0.x;
          if (n == 0) { ended = true; qk = false; break; }
          ++unit_no;
          j = static_cast<int>((g0 ^ X) & 1u);
          new_unit = true;
          if (j >= n) {  // a unit of one block, and it is the other stream's: its Q tile is none of this stream's business
            if (!mbar_wait(&tail->q_full[unit_no & 1], static_cast<uint32_t>(unit_no >> 1) & 1u, abort_flag)) { ok = false; break; }
            mbar_arrive(&tail->q_empty[unit_no & 1]);
          }
        }
        if (!ok) break;
        if (!qk && !pv) {  // a stream that had no block at all still passes the turn on
          if (i == 0u) mbar_arrive(&tail->turn[X ^ 1u]);
          break;
        }
        // ---- everything the batch needs
        if (pv) {
          if (!mbar_wait(&tail->full[2u + X], (i - 1u) & 1u, abort_flag)) break;
          if (pv_first) {  // O must have been read by the epilogue of this stream's previous unit
            if (units_started > 0u && !mbar_wait(&tail->o_free[X], (units_started - 1u) & 1u, abort_flag)) break;
            ++units_started;
          }
          if (!mbar_wait(&tail->p_most[X], (i - 1u) & 1u, abort_flag)) break;
        }
        // the two streams' batches alternate: interleaved in the pipe both would end when the second one does now
        if ((X != 0u || i != 0u) && !mbar_wait_spin(&tail->turn[X], (i & 1u) ^ (X ^ 1u), abort_flag)) break;
        tc_fence_after_sync();
        if (pv) {
          static_assert(kEarly == 4, "the PV is issued in two halves");
          umma_ts_x4(tmem_o, hi_v, idesc_pv, pv_first ? 0u : 1u, tp, lv);
          if (!mbar_wait_spin(&tail->p_full[X], (i - 1u) & 1u, abort_flag)) break;
          tc_fence_after_sync();
          umma_ts_x4(tmem_o, hi_v, idesc_pv, 1u, tp + 4, lv + 4);
        }
        if (pv && (new_unit || !qk)) umma_commit(&tail->o_full[X]);  // O of the unit is complete
        if (qk) {
          if (new_unit) {
            if (!mbar_wait(&tail->q_full[unit_no & 1], static_cast<uint32_t>(unit_no >> 1) & 1u, abort_flag)) break;
            q_lo = q_lo0 + static_cast<uint32_t>(((unit_no & 1) * kTileBytes) >> 4);
          }
          if (!mbar_wait(&tail->full[X], i & 1u, abort_flag)) break;
          uint32_t la[8];
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) la[kk] = q_lo + static_cast<uint32_t>(((kk >> 2) * kHalfBytes + (kk & 3) * 32) >> 4);
          if constexpr (kD == 128) umma_ss_x8(tmem_s, hi_k, hi_k, idesc_qk, 0u, la, lk);
          else umma_ss_x4(tmem_s, hi_k, hi_k, idesc_qk, 0u, la, lk);
        }
        mbar_arrive(&tail->turn[X ^ 1u]);
        umma_commit(&tail->batch[X]);
        if (qk && j + 2 >= n) umma_commit(&tail->q_empty[unit_no & 1]);
        ++i;
        pv = qk;
        pv_first = new_unit;
      }
    }
  } else if (warp == kWarpZero) {
    // ------------------------------------------------------------------ q-blocks without any work, beside the others
    const int grp = a.group_size, grp_shift = 31 - __clz(grp);
    // rows of a q-block of kv head h, 16 bytes per lane and step
    auto zero_rows = [&](int row0, int rows, int h, bool write_lse) {
      for (int i = lane; i < rows * (kD / 8); i += 32) {
        const int r = i / (kD / 8);
        const int64_t tok = static_cast<int64_t>(row0) + (r >> grp_shift);
        const int hq = h * grp + (r & (grp - 1));
        uint16_t* orow = reinterpret_cast<uint16_t*>(a.o) + tok * a.o_stride_n + static_cast<int64_t>(hq) * a.o_stride_h;
        reinterpret_cast<uint4*>(orow)[i % (kD / 8)] = make_uint4(0u, 0u, 0u, 0u);
        if (write_lse && i % (kD / 8) == 0 && a.lse != nullptr) a.lse[tok * a.lse_stride_n + hq] = -5e4f;
      }
    };
    // Inactive q-blocks of an output that reads as zero there. Zeroed by the launch that builds the lists instead, they kept this
    // one waiting: image layer at density 0.5 (12 MB of them), lists 13.8 -> 9.7 us and the call 108.9 -> 106.1 us on a B200.
    if (a.zero_rec != nullptr) {
      const int n_zero = *a.zero_count;
      for (int i = static_cast<int>(blockIdx.x); i < n_zero; i += static_cast<int>(gridDim.x)) {
        const int2 rec = a.zero_rec[i];
        zero_rows(rec.x, (rec.y >> 16) * grp, rec.y & 0xffff, false);
      }
    }
    // Active ones that keep nothing: zeros and lse = -5e4. Every CTA looks at its share of the positions, whoever draws them.
    for (int base = static_cast<int>(blockIdx.x); base < n_items; base += 32 * static_cast<int>(gridDim.x)) {
      const int mine = base + lane * static_cast<int>(gridDim.x);
      uint32_t todo = __ballot_sync(0xffffffffu, mine < n_items && a.units[8 * static_cast<int64_t>(mine)] <= 0);
      for (; todo != 0u; todo &= todo - 1u) {
        const int pos = base + (__ffs(static_cast<int>(todo)) - 1) * static_cast<int>(gridDim.x);
        const int4* up = reinterpret_cast<const int4*>(a.units + 8 * static_cast<int64_t>(pos));
        const int4 u0 = up[0], u1 = up[1];
        zero_rows(u0.w, (u1.x & 0xffff) * grp, (u0.z & 0xffff) - a.head_begin, true);
      }
    }
  }
  } else if (warp >= kWarpEpilogue) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
    // ------------------------------------------------------------------ epilogue warps: (O0 w0 + O1 w1) / l to global memory
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t tmem_o = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + kColO;
    uint8_t* stg = smem_stage + quad * kOutSlabBytes;
    const int grp = a.group_size;
    const int grp_shift = 31 - __clz(grp);   // 1, 2, 4, 8 or 16 q heads share a kv head
    const int row_tok = row >> grp_shift, row_head = row & (grp - 1), row_tok0 = (quad * 32) >> grp_shift;
    uint32_t item = 0;
    uint32_t g = 0;         // blocks in front of the current unit
    uint32_t o_phase = 0;   // bit X: parity of the units so far that had blocks of stream X
    ItemRead<true> src;
    src.init(tail, abort_flag);
    while (true) {
      int4 u0, u1;
      if (!src.next(u0, u1)) break;
      const int q_row0 = u0.w, q_valid = u1.x & 0xffff, h = (u0.z & 0xffff) - a.head_begin;
      // Row r of a tile is token q_row0 + r / group, q head h * group + r % group (group = 1: the row itself).
      const bool row_ok = row < q_valid * grp;
      const int64_t grow = static_cast<int64_t>(q_row0) + row_tok;
      const int hq = h * grp + row_head;
      float* lse = a.lse != nullptr ? a.lse + grow * a.lse_stride_n + hq : nullptr;
      const uint32_t ip = item & 1u;
      bool got = mbar_wait(&tail->stats_ready[ip], (item >> 1) & 1u, abort_flag);
      // 0 and 1 are the streams of the unit's first and second block from here on: which of the two that is depends on the
      // units that this CTA drew before, the rounding of the sums must not
      const uint32_t f = g & 1u;
      const float m0 = tail->stats_m[ip][f][row], m1 = tail->stats_m[ip][f ^ 1u][row];
      const float l0 = tail->stats_l[ip][f][row], l1 = tail->stats_l[ip][f ^ 1u][row];
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->stats_free[ip]);
      const float m_out = fmaxf(m0, m1);
      // a stream without a visible column has m = -inf, l = 0
      const float w_min = exp2_series(fminf(m0, m1) - m_out);
      float w0 = (m0 == m_out) ? 1.f : w_min, w1 = (m1 == m_out) ? 1.f : w_min;
      const float l_out = m0 == m_out ? fmaf(l1, w1, l0) : fmaf(l0, w0, l1);   // (the other weight is 1: one rounding)
      const float inv_out = l_out > 0.f ? __frcp_rn(l_out) : 0.f;
      // A unit of one block leaves the other stream's O as it was, which may be anything: O of the stream with the block stands in
      // for it, with a weight that rounds away beside w0 (at least 2^-40) and, unlike zero, leaves an infinity one.
      const bool has1 = u0.x > 1;
      w0 *= inv_out;
      w1 = has1 ? w1 * inv_out : 0x1p-126f;
      g += static_cast<uint32_t>(u0.x);
      got = mbar_wait(&tail->o_full[f], (o_phase >> f) & 1u, abort_flag) && got;
      if (has1) got = mbar_wait(&tail->o_full[f ^ 1u], (o_phase >> (f ^ 1u)) & 1u, abort_flag) && got;
      if (!__all_sync(0xffffffffu, got)) break;
      o_phase ^= has1 ? 3u : 1u << f;
      tc_fence_after_sync();
      const int rows = q_valid * grp - quad * 32;   // rows of this warp that are not past the request: all from 32 on
      const bool whole = rows >= 32;
      const uint32_t tmem_o0 = tmem_o + 128u * f, tmem_o1 = has1 ? tmem_o + 128u * (f ^ 1u) : tmem_o0;
      const uint64_t w0p = pack_f32x2(w0, w0), w1p = pack_f32x2(w1, w1);
#pragma unroll 1
      for (int half = 0; half < kHalves; ++half) {
        uint4 out[8];
        uint32_t* w = reinterpret_cast<uint32_t*>(out);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t v0[16], v1[16];
          tmem_ld_x16(tmem_o0 + 64u * half + 16u * c, v0);
          tmem_ld_x16(tmem_o1 + 64u * half + 16u * c, v1);
          tmem_wait_ld();
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const uint64_t b2 = ffma2(pack_f32x2(__uint_as_float(v1[2 * t]), __uint_as_float(v1[2 * t + 1])), w1p, 0ull);
            const uint64_t x2 = ffma2(pack_f32x2(__uint_as_float(v0[2 * t]), __uint_as_float(v0[2 * t + 1])), w0p, b2);
            float x0, x1;
            unpack_f32x2(x2, x0, x1);
            w[8 * c + t] = kBf16 ? pack_bf16x2(x0, x1) : pack_f16x2(x0, x1);
          }
        }
        if (half == kHalves - 1) {  // both O may be overwritten by the next unit
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&tail->o_free[f]);
            if (has1) mbar_arrive(&tail->o_free[f ^ 1u]);
          }
        }
        if (whole) {
          // Through a staging slab per warp (32 rows x 64 columns in the 128-byte swizzle pattern) and one TMA store: a store
          // instruction of a warp would write 32 scattered 16-byte pieces.
          if (lane == 0) tma_store_wait_read<0>();  // the slab is free once the store before has read it
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) * 16)) = out[c];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&a.tmap_o, stg, 64 * half, h * grp, q_row0 + row_tok0);
            tma_store_commit();
          }
        } else if (row_ok) {  // rows past the request must not be written
          uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(a.o) + grow * a.o_stride_n +
                                                static_cast<int64_t>(hq) * a.o_stride_h + 64 * half);
#pragma unroll
          for (int c = 0; c < 8; ++c) dst[c] = out[c];
        }
      }
      ++item;
      if (row_ok && lse != nullptr) *lse = (l_out > 0.f) ? add_log2(m_out, l_out) : -5e4f;
    }
    if (lane == 0) tma_store_wait_all<0>();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    // ------------------------------------------------------------------ softmax: one q row per thread
    const uint32_t X = static_cast<uint32_t>(warp >> 2);
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_base + kColS + X * 128u;
    const uint32_t tmem_o = tmem_base + lane_base + kColO + X * 128u;
    uint64_t* s_full = &tail->batch[X];
    uint64_t* p_full = &tail->p_full[X];
    ItemRead<true> src;
    src.init(tail, abort_flag);
    uint32_t g = 0;          // blocks in front of the current unit
    uint32_t phase = 0;      // parity of this stream's block count
    uint32_t item = 0;
    bool ok = true;
    const uint64_t scale2 = pack_f32x2(a.sm_scale_log2, a.sm_scale_log2);

    int4 u0, u1;
    while (ok && src.next(u0, u1)) {
      const int n = u0.x, rag = u1.x >> 16;
      int ragged_j = -1;   // visiting step of the request's partial last kv block
      if (rag != 0) {
        ragged_j = n - 1 - rot_of(u0.w >> 7, n);
        if (ragged_j < 0) ragged_j += n;
      }
      float m_ref = -INFINITY;
      float l_sum = 0.f;
      const int j0 = static_cast<int>((g ^ X) & 1u);
#pragma unroll 1
      for (int j = j0; j < n; j += 2) {
        const bool got = mbar_wait(s_full, phase, abort_flag);
        phase ^= 1u;
        tc_fence_after_sync();
        uint32_t s[128];
        tmem_ld_x32(tmem_s, s);
        tmem_ld_x32(tmem_s + 32u, s + 32);
        tmem_wait_ld();
        tmem_ld_x32(tmem_s + 64u, s + 64);   // ... while the maximum of the first half is taken
        tmem_ld_x32(tmem_s + 96u, s + 96);
        const bool ragged = j == ragged_j;
        float mxs[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        auto half_max = [&](int c0) {
          if (ragged) {
#pragma unroll
            for (int c = c0; c < c0 + 64; c += 32) {
              const int have = rag - c;   // existing columns from here on: as a mask of 32 bits
              const uint32_t keep = have >= 32 ? 0xffffffffu : (have <= 0 ? 0u : (1u << have) - 1u);
#pragma unroll
              for (int t = 0; t < 32; ++t)
                if (((keep >> t) & 1u) == 0u) s[c + t] = 0xff800000u;  // -inf: exp2 gives 0
            }
          }
#pragma unroll
          for (int t = 0; t < 8; ++t) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              mxs[i] = fmax3(mxs[i], __uint_as_float(s[c0 + 8 * t + 2 * i]), __uint_as_float(s[c0 + 8 * t + 2 * i + 1]));
          }
        };
        half_max(0);
        tmem_wait_ld_32(s + 64);
        tmem_wait_ld_32(s + 96);
        half_max(64);
        float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3]));
        // with a soft cap the logit is cap * tanh(s * sm_scale / cap): monotonic, so the maximum is transformed once
        if constexpr (kSoftCap) mx = (mx == -INFINITY) ? mx : tanh_approx(mx * a.soft_cap_pre);
        const bool first = j < 2;
        const float m_prev = m_ref;
        const float m_new = fmaxf(m_prev, mx * a.sm_scale_log2);
        const bool need = (m_new - m_prev) > kRescaleThreshold;
        const bool rescale = !first && __any_sync(0xffffffffu, need);
        float alpha = 1.f;
        if (first) {
          m_ref = m_new;
        } else if (need) {
          m_ref = m_new;
          alpha = ex2_approx(m_prev - m_new);
          l_sum *= alpha;
        }
        const float neg_m = (m_ref == -INFINITY) ? 0.f : -m_ref;
        const uint64_t negm2 = pack_f32x2(neg_m, neg_m);
        if (rescale) {  // the PV of this stream's previous block is done: it is in the batch that wrote S
#pragma unroll 1
          for (int c = 0; c < kD / 16; ++c) {
            uint32_t v[16];
            tmem_ld_x16(tmem_o + 16u * c, v);
            tmem_wait_ld();
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = __float_as_uint(__uint_as_float(v[t]) * alpha);
            tmem_st_x16(tmem_o + 16u * c, v);
          }
        }
        if constexpr (kSoftCap) {
#pragma unroll
          for (int t = 0; t < 128; ++t)  // masked columns stay at -inf
            if (s[t] != 0xff800000u) s[t] = __float_as_uint(tanh_approx(__uint_as_float(s[t]) * a.soft_cap_pre));
        }
        auto hand_over = [&](uint64_t* bar) {
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar);
        };
        // The sum and the conversion of a pair follow its exponentials by kLag pairs: between two volatile TMEM stores
        // nothing then waits for the last exponential in front of it. A block is summed up for itself: added one by one to the
        // sum of all blocks, small values fall below its last bit (log-sum-exp of 9216 tokens, logits N(0, 4^2): rms error
        // against 64 bits 4.0e-6, here 2.3e-6, at the same time; with four accumulators 2.2e-6, and 1.5 % slower).
        uint64_t l2[2];
#pragma unroll
        for (int t = 0; t < 64 + kLag; ++t) {
          if (t < 64) {
            const uint64_t x2 = ffma2(pack_f32x2(__uint_as_float(s[2 * t]), __uint_as_float(s[2 * t + 1])), scale2, negm2);
            float x0, x1;
            unpack_f32x2(x2, x0, x1);
            s[2 * t] = __float_as_uint(ex2_approx(x0));
            s[2 * t + 1] = __float_as_uint(ex2_approx(x1));
          }
          if (t >= kLag) {
            const int e = t - kLag;
            const float p0 = __uint_as_float(s[2 * e]), p1 = __uint_as_float(s[2 * e + 1]);
            const uint64_t p2 = pack_f32x2(p0, p1);
            l2[e & 1] = e < 2 ? p2 : fadd2(l2[e & 1], p2);
            s[e] = kBf16 ? pack_bf16x2(p0, p1) : pack_f16x2(p0, p1);   // (entry e of s is free by now)
            if ((e & 15) == 15) {   // P over S: this thread has its whole row in registers
              tmem_st_x16(tmem_s + static_cast<uint32_t>(e - 15), s + e - 15);
            }
            // (a few pairs after the store, so that nothing waits for it)
            if (e == kEarly * 8 + 4) hand_over(&tail->p_most[X]);
          }
        }
        hand_over(p_full);
        float la, lb;
        unpack_f32x2(fadd2(l2[0], l2[1]), la, lb);
        l_sum += la + lb;
        ok = __all_sync(0xffffffffu, got);
        if (!ok) break;
      }
      if (!ok) break;
      g += static_cast<uint32_t>(n);
      const uint32_t ip = item & 1u;
      // the statistics of the unit before the last one must have been read
      if (item >= 2u && !mbar_wait_all(&tail->stats_free[ip], ((item >> 1) - 1u) & 1u, abort_flag)) break;
      tail->stats_m[ip][X][row] = m_ref;
      tail->stats_l[ip][X][row] = l_sum;
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->stats_ready[ip]);
      ++item;
    }
  }

  // ------------------------------------------------------------------ common exit
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    if (threadIdx.x == 0) atomicExch(a.status, kDevWaitTimeout);
    __syncthreads();
  }
  if (list_bad && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(a.status, kDevOk, kDevBadIndex);
  if (warp == kWarpMma) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  // the last CTA to get here puts the cursor and the arrival count back to zero for the next launch
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(a.status + 2, 1) == static_cast<int>(gridDim.x) - 1) {
      atomicExch(a.status + 1, 0);
      atomicExch(a.status + 2, 0);
    }
  }
}

template <bool kBf16, bool kSoftCap, int kD>
cudaError_t launch_one(const AttnArgs& a, int ctas, cudaStream_t stream) {
  static std::atomic<uint64_t> done{0};
  const cudaError_t e = allow_smem(attention_streams_kernel<kBf16, kSoftCap, kD>, kSmemBytes, done);
  if (e != cudaSuccess) return e;
  return launch_dependent(attention_streams_kernel<kBf16, kSoftCap, kD>, ctas, kThreads, kSmemBytes, stream,
                          a.after_lists != 0, a);
}
template <bool kBf16, bool kSoftCap>
cudaError_t launch_two(const AttnArgs& a, int ctas, cudaStream_t stream) {
  return a.head_dim == 64 ? launch_one<kBf16, kSoftCap, 64>(a, ctas, stream) : launch_one<kBf16, kSoftCap, 128>(a, ctas, stream);
}
}  // namespace

cudaError_t launch_attention_streams(const AttnArgs& a, int max_ctas, cudaStream_t stream) {
  if (max_ctas <= 0) return cudaSuccess;
  const bool cap = a.soft_cap_pre > 0.f;
  if (a.is_bf16) return cap ? launch_two<true, true>(a, max_ctas, stream) : launch_two<true, false>(a, max_ctas, stream);
  return cap ? launch_two<false, true>(a, max_ctas, stream) : launch_two<false, false>(a, max_ctas, stream);
}

}  // namespace fo
