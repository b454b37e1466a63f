// Internal declarations shared by the translation units of libflashomni_b200.so.
// Nothing in this header is part of the C ABI (see include/flashomni_b200.h for that).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "ptx.cuh"

namespace fo {

// Raises a kernel's limit of dynamic shared memory, once per kernel and device (the call costs about a microsecond).
template <class Kernel>
inline cudaError_t allow_smem(Kernel* kernel, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_relaxed) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

// Launches a kernel whose arguments struct is `args`; with `dependent` it may start while the kernel in front of it in the
// stream still runs (programmatic dependent launch): it must then wait (griddepcontrol.wait) before it touches memory.
template <class Args>
inline cudaError_t launch_dependent(void (*kernel)(Args), int grid, int threads, size_t smem, cudaStream_t stream, bool dependent,
                                    const Args& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

// ------------------------------------------------------------------ mask path
struct CompactArgs {
  const uint8_t* sparse_info;
  const uint8_t* sparse_kv_info;
  const int32_t* info_indptr;      // byte offsets per request
  const int32_t* kv_info_indptr;   // byte offsets per request
  const int32_t* qo_indptr;        // token offsets per request
  const int32_t* kv_indptr;
  int64_t info_bytes;              // readable bytes of sparse_info
  int64_t kv_info_bytes;           // readable bytes of sparse_kv_info
  int batch, num_heads, head_begin, head_count, sbq, sbkv, is_full;
  int max_nkv;                     // upper bound of kv-blocks per request (histogram size - 1)
  int64_t n_cand;                  // sum_b nq(b) * head_count
  int64_t max_items, max_kept;     // capacities of the output lists
  // outputs
  int32_t* items;                  // [max_items, 4] (b, h, qb, n_kept)
  int32_t* kv_ptr;                 // [max_items + 1]
  int32_t* kv_idx;                 // [max_kept]
  int32_t* order;                  // [max_items]
  int32_t* counters;               // [4]: n_items, total_kept, status, max_nkv
  // scratch
  int32_t* cnt;                    // [n_cand]
  int32_t* item_pos;               // [n_cand]
  long long* kv_off;               // [n_cand]
  int32_t* hist;                   // [max_nkv + 1]
};

struct GemmListArgs {
  const uint8_t* sparse_info;
  const int32_t* info_indptr;
  int64_t info_bytes;
  int batch, m, n, k, num_heads, head_begin, head_dim, sparse_q_size, num_text_tokens;
  int is_full, is_for_cache;
  int32_t* tiles;                  // GEMM-Q: [max_tiles, 4] pair records (b, iy, ix0, ix1)
  int max_tiles;
  int n_ctas;                      // CTAs of the GEMM launch that will draw the records (GEMM-Q list rule)
  int32_t* row_indptr;             // GEMM-O: [rows + 1]
  int32_t* row_heads;              // GEMM-O: [rows * local_heads]
  int32_t* row_order;              // GEMM-O: [rows]
  int32_t* counters;               // [4]
};

cudaError_t launch_packbits(const uint8_t* x, int64_t n, int little, uint8_t* y, cudaStream_t stream);
cudaError_t launch_segment_packbits(const uint8_t* x, const int32_t* indptr, const int32_t* new_indptr,
                                    int num_segments, int64_t out_bytes, int little, uint8_t* y,
                                    cudaStream_t stream);
int segment_packbits_sized_blocks(int64_t capacity);
// every_block: each block writes the total to its own word when it is done (else block 0 to words[0])
cudaError_t launch_segment_packbits_sized(const uint8_t* x, int64_t n, const void* indptr, int indptr_is_64, int num_segments,
                                          int64_t capacity, int little, uint8_t* y, int32_t* new_indptr, long long* words,
                                          int every_block, cudaStream_t stream);
cudaError_t launch_attn_compact(const CompactArgs& a, cudaStream_t stream);

struct UnitArgs {
  const int32_t* items;      // [max_items, 4] as written by the compaction
  const int32_t* kv_ptr;     // [max_items + 1]
  const int32_t* kv_idx;
  const int32_t* order;      // [max_items]
  const int32_t* counters;   // the compaction's counters (n_items, total_kept, status, max_nkv)
  const int32_t* qo_indptr;
  const int32_t* kv_indptr;
  int64_t max_items, max_units, max_slots;
  int min_items, num_streams, min_chunk, max_nkv, sbq, sbkv;
  int32_t* units;            // [max_units, 8]
  int32_t* unit_counters;    // [4]: n_units, partial slots in use, chunk_max, status
  int32_t* arrive;           // [max_slots]
};
cudaError_t launch_attn_units(const UnitArgs& a, cudaStream_t stream);
struct ZeroLater {           // output rows of inactive q-blocks that the list builder only lists, for the attention kernel (rec null: none)
  int2* rec;                 // [n_cand] (first row in the output, valid rows << 16 | head inside the tensors)
  int32_t* count;
};
struct CastArgs {            // fp8 K and V to cast in the same launch (src null: none)
  const uint8_t* src[2];
  uint16_t* dst[2];
  int64_t n;                 // values of each
  int e5m2, is_bf16;
};
struct ZeroArgs {            // output rows of inactive q-blocks that the list builder zeroes (out null: none)
  uint8_t* out;              // first byte of token 0, first head of the mask window
  int64_t token_bytes;       // bytes between tokens
  int head_bytes;            // contiguous bytes of one token that belong to one mask head, a multiple of 16
};
bool attn_lists_small_fits(const CompactArgs& a, const UnitArgs& u);
bool attn_lists_small_applies(const CompactArgs& a, const UnitArgs& u, const ZeroArgs& z);
cudaError_t launch_attn_lists_small(const CompactArgs& a, const UnitArgs& u, const ZeroArgs& z, const ZeroLater& later,
                                    const CastArgs& cast, cudaStream_t stream);
// src1 / dst1: a second tensor of the same size, or null
cudaError_t launch_cast_fp8(const void* src0, const void* src1, int64_t n, int e5m2, int is_bf16, void* dst0, void* dst1,
                            int sm_count, cudaStream_t stream);
// the lists of a layer step in one launch (attn_lists_small_fits must hold)
cudaError_t launch_layer_lists(const CompactArgs& a, const UnitArgs& u, const GemmListArgs& q, const GemmListArgs& o,
                               cudaStream_t stream);
cudaError_t launch_gemm_q_tiles(const GemmListArgs& a, cudaStream_t stream);
cudaError_t launch_gemm_o_rows(const GemmListArgs& a, cudaStream_t stream);

// ------------------------------------------------------------------ GEMM
enum GemmMode : int { kGemmQ = 0, kGemmO = 1 };
enum GemmInit : int { kInitNone = 0, kInitBias1D = 1, kInitFull = 2 };

struct GemmArgs {
  CUtensorMap tmap_a;              // X as [batch*m, k], box 64 x 128, 128B swizzle
  CUtensorMap tmap_b;              // W as [n, k],       box 64 x 128, 128B swizzle
  CUtensorMap tmap_y;              // Y as [batch*m, n], box 64 x 128, 128B swizzle (TMA stores)
  CUtensorMap tmap_c;              // kInitFull: init as [batch*m, n]; it and Y with a box of 32 x 128, 64B swizzle
  CUtensorMap tmap_b64;            // W with a box of 64 x 64 (the 192-column tiles of gemm_tall.cu)
  void* y;                         // [batch, m, n]
  const void* init;                // bias [n] or cache [batch, m, n] or null
  int init_mode;
  int mode;
  int is_bf16;
  int batch, m, n, k;
  int kb_per_head;                 // GEMM-O: head_dim / 64
  const int32_t* tiles;            // GEMM-Q pair records (b, iy, ix0, ix1); null = every tile (dense)
  const int32_t* n_tiles_ptr;      // device count of GEMM-Q tiles
  const int32_t* row_indptr;       // GEMM-O lists
  const int32_t* row_heads;
  const int32_t* row_order;
  int32_t* status;                 // device status word (DevStatus)
  int32_t* cursor;                 // device-wide tile cursor, zero when the kernel starts
  int single;                      // no tile list: tiles of one column block instead of two (set by launch_gemm)
  int after_list;                  // the launch in front of this one builds the list (dependent launch)
  int own_first;                   // a CTA finds its first tile in the mask itself (set by launch_gemm); needs `list`
  GemmListArgs list;               // after_list: what that launch got
};
cudaError_t launch_gemm(const GemmArgs& a, int max_ctas, cudaStream_t stream);
// dense projections whose shape divides into 256x256 tiles take the tall-tile kernel (gemm_tall.cu)
bool gemm_tall_applies(const GemmArgs& a, int sm_count);
int tall_tile_cols(const GemmArgs& a, int sm_count);   // 256, 192 or 0 (not applicable)
cudaError_t launch_gemm_tall(const GemmArgs& a, int max_ctas, cudaStream_t stream);

// ------------------------------------------------------------------ block selection
struct SelectArgs {
  const float* score;        // [batch, heads, n, n]
  const float* q_thr;        // [batch], or null: q_thr_all for every request
  const float* kv_thr;       // [heads], or null: kv_thr_all for every head
  float q_thr_all, kv_thr_all;
  int batch, heads, n, t2t, zero_inactive;
  int64_t info_seg_bytes;    // ceil(n * heads / 8)
  int64_t kv_seg_bytes;      // ceil(n * heads * n / 8)
  int64_t kv_words;          // 32-bit words of sparse_kv_info (zeroed by the first launch)
  uint8_t* sparse_info;
  uint8_t* sparse_kv_info;
  int32_t* info_indptr;      // [batch + 1]
  int32_t* kv_info_indptr;   // [batch + 1]
  uint8_t* q_keep;           // scratch [batch, n]
};
cudaError_t launch_select_blocks(const SelectArgs& a, cudaStream_t stream);

// ------------------------------------------------------------------ strided gather (exchange)
constexpr int kMaxGatherSources = 16;
struct GatherArgs {
  const uint8_t* src[kMaxGatherSources];
  uint8_t* dst[kMaxGatherSources];
  int64_t src_stride[kMaxGatherSources];   // bytes between rows
  int64_t dst_stride[kMaxGatherSources];
  int64_t vec_prefix[kMaxGatherSources + 1];  // exclusive prefix of rows * row_vecs
  int64_t row_vecs;                         // 16-byte vectors per row
  int n_src;
};
cudaError_t launch_strided_gather(const GatherArgs& a, int sm_count, cudaStream_t stream);

struct ReduceArgs {
  const uint8_t* src[kMaxGatherSources];   // partial results (peer pointers allowed), rows src_stride bytes apart
  const uint8_t* init;                      // optional addend (local), rows init_stride bytes apart
  uint8_t* dst;
  int64_t src_stride, init_stride, dst_stride;
  int64_t rows, row_vecs;                   // 16-byte vectors per row
  int n_src;
};
cudaError_t launch_reduce_rows(const ReduceArgs& a, int is_bf16, int sm_count, cudaStream_t stream);

constexpr int kMaxBarrierRanks = 64;
struct BarrierArgs {
  int* pads[kMaxBarrierRanks];   // every rank's flag pad as mapped into this process: int32 [channels][world]
  int* epoch;                    // this GPU's own epoch counters: int32 [channels]
  int* status;                   // device status word
  int rank, world, channel;
  uint64_t timeout_ns;
};
cudaError_t launch_peer_barrier(const BarrierArgs& a, cudaStream_t stream);

// ------------------------------------------------------------------ attention
struct AttnArgs {
  CUtensorMap tmap_q;              // [D, H, Tq]   box 64 x 1 x 128
  CUtensorMap tmap_k;              // [D, Hkv, Tkv]
  CUtensorMap tmap_v;
  CUtensorMap tmap_o;              // [D, Hq, Tq], stores of whole q-blocks: box 64 x 1 x 32, 128-byte swizzle (streams kernel)
                                   // or 32 x 1 x 16, no swizzle (the other one)
  void* o;                         // [Tq, H, D] (strides below, in elements)
  float* lse;                      // [Tq, H] or null
  int64_t o_stride_n, o_stride_h;
  int64_t lse_stride_n;
  const int32_t* kv_idx;           // kept kv-block indices; unit records point into it
  const int32_t* units;            // 8 words per unit (see attn_units_kernel), processing order
  const int32_t* unit_counters;    // n_units, partial slots in use, chunk_max, status
  int max_units;                   // capacity of the unit list
  int32_t* arrive;                 // per partial slot (a split item counts at its first slot): parts delivered; zero between launches
  float* partials;                 // partial results of split items: partial_slots x kPartialFloats floats
  int partial_slots;
  int head_dim;                    // 128 or 64
  int mask_mode;                   // 0: none; 1: causal (kv position <= q token + kv_len - q_len); 2: custom bit mask
  const uint8_t* custom_mask;      // mode 2: per request a [q_len, kv_len] bit matrix, row-major, little-endian bits
  int64_t custom_mask_bytes;
  const int32_t* mask_indptr;      // mode 2: byte offset of each request's matrix [batch + 1]
  const int32_t* qo_indptr;        // mode 2: request rows and lengths
  const int32_t* kv_indptr;
  int head_begin;                  // tensor head = item head - head_begin
  int group_size;                  // H / Hkv
  int is_bf16;
  float sm_scale_log2;             // sm_scale * log2(e); with a soft cap: cap * log2(e)
  int after_lists;                 // the launch in front of this one builds the lists (dependent launch)
  const int2* zero_rec;            // q-blocks to zero (ZeroLater), or null; streams kernel only
  const int32_t* zero_count;
  float soft_cap_pre;              // 0: no soft cap; else sm_scale / cap (logits = cap * tanh(q.k * sm_scale / cap))
  int32_t* status;
};
// floats of one partial result: O (32 column groups x 128 rows x 4), then the row maxima and the row sums
constexpr int kPartialFloats = 128 * 128 + 2 * 128;
// whole items without a causal or custom mask, head dimension 64 or 128: attention_streams.cu, which was faster at every
// shape measured (named there); the other launches keep attention.cu
inline bool attention_streams_applies(const AttnArgs& a) {
  return a.mask_mode == 0 && a.partial_slots <= 0 && (a.head_dim == 64 || a.head_dim == 128);
}
cudaError_t launch_attention_streams(const AttnArgs& a, int max_ctas, cudaStream_t stream);
cudaError_t launch_attention(const AttnArgs& a, int max_ctas, cudaStream_t stream);

// ------------------------------------------------------------------ host helpers
// Encodes a tiled tensor map (bf16/f16 elements; swizzle of 128 or 64 bytes, or 0 for none). dims/strides innermost first;
// strides in bytes for dims 1..rank-1. Returns 0 on success.
int encode_tmap_16bit(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box, int swizzle = 128);

}  // namespace fo
