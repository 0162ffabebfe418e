// Kernel-side parameter blocks shared by the host launchers and the sm_100a kernels.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace fa2 {

// Error codes a kernel leaves in its status word when a bounded wait runs out.
enum WaitSite : int {
  kWaitNone = 0,
  kWaitLoadQEmpty = 11,
  kWaitLoadKVEmpty = 12,
  kWaitMmaQFull = 21,
  kWaitMmaKVFull = 22,
  kWaitMmaPFull = 23,
  kWaitMmaOFree = 24,
  kWaitMmaSFree = 25,
  kWaitSoftmaxSFull = 31,
  kWaitSoftmaxPvDone = 32,
  kWaitSoftmaxExchange = 33,
  kWaitEpiFinal = 41,
  kWaitEpiPvDone = 42,
  kWaitBwd = 50,
  kWaitDecode = 80,
  kWaitBwdDq = 90,
};

constexpr int kMaxStreamBlocks = 64;   // 256-row query blocks of a head in a forward that shares tiles between CTAs

struct FwdParams {
  CUtensorMap tm_q, tm_k, tm_v, tm_o;  // 4-D maps: (D, heads, rows, batch), box (64, 1, 128, 1)
  void* o_ptr;                         // for the predicated (non-TMA) output path
  float* lse_ptr;
  const int32_t* cu_q;                 // packed (varlen) mode when non-null
  const int32_t* cu_k;
  const float* alibi;                  // [H] or [B,H] slopes, or null
  int64_t o_row_stride, o_head_stride, o_batch_stride;  // elements
  int64_t lse_head_stride, lse_batch_stride;            // elements
  int alibi_batch_stride;
  int batch, heads, heads_k, seqlen_q, seqlen_k;        // seqlen_* = maxima in packed mode
  int group;                           // heads / heads_k
  int num_mblk;                        // ceil(seqlen_q / 256)
  int num_tiles;                       // num_mblk * batch * heads
  int window_left, window_right;       // normalised; < 0 = open side
  int causal_alibi;                    // causal ALiBi depends on the key position only
  float scale;                         // softmax scale (applied before softcap / mask)
  float scale_log2;                    // scale * log2(e)
  float softcap;                       // 0 = off
  int* status;                         // device status word (0 = ok)
  int head_dim;                         // real head dim (<= the kernel's D; columns beyond it are padding)
  // Tiles shared between CTAs (null = none): the (work tile, key block) pairs of all heads form one list, which is cut
  // into equal shares. A share's part of a tile that it does not cover alone goes to slot 2 * CTA (+ 1 if the part has
  // the tile's first key block): O of [256 rows][D] fp32, unnormalised, then the rows' maxima and sums.
  float* parts;
  int stream_grid;                      // CTAs
  int units_per_head;                   // = block_start[num_mblk]
  uint16_t block_start[kMaxStreamBlocks + 1];  // units of a head before query block m
};
__host__ __device__ constexpr int64_t stream_slot_floats(int d) { return 256 * (static_cast<int64_t>(d) + 2); }

// Forward for few query rows (fwd_decode_sm100.cu). A unit is one (batch, kv head): its rows are the query rows of all
// the group's heads, row r = query r / group, head r % group.
constexpr int kDecodeMaxRows = 64;
constexpr int decode_row_tiles(int rows) { return rows <= 16 ? 1 : rows <= 32 ? 2 : 4; }  // 16-row tiles of a unit's kernel
struct DecodeParams {
  CUtensorMap tm_k, tm_v;              // box (64, 1, 128, 1)
  const void* q_ptr;
  void* o_ptr;
  float* lse_ptr;
  const float* alibi;
  float* partials;                     // 2 slots per CTA (null when no unit is split)
  unsigned long long* flags;           // one per partial slot: launch_tag once the part is in memory
  unsigned long long launch_tag;
  int64_t q_row_stride, q_head_stride, q_batch_stride;  // elements
  int64_t o_row_stride, o_head_stride, o_batch_stride;
  int64_t lse_head_stride, lse_batch_stride;
  int alibi_batch_stride;
  int units, heads_k, group, rows;     // rows = seqlen_q * group
  int tiles_per_unit, tile_lo;         // 128-key tiles [tile_lo, tile_lo + tiles_per_unit) hold every visible key
  int seqlen_k, off;                   // off = seqlen_k - seqlen_q
  int full_lo, full_hi;                // every row sees all of the keys [full_lo, full_hi)
  int window_left, window_right, causal_alibi;
  float scale, scale_log2, softcap;
  int head_dim;
  int* status;
};

constexpr int kMaxSplitBlocks = 160;   // a grid of more key blocks fills the GPU by itself

struct BwdParams {
  // Boxes as in fa2_launch.h where a kernel has others.
  CUtensorMap tm_q, tm_k, tm_v, tm_do;  // 16-bit inputs, box (64, 1, 128, 1)
  CUtensorMap tm_dk, tm_dv;             // 16-bit outputs, box (64, 1, 128, 1)
  CUtensorMap tm_dqa;                   // fp32 dQ accumulator, box (32, 1, 32, 1): one drain warp's rows
  const float* lse;
  const float* delta;
  void* dk_ptr;
  void* dv_ptr;
  const int32_t* cu_q;
  const int32_t* cu_k;
  int64_t lse_head_stride, lse_batch_stride;
  int64_t delta_head_stride, delta_batch_stride;
  int64_t dkv_row_stride, dkv_head_stride, dkv_batch_stride;  // elements
  int delta_seq_pad;                    // 128 in packed mode (sequence b starts at cu_q[b] + 128 b), else 0
  int batch, heads, heads_k, group, seqlen_q, seqlen_k;
  int num_nblk;                         // ceil(seqlen_k / 128)
  int head_group;                       // (batch, kv head) pairs whose key blocks are listed together, heaviest first
  int window_left, window_right;
  int which;                            // bit 0: dQ, bit 1: dK and dV
  float scale, scale_log2;
  int* status;
  // Score transforms of the forward that the gradients have to follow (null / 0 when unused).
  const float* alibi;                   // [heads] or [batch, heads] slopes
  int alibi_batch_stride;
  int causal_alibi;                     // bias = slope * key index instead of -slope * |distance|
  float softcap;                        // scores = softcap * tanh(raw * scale / softcap)
  int head_dim;                         // real head dim (<= the kernel's D; columns beyond it are padding)
  // Split key blocks (null = none): the walk over (query head, query block) of key block n is shared by
  // part_start[n + 1] - part_start[n] CTAs, each of which leaves its fp32 dK and dV in a slot of its own,
  // dk_part + part * part_stride in the layout of dK; a block with one part is written as usual.
  float* dk_part;
  float* dv_part;
  int64_t part_stride;                  // elements
  int items_per_head;                   // part_start[num_nblk]
  uint16_t part_start[kMaxSplitBlocks + 1];
  // Ordered dQ accumulation (null = arrival order). dq_turn[((batch * heads + head) * num_mblk_q + query
  // block) * 4 + drain warp] counts the key blocks whose adds into those 32 rows have landed; it is
  // zero at launch. A CTA adds only when the count equals the number of higher key blocks that add into the
  // same rows, so every element is summed in descending key-block order and dQ is bit-reproducible.
  int* dq_turn;
  int num_mblk_q;                       // ceil(seqlen_q / 128)
  // The kernel for head dims above 128 adds into the accumulator with plain reductions:
  // dq_acc[((batch * dq_rows + row) * heads + head) * head_dim + d], dq_rows rows per batch entry.
  float* dq_acc;
  int64_t dq_rows;
  // That kernel reads V row by row from global memory (it keeps V in TMEM): element strides of [batch, row, head].
  const void* v_ptr;
  int64_t v_batch_stride, v_row_stride, v_head_stride;
};

// dQ alone, dense, head dims up to 128 (bwd_dq_sm100.cu).
struct DqParams {
  CUtensorMap tm_q, tm_k, tm_v, tm_do, tm_dq;  // box (64, 1, 128, 1)
  const float* lse;
  const float* delta;
  const float* alibi;
  int64_t lse_head_stride, lse_batch_stride;
  int64_t delta_head_stride, delta_batch_stride;
  int alibi_batch_stride, causal_alibi;
  int batch, heads, group, seqlen_q, seqlen_k;
  int num_mblk;                         // ceil(seqlen_q / 128)
  int head_group;                       // (batch, head) pairs whose query blocks are listed together, heaviest first
  int window_left, window_right;
  float scale, scale_log2, softcap;
  int head_dim;
  int* status;
};

// What is left after the main backward kernel: dQ = 16-bit(scale * accumulator), and the sum of the parts of split key
// blocks, dK (scaled) and dV as 16-bit.
struct FinishParams {
  const float* dq_acc;                  // null: no dQ
  void* dq;
  int64_t n_dq;                         // elements, a multiple of 8
  const float* dk_part;                 // null: no split key blocks
  const float* dv_part;
  void* dk;
  void* dv;
  int64_t part_stride;
  int batch, rows, row_elems;           // dK and dV are [batch][rows][row_elems]
  float scale;
  int bf16;
  uint16_t part_start[kMaxSplitBlocks + 1];
};

struct PreprocessParams {
  float* zero_acc;                      // dense: clears the fp32 [batch, seqlen_q, heads, head_dim] accumulator too (or null)
  const void* dout;
  const void* out;
  float* delta;
  const int32_t* cu_q;
  int64_t do_batch_stride, do_row_stride, do_head_stride;
  int64_t o_batch_stride, o_row_stride, o_head_stride;
  int64_t delta_head_stride, delta_batch_stride;
  int batch, heads, seqlen_q, seqlen_pad, head_dim;
  int bf16;
};

}  // namespace fa2
