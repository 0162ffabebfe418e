// Internal launch entry points of the sm_100a kernels (one translation unit per kernel family).
#pragma once
#include <cuda_runtime.h>
#include "fa2_params.h"

namespace fa2 {

// What happens to a score besides the scale, as a template argument of the kernels for head dims up to 128: one
// transform alone has code of its own, without a test per score for the other one. kScoreAny takes everything
// (both transforms; in the forward also a negative scale without a transform) and is what packed batches use.
enum ScoreMode : int { kScorePlain = 0, kScoreSoftcap = 1, kScoreAlibi = 2, kScoreAny = 3 };

// early: the kernel, which calls early_wait, may start while the kernel before it in the stream ends. Packed batches are launched
// the usual way, and let the next grid in when they end: the forward of a large packed batch, looped with other kernels, once
// ended in a launch failure that was never explained, and grids that overlap are one more thing that could have a part in it.
template <typename... P, typename... A>
cudaError_t launch_grid(bool early, void (*kernel)(P...), dim3 grid, int threads, size_t smem_bytes, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[1] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// Dense and packed (varlen) forward; head_dim is a multiple of 8 up to 128 (kernels for D = 64 and 128).
cudaError_t launch_fwd(const FwdParams& p, int head_dim, bool bf16, int num_sms, cudaStream_t stream);

// The same for head_dim a multiple of 8 in 136..256: one CTA per 128-row query block, 64-key tiles; p.tm_k and
// p.tm_v carry boxes of 64 rows.
cudaError_t launch_fwd_wide(const FwdParams& p, int head_dim, bool bf16, cudaStream_t stream);

// Dense forward with at most kDecodeMaxRows query rows per kv head, head_dim a multiple of 8 up to 256; `grid` CTAs
// share the tile list evenly. The workspace behind p.partials and p.flags holds 2 * grid partial results of
// 16 * decode_row_tiles(rows) rows x (D + 2) floats (D: head_dim rounded up to 64) and as many 8-byte flags.
// early: it may start beside the end of the kernel before it (decode_starts_early).
cudaError_t launch_fwd_decode(const DecodeParams& p, int grid, bool bf16, bool early, cudaStream_t stream);

// dQ / dK / dV for head_dim a multiple of 8 up to 128; the fp32 dQ accumulator behind p.tm_dqa (and the turn
// counters p.dq_turn, when given) must be zero.
cudaError_t launch_bwd(const BwdParams& p, int head_dim, bool bf16, int num_sms, cudaStream_t stream);

// The same on pairs of CTAs with 256 keys, for the calls of bwd_takes_pairs; p.tm_q and p.tm_do carry boxes of 64 rows.
cudaError_t launch_bwd_pair(const BwdParams& p, bool bf16, cudaStream_t stream);

// The same for head_dim a multiple of 8 in 136..256: one CTA per (128 keys, half of the head dim), query blocks of
// 64 rows; p.tm_q and p.tm_do carry boxes of 64 rows, dQ goes through p.dq_acc, dK and dV through p.dk_ptr / p.dv_ptr.
cudaError_t launch_bwd_wide(const BwdParams& p, int head_dim, bool bf16, cudaStream_t stream);

// Head dims 192 and 256, dense calls that want all three, on pairs of CTAs (bwd_wide_takes_pairs); the maps of Q, K, V and dO
// are those of make_atom_map, the ones of dK and dV have boxes of 64 rows, p.tm_dqa has boxes of 32 columns and 16 rows.
cudaError_t launch_bwd_wide_pair(const BwdParams& p, bool bf16, cudaStream_t stream);

// dQ alone, dense, head_dim a multiple of 8 up to 128: summed in key order, written as 16-bit.
cudaError_t launch_bwd_dq(const DqParams& p, bool bf16, cudaStream_t stream);

// delta = rowsum(dO * O) into the padded layouts (dense [B,H,Sq_pad], packed [H,total_q+128*B]).
cudaError_t launch_bwd_preprocess(const PreprocessParams& p, cudaStream_t stream);

// Copy of a 16-bit [n0, n1, n2, d] tensor (unit last stride) between two layouts given by their outer element strides.
cudaError_t launch_copy_rows(const void* src, void* dst, int64_t n0, int64_t n1, int64_t n2, int64_t d,
                             const int64_t src_strides[3], const int64_t dst_strides[3], cudaStream_t stream);
// The conversions after the main backward kernel, in one launch.
cudaError_t launch_bwd_finish(const FinishParams& p, cudaStream_t stream);

}  // namespace fa2
