// What the backward kernels with query blocks of 128 rows have in common: the walk over the blocks, and on pairs of CTAs the tail of a walk.
#pragma once
#include "fa2_params.h"
#include "sm100_ptx.cuh"

namespace fa2 {
namespace {

constexpr int kBlk = 128;  // keys per CTA and query rows per iteration
constexpr float kLog2e = 1.4426950408889634f;

// Query blocks [m_start, m_start + n_m) whose rows can see one of `keys` keys from n0 on.
__device__ __forceinline__ void q_block_range(const BwdParams& p, int sq, int sk, int n0, int keys, int& m_start, int& n_m) {
  int q_lo = 0, q_hi = sq;  // [q_lo, q_hi)
  const int off = sk - sq;
  const int n_last = min(n0 + keys - 1, sk - 1);
  if (p.window_right >= 0) q_lo = max(0, n0 - off - p.window_right);
  if (p.window_left >= 0) q_hi = min(sq, n_last - off + p.window_left + 1);
  m_start = q_lo / kBlk;
  n_m = (q_hi > q_lo) ? ((q_hi + kBlk - 1) / kBlk - m_start) : 0;
}

// Position of an iteration in the CTA's walk over (query head of the GQA group, query block), advanced
// without integer divisions: iteration it is head g = it / n_m of the group, query block m_start + it % n_m.
struct Walk {
  int g, mi;
};
__device__ __forceinline__ Walk walk_next(Walk w, int n_m) {
  if (++w.mi == n_m) {
    w.mi = 0;
    ++w.g;
  }
  return w;
}

// What a pair of CTAs works on: 2 * kBlk or kBlk keys of one (batch, kv head) and the query blocks that see them.
struct PairTile {
  int b, hk, n0;  // n0: first key of the pair
  int m_start, n_m, n_iter;
};

// A warp's part on pairs of CTAs: -LSE (log2 domain) and -delta of each query block of the walk. Rows past the sequence give P = 0. Two
// buffers, [lse, delta][kBlk] each: the next iteration's values are there before the compute warps ask for them.
__device__ __forceinline__ bool pair_statistics(const BwdParams& p, const PairTile& ti, float* s_stat, uint64_t* stat_full, uint64_t* stat_empty,
                                                int lane, const WaitCtl& ctl) {
  Walk w{0, 0};
  bool ok = ti.n_iter > 0;
  for (int it = 0; it < ti.n_iter && ok; ++it, w = walk_next(w, ti.n_m)) {
    const int hq = ti.hk * p.group + w.g, q0 = (ti.m_start + w.mi) * kBlk + lane;
    const float* lse = p.lse + ti.b * p.lse_batch_stride + hq * p.lse_head_stride;
    const float* delta = p.delta + ti.b * p.delta_batch_stride + hq * p.delta_head_stride;
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = q0 + 32 * i;
      v[i] = q < p.seqlen_q ? lse[q] * -kLog2e : -INFINITY;
      v[4 + i] = q < p.seqlen_q ? -delta[q] : 0.f;
    }
    const uint32_t buf = it & 1;
    ok = warp_wait(&stat_empty[buf], ((it >> 1) & 1) ^ 1, ctl, kWaitBwd + 15);
    float* stat = s_stat + buf * (2 * kBlk) + lane;
#pragma unroll
    for (int i = 0; i < 8; ++i) stat[32 * i] = v[i];
    __syncwarp();
    if (lane == 0) mbar_arrive(&stat_full[buf]);
  }
  return ok;
}

// The end of both kernels on pairs of CTAs, by all threads.
__device__ __forceinline__ void end_pair(const BwdParams& p, const volatile int* abort_flag, int tid, int warp, uint32_t tmem) {
  __syncwarp();
  if (*abort_flag) {
    // A wait ran out somewhere in this CTA: give MMAs, commits and copies in flight about a millisecond to land.
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0) report_abort(abort_flag, p.status);
  // A CTA stays until the other one has read its operands and sent it everything. The barrier takes converged warps.
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

}  // namespace
}  // namespace fa2
