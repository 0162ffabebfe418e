// The walk over the query blocks of the backward kernels for head dims up to 128.
#pragma once
#include "fa2_params.h"

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

}  // namespace
}  // namespace fa2
