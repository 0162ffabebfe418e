// dQ alone for sm_100a (B200), dense, head dims up to 128: the first half of a bit-reproducible backward call.
//
// One CTA owns 128 query rows of one (batch, head) and walks the key blocks that they can see, so dQ is summed in
// TMEM in key order: no accumulator in memory, no clearing, no conversion, no order to enforce between CTAs. (The
// combined kernel called for dQ alone added every 32-row slab of the fp32 accumulator in a fixed order of its key
// blocks, each CTA waiting for the one before it: 1.5 ms causal and 3.2 ms without a mask at B16 H16 S2048 D128,
// for products that take 0.3.)
//
//   S  = Q K^T      smem x smem -> TMEM [128 q x 128 keys], two buffers
//   dP = dO V^T     smem x smem -> TMEM
//   dS = exp2(S c - lse) (dP - delta)   compute warps, one query row per thread and half of the keys per warpgroup;
//                   16-bit, written back over S as the A operand of
//   dQ += dS K      TMEM x smem (K as an MN-major operand)
//
// Three products per tile pair, 1536 tensor cycles at D = 128; the exponentials take 1024 MUFU cycles next to them.
// Warps: 0-7 compute, 8 loader (TMA ring of five tiles: K(0) V(0) K(1) V(1) ...), 9 MMA issuer.
// The CTAs of a group of heads are listed together, heaviest first (bwd_dq_head_group), so the group's K and V stay in L2.
//
// Stands in for the reference's register-accumulating dQ kernel (flash-attn2-rs/src/device/backward/dq.rs:12-302).
#include "sm100_ptx.cuh"
#include "fa2_params.h"
#include "fa2_launch.h"

namespace fa2 {

namespace {

constexpr int kBlk = 128;
constexpr int kThreads = 384;
constexpr int kLoadWarp = 8;
constexpr int kMmaWarp = 9;
constexpr int kSlots = 5;
constexpr float kLog2e = 1.4426950408889634f;

template <int D>
struct DqCfg {
  static constexpr int kAtoms = D / 64;
  static constexpr int kTileBytes = kBlk * D * 2;
  static constexpr int kQOff = 0;
  static constexpr int kDOOff = kTileBytes;
  static constexpr int kRingOff = 2 * kTileBytes;
  static constexpr int kBarOff = kRingOff + kSlots * kTileBytes;
  static constexpr int kNumBars = 2 * kSlots + 9;
  static constexpr int kMiscOff = (kBarOff + kNumBars * 8 + 15) / 16 * 16;
  static constexpr int kSmemBytes = kMiscOff + 16;
  static constexpr uint32_t kTmemS = 0, kTmemDP = 256, kTmemDQ = 384;
};

template <int D, bool BF16, int MODE>
__global__ void __launch_bounds__(kThreads, 1) bwd_dq_kernel(const __grid_constant__ DqParams p) {
  using Cfg = DqCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    early_wait();
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, kWaitNone + 1);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOff);
  uint64_t* kv_full = bars;
  uint64_t* kv_empty = bars + kSlots;
  uint64_t* q_full = bars + 2 * kSlots;
  uint64_t* do_full = q_full + 1;
  uint64_t* s_full = q_full + 2;   // [2], one per S buffer
  uint64_t* dp_full = q_full + 4;
  uint64_t* dp_free = q_full + 5;  // dP has been read out of TMEM
  uint64_t* ds_full = q_full + 6;  // [2], one per S buffer
  uint64_t* dq_done = q_full + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const WaitCtl ctl{abort_flag};

  const int first_bh = static_cast<int>(blockIdx.x) / (p.head_group * p.num_mblk) * p.head_group;
  const int n_bh = min(p.head_group, p.batch * p.heads - first_bh);
  const int in_group = static_cast<int>(blockIdx.x) - first_bh * p.num_mblk;
  const int m_rev = in_group / n_bh;
  const int bh = first_bh + in_group - m_rev * n_bh;
  const int m0 = (p.num_mblk - 1 - m_rev) * kBlk;
  const int b = bh / p.heads, h = bh - b * p.heads, hk = h / p.group;
  const int off = p.seqlen_k - p.seqlen_q;
  // Key blocks [nb, ne) that some row of this block sees.
  int nb = 0, ne = 0;
  {
    const int r_hi = min(m0 + kBlk, p.seqlen_q) - 1;
    int hi = p.seqlen_k, lo = 0;
    if (p.window_right >= 0) hi = min(hi, r_hi + off + p.window_right + 1);
    if (p.window_left >= 0) lo = max(0, m0 + off - p.window_left);
    if (hi > lo) {
      nb = lo / kBlk;
      ne = (hi + kBlk - 1) / kBlk;
    }
  }
  const int n_iter = ne - nb;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < Cfg::kNumBars; ++i) {
      const bool compute_arrives = bars + i == dp_free || bars + i == ds_full || bars + i == ds_full + 1;
      mbar_init(bars + i, compute_arrives ? 256 : 1);
    }
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == kLoadWarp && lane == 0) {
    tma_prefetch_desc(&p.tm_q);
    tma_prefetch_desc(&p.tm_k);
    tma_prefetch_desc(&p.tm_do);
    tma_prefetch_desc(&p.tm_v);
  }
  tc_fence_before();
  early_wait();
  __syncthreads();
  tc_fence_after();
  early_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp < 8) {
    // ------------------------------------------------------------------ compute
    const int wg = warp >> 2;
    const int row_in = tid & 127;
    const int row = m0 + row_in;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float lse = INFINITY, delta = 0.f;  // rows past the end: P = 0
    if (row < p.seqlen_q) {
      lse = p.lse[b * p.lse_batch_stride + h * p.lse_head_stride + row] * kLog2e;
      delta = p.delta[b * p.delta_batch_stride + h * p.delta_head_stride + row];
    }
    const float slope = (MODE & kScoreAlibi) ? p.alibi[b * p.alibi_batch_stride + h] * kLog2e : 0.f;
    const float inv_cap = (MODE & kScoreSoftcap) ? p.scale / p.softcap : 0.f;
    const float cap_l2 = p.softcap * kLog2e;
    bool ok = true;
    for (int it = 0; it < n_iter; ++it) {
      const int buf = it & 1;
      const uint32_t t_s = tmem + lane_addr + Cfg::kTmemS + buf * kBlk + wg * 64;
      const uint32_t t_dp = tmem + lane_addr + Cfg::kTmemDP + wg * 64;
      const int col0 = (nb + it) * kBlk + wg * 64;
      if (!warp_wait(&s_full[buf], (it >> 1) & 1, ctl, kWaitBwdDq + 1)) { ok = false; break; }
      tc_fence_after();
      uint32_t sr[64];
      tmem_ld32(t_s, sr);
      tmem_ld32(t_s + 32, sr + 32);
      tmem_wait_ld();
      float pr[64];
      if constexpr (MODE == kScorePlain) {
#pragma unroll
        for (int i = 0; i < 64; ++i) pr[i] = ex2(fmaf(__uint_as_float(sr[i]), p.scale_log2, -lse));
      } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          float x, deriv = 1.f;
          if constexpr ((MODE & kScoreSoftcap) != 0) {
            const float t = tanh_approx(__uint_as_float(sr[i]) * inv_cap);
            x = cap_l2 * t;
            deriv = fmaf(-t, t, 1.f);
          } else {
            x = __uint_as_float(sr[i]) * p.scale_log2;
          }
          if constexpr ((MODE & kScoreAlibi) != 0) {
            const float key = static_cast<float>(col0 + i);
            x += p.causal_alibi ? slope * key : -slope * fabsf(static_cast<float>(row + off) - key);
          }
          pr[i] = ex2(x - lse) * deriv;
        }
      }
      const int tile0 = (nb + it) * kBlk;
      bool need_mask = tile0 + kBlk > p.seqlen_k;
      if (p.window_right >= 0) need_mask |= tile0 + kBlk - 1 > m0 + off + p.window_right;
      if (p.window_left >= 0) need_mask |= tile0 < m0 + kBlk - 1 + off - p.window_left;
      if (need_mask) {
        int hi = p.seqlen_k, lo = 0;
        if (p.window_right >= 0) hi = min(hi, row + off + p.window_right + 1);
        if (p.window_left >= 0) lo = row + off - p.window_left;
        hi -= col0;
        lo -= col0;
        fill_outside<64>(pr, lo, hi, 0.f);
      }
      if (!warp_wait(dp_full, it & 1, ctl, kWaitBwdDq + 2)) { ok = false; break; }
      tc_fence_after();
      tmem_ld32(t_dp, sr);
      tmem_ld32(t_dp + 32, sr + 32);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive(dp_free);
#pragma unroll
      for (int i = 0; i < 32; ++i)
        sr[i] = pack2<BF16>(pr[2 * i] * (__uint_as_float(sr[2 * i]) - delta), pr[2 * i + 1] * (__uint_as_float(sr[2 * i + 1]) - delta));
      tmem_st32(t_s, sr);  // each warpgroup writes into the columns that it has read itself
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&ds_full[buf]);
    }
    // ---- dQ * scale -> 16-bit -> the Q tile (its last reader has completed) -> TMA store; warpgroup wg takes half
    // of the columns
    if (ok && n_iter > 0) ok = warp_wait(dq_done, 0, ctl, kWaitBwdDq + 3);
    if (ok) {
      constexpr int kCols = D / 2;
      uint32_t acc[kCols];
      if (n_iter > 0) {
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < kCols / 32; ++c) tmem_ld32(tmem + lane_addr + Cfg::kTmemDQ + wg * kCols + c * 32, acc + c * 32);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < kCols; ++i) acc[i] = 0;
      }
#pragma unroll
      for (int c = 0; c < kCols / 8; ++c) {
        const int ch = wg * (kCols / 8) + c;  // 16-byte chunk of the row
        uint4 w;
        w.x = pack2<BF16>(__uint_as_float(acc[8 * c]) * p.scale, __uint_as_float(acc[8 * c + 1]) * p.scale);
        w.y = pack2<BF16>(__uint_as_float(acc[8 * c + 2]) * p.scale, __uint_as_float(acc[8 * c + 3]) * p.scale);
        w.z = pack2<BF16>(__uint_as_float(acc[8 * c + 4]) * p.scale, __uint_as_float(acc[8 * c + 5]) * p.scale);
        w.w = pack2<BF16>(__uint_as_float(acc[8 * c + 6]) * p.scale, __uint_as_float(acc[8 * c + 7]) * p.scale);
        *reinterpret_cast<uint4*>(smem + Cfg::kQOff + (ch / 8) * (kBlk * 128) + row_in * 128 + (((ch & 7) ^ (row_in & 7)) << 4)) = w;
      }
      fence_proxy_async_smem();
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (tid == 0 && ok) {
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a)
        if (a * 64 < p.head_dim) tma_store_4d(&p.tm_dq, smem + Cfg::kQOff + a * (kBlk * 128), a * 64, h, m0, b);
      tma_commit_group();
      tma_wait_group_read<0>();
    }
    __syncwarp();
  } else if (warp == kLoadWarp && elect_one()) {
    // ---------------------------------------------------------------- loader; it leaves last: it waits until the
    // issuer's commits on every ring slot have landed
    bool ok = true;
    uint32_t slot = 0, phase = 0;
    auto load = [&](const CUtensorMap* tm, int row) -> bool {
      if (!mbar_wait(&kv_empty[slot], phase ^ 1, ctl, kWaitBwdDq + 4)) return false;
      mbar_expect_tx(&kv_full[slot], Cfg::kTileBytes);
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a)
        tma_load_4d(smem + Cfg::kRingOff + slot * Cfg::kTileBytes + a * (kBlk * 128), tm, &kv_full[slot], a * 64, hk, row, b);
      if (++slot == kSlots) {
        slot = 0;
        phase ^= 1;
      }
      return true;
    };
    if (n_iter > 0) {
      mbar_expect_tx(q_full, Cfg::kTileBytes);
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a) tma_load_4d(smem + Cfg::kQOff + a * (kBlk * 128), &p.tm_q, q_full, a * 64, h, m0, b);
      load(&p.tm_k, nb * kBlk);
      mbar_expect_tx(do_full, Cfg::kTileBytes);
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a) tma_load_4d(smem + Cfg::kDOOff + a * (kBlk * 128), &p.tm_do, do_full, a * 64, h, m0, b);
      ok = load(&p.tm_v, nb * kBlk);
    }
    for (int j = nb + 1; j < ne && ok; ++j) ok = load(&p.tm_k, j * kBlk) && load(&p.tm_v, j * kBlk);
    for (int i = 0; i < kSlots && ok; ++i) {
      ok = mbar_wait(&kv_empty[slot], phase ^ 1, ctl, kWaitBwdDq + 5);
      if (++slot == kSlots) {
        slot = 0;
        phase ^= 1;
      }
    }
  } else if (warp == kMmaWarp && elect_one()) {
    // ---------------------------------------------------------------- MMA issuer
    constexpr uint32_t kBase = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) | (static_cast<uint32_t>(kBlk >> 4) << 24);
    constexpr uint32_t idesc_s = kBase | (static_cast<uint32_t>(kBlk >> 3) << 17);            // S, dP: both K-major
    constexpr uint32_t idesc_dq = kBase | (static_cast<uint32_t>(D >> 3) << 17) | (1u << 16);  // dQ: B MN-major
    constexpr uint32_t kTile16 = Cfg::kTileBytes >> 4;
    constexpr uint32_t kAtom16 = (kBlk * 128) >> 4;
    const uint64_t base = make_smem_desc(smem_u32(smem), 16, 1024);
    constexpr uint64_t kMn = static_cast<uint64_t>(((kBlk * 128) >> 4) - 1) << 16;
    const uint64_t q_desc = base + (Cfg::kQOff >> 4), do_desc = base + (Cfg::kDOOff >> 4), ring = base + (Cfg::kRingOff >> 4);
    auto kmajor_pair = [&](uint32_t d_tmem, uint64_t a, uint64_t bd) {
      static_for<D / 16>([&](auto ks) {
        constexpr uint32_t o = (ks.value / 4) * kAtom16 + (ks.value % 4) * 2;
        mma_ss_o<o, o>(d_tmem, a, bd, idesc_s, ks.value > 0 ? 1u : 0u);
      });
    };
    // K(j) is load 2j of the ring, V(j) load 2j + 1.
    auto slot_of = [](int load) { return static_cast<uint32_t>(load) % kSlots; };
    auto ready = [&](int load) { return mbar_wait(&kv_full[slot_of(load)], (static_cast<uint32_t>(load) / kSlots) & 1, ctl, kWaitBwdDq + 6); };
    auto do_s = [&](int it) -> bool {
      if (!ready(2 * it)) return false;
      tc_fence_after();
      // The buffer's previous dS has been read: the dQ product that did was issued before this one.
      kmajor_pair(tmem + Cfg::kTmemS + (it & 1) * kBlk, q_desc, ring + slot_of(2 * it) * kTile16);
      mma_commit(&s_full[it & 1]);
      return true;
    };
    auto do_dp = [&](int it) -> bool {
      if (!ready(2 * it + 1)) return false;
      if (it > 0 && !mbar_wait(dp_free, (it - 1) & 1, ctl, kWaitBwdDq + 7)) return false;
      tc_fence_after();
      kmajor_pair(tmem + Cfg::kTmemDP, do_desc, ring + slot_of(2 * it + 1) * kTile16);
      mma_commit(dp_full);
      mma_commit(&kv_empty[slot_of(2 * it + 1)]);
      return true;
    };
    bool ok = n_iter > 0;
    if (ok) ok = mbar_wait(q_full, 0, ctl, kWaitBwdDq + 8) && do_s(0) && mbar_wait(do_full, 0, ctl, kWaitBwdDq + 9) && do_dp(0);
    for (int it = 0; it < n_iter && ok; ++it) {
      if (it + 1 < n_iter) ok = do_s(it + 1) && do_dp(it + 1);
      if (ok) ok = mbar_wait(&ds_full[it & 1], (it >> 1) & 1, ctl, kWaitBwdDq + 10);
      if (!ok) break;
      tc_fence_after();
      const uint64_t kb = ring + kMn + slot_of(2 * it) * kTile16;
      const uint32_t ds = tmem + Cfg::kTmemS + (it & 1) * kBlk;
      static_for<kBlk / 16>([&](auto ks) {
        // dS: two 32-column halves of 64 keys at S + 0 and S + 64
        mma_ts_o<(ks.value / 4) * 64 + (ks.value % 4) * 8, ks.value * (2048 >> 4)>(tmem + Cfg::kTmemDQ, ds, kb, idesc_dq,
                                                                                   ks.value > 0 ? 1u : (it > 0 ? 1u : 0u));
      });
      mma_commit(&kv_empty[slot_of(2 * it)]);
    }
    if (ok) mma_commit(dq_done);
  }
  __syncwarp();
  if (*abort_flag) {
    // A wait ran out: what is in flight gets about a millisecond to land before barriers and TMEM are given back.
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0) report_abort(abort_flag, p.status);
  if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
}

template <int D, bool BF16, int MODE>
cudaError_t launch_one(const DqParams& p, cudaStream_t stream) {
  using Cfg = DqCfg<D>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_dq_kernel<D, BF16, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_grid(true, bwd_dq_kernel<D, BF16, MODE>, dim3(p.num_mblk * p.batch * p.heads), kThreads, Cfg::kSmemBytes, stream, p);
}

template <int D, bool BF16>
cudaError_t pick_mode(const DqParams& p, cudaStream_t stream) {
  switch ((p.softcap > 0.f ? kScoreSoftcap : 0) | (p.alibi != nullptr ? kScoreAlibi : 0)) {
    case kScorePlain: return launch_one<D, BF16, kScorePlain>(p, stream);
    case kScoreSoftcap: return launch_one<D, BF16, kScoreSoftcap>(p, stream);
    case kScoreAlibi: return launch_one<D, BF16, kScoreAlibi>(p, stream);
    default: return launch_one<D, BF16, kScoreAny>(p, stream);
  }
}

}  // namespace

cudaError_t launch_bwd_dq(const DqParams& p, bool bf16, cudaStream_t stream) {
  if (p.num_mblk * p.batch * p.heads <= 0) return cudaSuccess;
  if (p.head_dim <= 0 || p.head_dim > 128) return cudaErrorInvalidValue;
  if (p.head_dim > 64) return bf16 ? pick_mode<128, true>(p, stream) : pick_mode<128, false>(p, stream);
  return bf16 ? pick_mode<64, true>(p, stream) : pick_mode<64, false>(p, stream);
}

}  // namespace fa2
