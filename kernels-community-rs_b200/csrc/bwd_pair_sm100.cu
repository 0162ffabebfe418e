// FlashAttention-2 backward for sm_100a (B200) on pairs of CTAs: dQ, dK, dV of dense calls at head dims 104 ... 128.
//
// A pair owns 256 keys of one (batch, kv head), 128 in each CTA, and walks the 128-row query blocks (and the query heads of the GQA
// group) that can see them. Its MMAs are issued by one thread of CTA 0 for both tensor cores. Keys are on the TMEM lanes:
//
//   S^T  = K Q^T        256 x 128 x d    A: own keys in smem       B: Q rows, 64 in each CTA
//   dP^T = V dO^T       256 x 128 x d    A: own keys in smem       B: dO rows, 64 in each CTA
//   dV  += P^T dO       256 x d x 128    A: own keys in TMEM       B: dO columns, 64 in each CTA
//   dK  += dS^T Q       256 x d x 128    A: own keys in TMEM       B: Q columns, 64 in each CTA
//   dQ   = dS K         128 x d x 256    A: 64 own queries in smem B: K columns, 64 in each CTA
//
// dQ contracts over the keys of both CTAs, so each CTA sends its dS^T of the other one's 64 queries to that CTA's shared memory.
// What leaves the pair for the fp32 dQ accumulator is one tile of 128 queries for 256 keys, half of what two CTAs with 128 keys
// add (bwd_sm100.cu), and that traffic is what bounds those: 64 KB of reductions leave an SM in 2850-3100 cycles, of 3800 an
// iteration. Operands are halves too: 192 KB of shared memory are read per iteration and CTA in place of 288 (48 each for S^T and
// dP^T, 16 each for dV and dK, 64 for dQ).
//
// TMEM (columns): dK 0, dV 128, S^T 256 ... 383, dP^T 384 ... 511. P^T goes over the first half of S^T as soon as both warpgroups have
// read their scores, dQ over the second half; dS^T of a warpgroup over its own half of dP^T.
//
// Order of an iteration: dV, the next S^T, dK, the next dP^T, dQ. dK takes dS^T from TMEM at once, while the exchange through
// shared memory is under way, and dQ, which nothing in the iteration waits for, comes last: the drain has until the next dV.
//
// What bounds it: large calls run at the power limit (990 W, SM clock 1.45 GHz), where what counts is the energy of an iteration: the
// reductions into the accumulator are 13 % of a training step of B1 H32 S16384, and a pair issues half of them (7478 -> 7223 us). In
// cycles the compute warps, 3600 of an iteration: 1300 in the exponentials, both warpgroups at once; 550 for dS^T; 500 to hand dS^T on;
// the rest in waits and TMEM accesses. The exchange takes 1100 cycles and more (32 B/clk); the same stores straight to the other CTA, with
// their proxy fence, took 2000 that the compute warps had to wait for.
//
// The issuer's and the loader's steps are loops with one place in the code for each: the roles share the SM's instruction cache. With
// a prologue of its own for each and the loader's steps written out (65 KB of machine code) B1 H32 S16384 took 7241 us, now 7223,
// B4 H16/4 S4096 without a mask 1909, now 1893.
//
// Warps: 0 loader, 1 MMA issuer (CTA 0), 2 reports what CTA 1 has received, 3 statistics, 4-11 compute (two warpgroups, 64 queries each, one key per thread),
// 12-15 dQ drain (64 queries, warps 12 and 13 columns 0-63, 14 and 15 columns 64-127).
#include "sm100_ptx.cuh"
#include "fa2_params.h"
#include "fa2_launch.h"
#include "bwd_tile.cuh"

namespace fa2 {

namespace {

constexpr int kThreads = 512;
constexpr int kComputeRegs = 168;
constexpr int kDrainRegs = 104;
constexpr int kMiscRegs = 56;
// setmaxnreg moves registers inside the CTA's own allocation (128 per thread at launch).
static_assert(8 * (kComputeRegs - 128) <= 4 * (128 - kMiscRegs) + 4 * (128 - kDrainRegs), "setmaxnreg: more registers asked for than released");

struct PairCfg {
  static constexpr int D = 128;
  static constexpr int kAtomBytes = kBlk * 128;          // 128 rows of 64 16-bit values
  static constexpr int kTileBytes = 2 * kAtomBytes;
  static constexpr int kKOff = 0;                        // own 128 keys, K-major
  static constexpr int kKColOff = kKOff + kTileBytes;    // 64 columns of all 256 keys
  static constexpr int kVOff = kKColOff + kTileBytes;    // own 128 keys
  static constexpr int kQOff = kVOff + kTileBytes;       // own 64 query rows
  static constexpr int kQColOff = kQOff + kAtomBytes;    // 64 columns of all 128 query rows
  static constexpr int kDOOff = kQColOff + kAtomBytes;
  static constexpr int kDOColOff = kDOOff + kAtomBytes;
  static constexpr int kDSOff = kDOColOff + kAtomBytes;  // dS^T of own 64 queries: [256 keys][64]
  static constexpr int kSendOff = kDSOff + kTileBytes;   // dS^T of the other CTA's queries on its way there: [128 own keys][64]
  static constexpr int kPieceBytes = 32 * 128;           // dQ staging piece of a drain warp: [32 rows][32 fp32]
  static constexpr int kDQOff = kSendOff + kAtomBytes;
  static constexpr int kBarOff = kDQOff + 4 * kPieceBytes;
  static constexpr int kNumBars = 30;
  static constexpr int kMiscOff = kBarOff + kNumBars * 8;
  static constexpr int kStatOff = kMiscOff + 16;         // lse / delta: [2 buffers][2][128] fp32
  static constexpr int kSmemBytes = kStatOff + 2 * 2 * kBlk * 4;
  static_assert(kStatOff % 16 == 0 && kSmemBytes <= 227 * 1024, "shared memory");
  static constexpr uint32_t kTmemDK = 0, kTmemDV = 128, kTmemS = 256, kTmemDQ = 320, kTmemDP = 384;
};

__device__ __forceinline__ PairTile get_pair_tile(const BwdParams& p, int t) {
  PairTile ti;
  const int per_head = (p.num_nblk + 1) >> 1;
  const int first_bh = t / (p.head_group * per_head) * p.head_group;
  const int n_bh = min(p.head_group, p.batch * p.heads_k - first_bh);
  const int in_group = t - first_bh * per_head;
  const int i = in_group / n_bh;
  const int bh = first_bh + in_group - i * n_bh;
  ti.b = bh / p.heads_k;
  ti.hk = bh - ti.b * p.heads_k;
  ti.n0 = i * (2 * kBlk);
  q_block_range(p, p.seqlen_q, p.seqlen_k, ti.n0, 2 * kBlk, ti.m_start, ti.n_m);
  ti.n_iter = ti.n_m * p.group;
  return ti;
}

template <bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) bwd_pair_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = PairCfg;
  constexpr int D = Cfg::D;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    early_wait();
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, kWaitNone + 1);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOff);
  // Barriers that both CTAs feed and the issuer waits for: only those of CTA 0 are used.
  uint64_t* k_full = bars + 0;      // K and, on barriers of their own, its columns and V
  uint64_t* kcol_full = bars + 1;
  uint64_t* v_full = bars + 2;
  uint64_t* q_full = bars + 3;
  uint64_t* qcol_full = q_full + 1;
  uint64_t* do_full = bars + 5;
  uint64_t* docol_full = do_full + 1;
  uint64_t* p_full = bars + 7;      // P^T is in TMEM
  uint64_t* ds_full = bars + 8;     // dS^T is in TMEM
  uint64_t* dsx_full = bars + 9;    // dS^T is in shared memory: what stays in its CTA, and what CTA 1 has received
  uint64_t* s_read = bars + 10;     // the second warpgroups have read their scores: dQ may overwrite them
  uint64_t* dq_free = bars + 11;    // dQ has left TMEM
  // Barriers of each CTA; commits arrive at those of both.
  uint64_t* q_empty = bars + 12;
  uint64_t* qcol_empty = q_empty + 1;
  uint64_t* do_empty = bars + 14;
  uint64_t* docol_empty = do_empty + 1;
  uint64_t* s_full = bars + 16;
  uint64_t* dp_full = bars + 17;
  uint64_t* dq_full = bars + 18;
  uint64_t* dv_done = bars + 19;
  uint64_t* dk_done = bars + 20;
  uint64_t* s_read0 = bars + 21;    // the first warpgroup has read its scores: the second one's P^T may overwrite them
  uint64_t* stat_full = bars + 22;  // [2]
  uint64_t* stat_empty = bars + 24; // [2]
  uint64_t* epi_full = bars + 26;   // [2] dK, dV are staged for their bulk store
  uint64_t* received = bars + 28;   // dS^T of the other CTA's keys has arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff + 8);
  float* s_stat = reinterpret_cast<float*>(smem + Cfg::kStatOff);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const WaitCtl ctl{abort_flag};
  const PairTile ti = get_pair_tile(p, blockIdx.x >> 1);
  const int n_iter = ti.n_iter;
  const int n0 = ti.n0 + static_cast<int>(rank) * kBlk;  // first key of this CTA
  const int off = p.seqlen_k - p.seqlen_q;

  if (warp == 2 && lane == 0) {
    tma_prefetch_desc(&p.tm_k);
    tma_prefetch_desc(&p.tm_q);
    tma_prefetch_desc(&p.tm_v);
    tma_prefetch_desc(&p.tm_do);
    tma_prefetch_desc(&p.tm_dqa);
  }
  if (warp == 0) {
    if (lane < Cfg::kNumBars) {
      uint64_t* bar = bars + lane;
      uint32_t count = 1;
      if (bar == p_full || bar == ds_full) count = 16;  // compute warps of both CTAs
      if (bar == dsx_full) count = 9;                   // a warpgroup of each, and CTA 1's word that it has received
      if (bar == s_read || bar == dq_free) count = 8;
      if (bar == s_read0) count = 4;
      if (bar == stat_empty || bar == stat_empty + 1) count = 8;
      if (bar == epi_full || bar == epi_full + 1) count = kBlk;
      mbar_init(bar, count);
    }
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
    __syncwarp();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  // No barrier of a CTA is touched, and no MMA issued, before both have set theirs up and have their TMEM.
  tc_fence_before();
  __syncwarp();
  cluster_arrive();
  early_wait();
  cluster_wait();

  auto leader = [&](uint64_t* bar) { return peer_smem(smem_u32(bar), 0); };
  // One operand tile of both CTAs: CTA 0 announces the bytes of the two.
  auto expect = [&](uint64_t* full, uint32_t bytes_each) {
    if (rank == 0) mbar_expect_tx(full, 2 * bytes_each);
  };
  // Two pieces of a tile: 128 or 64 rows of two 64-column atoms.
  auto load2 = [&](int dst, int step, const CUtensorMap* tm, uint64_t* full, int head, int c0, int c1, int r0, int r1) {
    expect(full, 2 * step);
    tma_load_4d_pair(smem + dst, tm, leader(full), c0, head, r0, ti.b);
    tma_load_4d_pair(smem + dst + step, tm, leader(full), c1, head, r1, ti.b);
  };
  if (tid == 0 && n_iter > 0) {
    const int col = static_cast<int>(rank) * 64;
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
      const bool cols = i == 2;  // K, V, K's columns
      load2(i == 0 ? Cfg::kKOff : i == 1 ? Cfg::kVOff : Cfg::kKColOff, Cfg::kAtomBytes, i == 1 ? &p.tm_v : &p.tm_k,
            i == 0 ? k_full : i == 1 ? v_full : kcol_full, ti.hk, cols ? col : 0, cols ? col : 64, cols ? ti.n0 : n0, cols ? ti.n0 + kBlk : n0);
    }
  }
  __syncthreads();
  tc_fence_after();
  early_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    reg_dealloc<kMiscRegs>();
    if (warp == 0 && elect_one()) {
      // ---------------------------------------------------------------- loader
      // In the order in which the stages come back: dO columns, the next Q rows, Q columns, the next dO rows. One place in the code:
      // the roles of the CTA share the SM's instruction cache.
      Walk w{0, -1}, next{0, 0};
      bool ok = true;
#pragma unroll 1
      for (int it = -1; it < n_iter && ok; ++it) {
#pragma unroll 1
        for (int i = 0; i < 4 && ok; ++i) {
          const bool rows = (i & 1) != 0, is_q = i == 1 || i == 2;
          if (rows ? it + 1 >= n_iter : it < 0) continue;
          // own 64 rows of both halves of the head dim, or the own half of the head dim of both halves of the rows
          const int use = rows ? it + 1 : it, r = static_cast<int>(rank) * 64;
          const Walk& at = rows ? next : w;
          const int row = (ti.m_start + at.mi) * kBlk;
          ok = mbar_wait((is_q ? q_empty : do_empty) + (rows ? 0 : 1), (use & 1) ^ 1, ctl, kWaitBwd + 1);
          if (ok)
            load2((is_q ? Cfg::kQOff : Cfg::kDOOff) + (rows ? 0 : Cfg::kAtomBytes), Cfg::kAtomBytes / 2, is_q ? &p.tm_q : &p.tm_do,
                  (is_q ? q_full : do_full) + (rows ? 0 : 1), ti.hk * p.group + at.g, rows ? 0 : r, rows ? 64 : r, rows ? row + r : row,
                  rows ? row + r : row + 64);
        }
        w = next;
        next = walk_next(next, ti.n_m);
      }
    } else if (warp == 1 && rank == 0 && elect_one()) {
      // ---------------------------------------------------------------- mma issuer, for both CTAs
      constexpr uint32_t kBase = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) | (static_cast<uint32_t>(kBlk >> 3) << 17);
      constexpr uint32_t idesc_qk = kBase | (static_cast<uint32_t>(256 >> 4) << 24);                           // S^T, dP^T
      constexpr uint32_t idesc_dv = idesc_qk | (1u << 16);                                                     // dV, dK: B MN-major
      constexpr uint32_t idesc_dq = kBase | (static_cast<uint32_t>(128 >> 4) << 24) | (1u << 15) | (1u << 16);  // A and B MN-major
      const uint64_t base = make_smem_desc(smem_u32(smem), 16, 1024);
      constexpr uint64_t kMn = static_cast<uint64_t>((Cfg::kAtomBytes >> 4) - 1) << 16;  // one chunk of 64 along M or N
      const uint64_t k_d = base + (Cfg::kKOff >> 4), v_d = base + (Cfg::kVOff >> 4), kcol_d = base + (Cfg::kKColOff >> 4) + kMn;
      const uint64_t q_d = base + (Cfg::kQOff >> 4), do_d = base + (Cfg::kDOOff >> 4);
      const uint64_t qcol_d = base + (Cfg::kQColOff >> 4) + kMn, docol_d = base + (Cfg::kDOColOff >> 4) + kMn;
      const uint64_t ds_d = base + (Cfg::kDSOff >> 4) + kMn;
      // [256 keys x 128 q] over d in steps of 16: A atoms of 128 rows, B atoms of 64
      auto kmajor = [&](uint32_t d_tmem, uint64_t a, uint64_t b) {
        static_for<D / 16>([&](auto ks) {
          mma_pair_ss_o<(ks.value / 4) * (Cfg::kAtomBytes >> 4) + (ks.value % 4) * 2,
                        (ks.value / 4) * (Cfg::kAtomBytes >> 5) + (ks.value % 4) * 2>(d_tmem, a, b, idesc_qk, ks.value > 0 ? 1u : 0u);
        });
      };
      bool ok = n_iter > 0;
#pragma unroll 1
      for (int it = -1; it < n_iter && ok; ++it) {
        const uint32_t ph = it & 1;
        const bool has_next = it + 1 < n_iter;
        const uint32_t acc = it > 0 ? 1u : 0u;
        // dV += P^T dO
        if (it >= 0) {
          ok = mbar_wait(docol_full, ph, ctl, kWaitBwd + 5) && mbar_wait(p_full, ph, ctl, kWaitBwd + 6);
          if (!ok) break;
          tc_fence_after();
          static_for<kBlk / 16>([&](auto ks) {
            mma_pair_ts_o<ks.value * 8, ks.value * (2048 >> 4)>(tmem + Cfg::kTmemDV, tmem + Cfg::kTmemS, docol_d, idesc_dv,
                                                                ks.value > 0 ? 1u : acc);
          });
          mma_pair_commit(docol_empty);
          if (!has_next) mma_pair_commit(dv_done);
        }
        // S^T of the next iteration: over P^T, which dV has read, and dQ of the iteration before, which has been drained
        if (has_next) {
          ok = mbar_wait(q_full, ph ^ 1, ctl, kWaitBwd + 8) &&
               (it > 0 ? mbar_wait(dq_free, ph ^ 1, ctl, kWaitBwd + 10) : it == 0 || mbar_wait(k_full, 0, ctl, kWaitBwd + 3));
          if (!ok) break;
          tc_fence_after();
          kmajor(tmem + Cfg::kTmemS, k_d, q_d);
          mma_pair_commit(s_full);
          mma_pair_commit(q_empty);
        }
        // dK += dS^T Q
        if (it >= 0) {
          ok = mbar_wait(qcol_full, ph, ctl, kWaitBwd + 4) && mbar_wait(ds_full, ph, ctl, kWaitBwd + 7);
          if (!ok) break;
          tc_fence_after();
          static_for<kBlk / 16>([&](auto ks) {
            mma_pair_ts_o<(ks.value / 4) * 64 + (ks.value % 4) * 8, ks.value * (2048 >> 4)>(tmem + Cfg::kTmemDK, tmem + Cfg::kTmemDP, qcol_d,
                                                                                          idesc_dv, ks.value > 0 ? 1u : acc);
          });
          mma_pair_commit(qcol_empty);
        }
        // dP^T of the next iteration, over dP^T and dS^T of this one
        if (has_next) {
          ok = mbar_wait(do_full, ph ^ 1, ctl, kWaitBwd + 9) && (it >= 0 || mbar_wait(v_full, 0, ctl, kWaitBwd + 3));
          if (!ok) break;
          tc_fence_after();
          kmajor(tmem + Cfg::kTmemDP, v_d, do_d);
          mma_pair_commit(dp_full);
          mma_pair_commit(do_empty);
        }
        if (it < 0) continue;
        // dQ = dS K, over the second half of the next S^T, which has been read
        mbar_expect_tx(received, Cfg::kAtomBytes);
        ok = (it > 0 || mbar_wait(kcol_full, 0, ctl, kWaitBwd + 3)) && mbar_wait(received, ph, ctl, kWaitBwd + 19) &&
             mbar_wait(dsx_full, ph, ctl, kWaitBwd + 7) &&
             (has_next ? mbar_wait(s_read, ph ^ 1, ctl, kWaitBwd + 11) : it == 0 || mbar_wait(dq_free, ph ^ 1, ctl, kWaitBwd + 10));
        if (!ok) break;
        tc_fence_after();
        static_for<2 * kBlk / 16>([&](auto ks) {
          mma_pair_ss_o<ks.value * (2048 >> 4), ks.value * (2048 >> 4)>(tmem + Cfg::kTmemDQ, ds_d, kcol_d, idesc_dq, ks.value > 0 ? 1u : 0u);
        });
        mma_pair_commit(dq_full);
      }
      // Only for who waits: an arrival that nobody waits for could land in the other CTA after its end.
      if (ok) mma_pair_commit(dk_done);
    } else if (warp == 2 && rank == 1 && elect_one()) {
      // ---------------------------------------------------------------- tells the issuer what this CTA has received
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        mbar_expect_tx(received, Cfg::kAtomBytes);
        ok = mbar_wait(received, it & 1, ctl, kWaitBwd + 19);
        if (ok) mbar_arrive_cluster(leader(dsx_full));
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- -LSE (log2 domain) and -delta of a query block
      bool ok = pair_statistics(p, ti, s_stat, stat_full, stat_empty, lane, ctl);
      // The stages' last commits land before the CTA ends: q_empty, qcol_empty, do_empty, docol_empty.
#pragma unroll 1
      for (int i = 0; i < 4 && ok; ++i) ok = mbar_wait(q_empty + i, (n_iter - 1) & 1, ctl, kWaitBwd + 1);
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ compute
    reg_alloc<kComputeRegs>();
    const int cw = warp - 4;
    const int wg = cw >> 2;                 // which 64 queries: those of CTA wg's dQ rows
    const int key_in = (cw & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((cw & 3) * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + Cfg::kTmemS + wg * 64;
    const uint32_t t_p = tmem + lane_addr + Cfg::kTmemS + wg * 32;
    const uint32_t t_dp = tmem + lane_addr + Cfg::kTmemDP + wg * 64;
    const uint32_t p_bar = leader(p_full), ds_bar = leader(ds_full), dsx_bar = leader(dsx_full);
    const uint32_t read_bar = wg == 0 ? smem_u32(s_read0) : leader(s_read);
    // dS^T of this CTA's queries is written where its dQ reads it, that of the other's is sent there, 4 KB a warp.
    const bool keeps = wg == static_cast<int>(rank);
    uint8_t* ds_row = smem + (keeps ? Cfg::kDSOff + rank * Cfg::kAtomBytes : Cfg::kSendOff) + key_in * 128;
    const uint32_t send_from = smem_u32(smem + Cfg::kSendOff) + (cw & 3) * 4096;
    const uint32_t send_to = peer_smem(smem_u32(smem + Cfg::kDSOff + rank * Cfg::kAtomBytes) + (cw & 3) * 4096, wg);
    const uint32_t send_bar = peer_smem(smem_u32(received), wg);
    const int kpos = n0 + key_in;
    bool ok = true;
    Walk w{0, 0};
    for (int it = 0; it < n_iter; ++it) {
      const int m0 = (ti.m_start + w.mi) * kBlk;
      w = walk_next(w, ti.n_m);
      const uint32_t par = it & 1;
      const float* stat = s_stat + par * (2 * kBlk);
      const bool stat_ok = mbar_wait(&stat_full[par], (it >> 1) & 1, ctl, kWaitBwd + 15);  // voted on with s_full below
      const float4* lse4 = reinterpret_cast<const float4*>(stat + wg * 64);
      const float4* dl4 = reinterpret_cast<const float4*>(stat + kBlk + wg * 64);

      // ---- phase A: P^T = exp2(S^T c - lse)
      if (!__all_sync(0xffffffffu, mbar_wait(s_full, par, ctl, kWaitBwd + 11) && stat_ok)) { ok = false; break; }
      tc_fence_after();
      uint32_t sr[64];
      tmem_ld32(t_s, sr);
      tmem_ld32(t_s + 32, sr + 32);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (wg == 0) mbar_arrive(s_read0);
        else mbar_arrive_cluster(read_bar);
      }
      const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
      float pr[64];
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float4 l4 = lse4[i / 4];
        unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, pack_f32x2(l4.x, l4.y)), pr[i], pr[i + 1]);
        unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), c2, pack_f32x2(l4.z, l4.w)), pr[i + 2], pr[i + 3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) pr[i + e] = ex2(pr[i + e]);
      }
      bool need_mask = (n0 + kBlk > p.seqlen_k);
      if (p.window_right >= 0) need_mask |= (n0 + kBlk - 1 > m0 + off + p.window_right);
      if (p.window_left >= 0) need_mask |= (n0 < m0 + kBlk - 1 + off - p.window_left);
      if (need_mask) {
        const int qbase = m0 + wg * 64;
        int lo = 0, hi = 64;
        if (p.window_right >= 0) lo = kpos - off - p.window_right - qbase;
        if (p.window_left >= 0) hi = kpos - off + p.window_left + 1 - qbase;
        if (kpos >= p.seqlen_k) hi = -1;
        fill_outside<64>(pr, lo, hi, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) sr[i] = pack2<BF16>(pr[2 * i], pr[2 * i + 1]);
      if (wg == 1 && !warp_wait(s_read0, par, ctl, kWaitBwd + 17)) { ok = false; break; }
      tc_fence_after();
      tmem_st32(t_p, sr);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(p_bar);

      // ---- phase B: dS^T = P^T (dP^T - delta), to TMEM for dK and to the queries' owner for dQ
      // dQ of the iteration before has read the buffers that dS^T goes to.
      if (!__all_sync(0xffffffffu, mbar_wait(dp_full, par, ctl, kWaitBwd + 12) && (it == 0 || mbar_wait(dq_full, par ^ 1, ctl, kWaitBwd + 18)))) {
        ok = false;
        break;
      }
      tc_fence_after();
      tmem_ld32(t_dp, sr);
      tmem_ld32(t_dp + 32, sr + 32);
      tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float4 d = dl4[i / 4];
        float a, b;
        unpack_f32x2(mul2(pack_f32x2(pr[i], pr[i + 1]),
                          add2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), pack_f32x2(d.x, d.y))), a, b);
        sr[i / 2] = pack2<BF16>(a, b);
        unpack_f32x2(mul2(pack_f32x2(pr[i + 2], pr[i + 3]),
                          add2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), pack_f32x2(d.z, d.w))), a, b);
        sr[i / 2 + 1] = pack2<BF16>(a, b);
      }
      // The way to the other CTA takes 1100 cycles and more, so it is taken first.
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(ds_row + ((c ^ (key_in & 7)) << 4)) = make_uint4(sr[4 * c], sr[4 * c + 1], sr[4 * c + 2], sr[4 * c + 3]);
      tmem_st32(t_dp, sr);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (keeps) mbar_arrive_cluster(dsx_bar);
        else bulk_copy_cluster(send_to, send_from, 4096, send_bar);
        mbar_arrive(&stat_empty[par]);
      }
      __syncwarp();
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(ds_bar);
    }
    // ---- epilogue: warpgroup 0 writes dK (scaled), warpgroup 1 writes dV, through the K and V tiles
    if (ok && n_iter > 0) ok = warp_wait(wg == 0 ? dk_done : dv_done, 0, ctl, kWaitBwd + 13);
    if (ok && n0 < p.seqlen_k) {
      tc_fence_after();
      const uint32_t t_acc = tmem + lane_addr + (wg == 0 ? Cfg::kTmemDK : Cfg::kTmemDV);
      const float mul = (wg == 0) ? p.scale : 1.f;
      uint8_t* stage = smem + (wg == 0 ? Cfg::kKOff : Cfg::kVOff);
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        uint32_t acc[64];
        if (n_iter > 0) {
          tmem_ld32(t_acc + h * 64, acc);
          tmem_ld32(t_acc + h * 64 + 32, acc + 32);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) acc[i] = 0;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t o[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            o[q] = pack2<BF16>(__uint_as_float(acc[8 * c + 2 * q]) * mul, __uint_as_float(acc[8 * c + 2 * q + 1]) * mul);
          *reinterpret_cast<uint4*>(stage + h * Cfg::kAtomBytes + key_in * 128 + ((c ^ (key_in & 7)) << 4)) =
              make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(&epi_full[wg]);
      if (key_in == 0 && mbar_wait(&epi_full[wg], 0, ctl, kWaitBwd + 16)) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
          if (a * 64 < p.head_dim) tma_store_4d(wg == 0 ? &p.tm_dk : &p.tm_dv, stage + a * Cfg::kAtomBytes, a * 64, ti.hk, n0, ti.b);
        tma_commit_group();
        tma_wait_group_read<0>();
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ dQ drain
    // Rows 64 rank + 32 (warp & 1) + lane of the query block, columns 64 (dw / 2) + 0 ... 63. The tile leaves TMEM at once and
    // goes through a staging buffer of the warp's own, 32 columns at a time, as reductions into the fp32 accumulator.
    reg_dealloc<kDrainRegs>();
    const int dw = warp & 3;
    const uint32_t t_dq = tmem + (static_cast<uint32_t>(dw * 32) << 16) + Cfg::kTmemDQ;
    const uint32_t free_bar = leader(dq_free);
    const int col0 = (dw >> 1) * 64;
    uint8_t* buf = smem + Cfg::kDQOff + dw * Cfg::kPieceBytes;
    Walk w{0, 0};
    bool ok = true;
    for (int it = 0; it < n_iter; ++it, w = walk_next(w, ti.n_m)) {
      const int hq = ti.hk * p.group + w.g;
      const int row = (ti.m_start + w.mi) * kBlk + static_cast<int>(rank) * 64 + (dw & 1) * 32;
      ok = warp_wait(dq_full, it & 1, ctl, kWaitBwd + 14);
      if (!ok) break;
      tc_fence_after();
      uint32_t acc[64];
      tmem_ld32(t_dq, acc);
      tmem_ld32(t_dq + 32, acc + 32);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(free_bar);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        // The buffer is free once the reduction before has read it.
        if (lane == 0) tma_wait_group_read<0>();
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(buf + lane * 128 + ((c ^ (lane & 7)) << 4)) =
              make_uint4(acc[k * 32 + 4 * c], acc[k * 32 + 4 * c + 1], acc[k * 32 + 4 * c + 2], acc[k * 32 + 4 * c + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (col0 + k * 32 < p.head_dim) tma_reduce_add_4d(&p.tm_dqa, buf, col0 + k * 32, hq, row, ti.b);
          tma_commit_group();
        }
      }
    }
    if (lane == 0) tma_wait_group_read<0>();
  }
  end_pair(p, abort_flag, tid, warp, tmem);
}

template <bool BF16>
cudaError_t launch_one(const BwdParams& p, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_pair_kernel<BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int64_t blocks = static_cast<int64_t>(p.num_nblk + 1) / 2 * 2 * p.batch * p.heads_k;
  if (blocks <= 0) return cudaSuccess;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  return launch_grid(true, bwd_pair_kernel<BF16>, dim3(static_cast<unsigned>(blocks)), kThreads, PairCfg::kSmemBytes, stream, p);
}

}  // namespace

cudaError_t launch_bwd_pair(const BwdParams& p, bool bf16, cudaStream_t stream) {
  return bf16 ? launch_one<true>(p, stream) : launch_one<false>(p, stream);
}

}  // namespace fa2
