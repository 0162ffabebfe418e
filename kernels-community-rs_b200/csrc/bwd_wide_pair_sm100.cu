// FlashAttention-2 backward for sm_100a (B200) on pairs of CTAs, head dims 192 and 256: dQ, dK, dV of dense calls.
//
// A pair owns 128 keys of one (batch, kv head), 64 in each CTA, and walks the 128-row query blocks (and the query heads of the GQA
// group) that can see them. Its MMAs are issued by one thread of CTA 0 for both tensor cores:
//
//   S^T  = K Q^T       128 x 128 x 256   A: own 64 keys                 B: Q rows, 64 in each CTA
//   dP^T = V dO^T      128 x 128 x 256   A: own 64 keys                 B: dO rows, 64 in each CTA
//   dV  += P^T dO      128 x 256 x 128   A: own keys                    B: dO columns, 128 in each CTA
//   dK  += dS^T Q      128 x 256 x 128   A: own keys                    B: Q columns, 128 in each CTA
//   dQ^T = K^T dS^T    256 x 128 x 128   A: 128 K columns in each CTA   B: dS^T of 64 queries in each CTA
//
// all from shared memory (figures for head dim 256; at 192 the last 64 columns are zeros, which S^T and dP^T leave out). In each CTA's TMEM a result of 128 rows has 64 of them: lanes 0-63 hold the first half of the columns,
// lanes 64-127 the second. So dK and dV of the pair take 128 columns each, S^T and dP^T 64, dQ^T 128. In the kernel with one CTA per
// 128 keys and half of the head dim (bwd_wide_sm100.cu) S^T and dP^T, which contract over all of the head dim, are computed twice,
// exponentials included, and most MMAs have N = 64, which costs 35-54 cycles in place of 32.
//
// dQ contracts over the keys of both CTAs: each sends its dS^T of the other one's 64 queries there (8 KB through distributed shared
// memory). Order of an iteration: dV, the next S^T, dK, the next dP^T, dQ^T; the exchange runs beside dK and dP^T.
//
// K, V and K's columns take 96 KB of shared memory, the rest leaves a ring of 64 KB for the 128 KB of Q and dO that an iteration
// reads. A load brings 16 KB, 64 rows of two 64-column atoms, with a map that lists the atoms as a dimension: with boxes of one atom the
// loading thread was what everything waited for (32 loads an iteration, 350 cycles each: 661 us for the kernel at B4 H16/8 S2048 causal,
// with 16 KB a load 465).
//
// The roles share the SM's instruction cache: with the issuer's and the loader's steps unrolled and a prologue of its own for
// each, 88 KB of machine code, a wait for a barrier that had completed long ago took 150-400 cycles and an iteration 9000. Loops with one
// place in the code for each step, 54 KB: 5350 cycles (the old kernel: 6600), the kernel 410 us (old: 476).
// Forward and backward in a steady loop, old kernel -> this one, us, causal: B4 H16/8 S2048 808 -> 720, B1 H16 S8192 2544 -> 2247,
// B2 H16/4 S2048 softcap 612 -> 477, B2 H16 S4096 window 256 479 -> 423; B4 H8 S1000 without a mask 221 -> 197, B16 H8 S300 156 -> 157; at head dim 192
// B4 H16/8 S2048 711 -> 638, B2 H16/4 S2048 softcap 588 -> 430, B4 H8 S1000 without a mask 194 -> 175.
//
// What bounds it: the latency of the ring, a turn of which takes a load's 900-1400 cycles twice an iteration, and the MMAs, 2600.
//
// Warps: 0 loader, 1 MMA issuer (CTA 0), 2 reports what CTA 1 has received, 3 statistics, 4-11 compute (one key and 32 queries a
// thread), 12-15 dQ drain (one column of the head dim a thread; transposed through staging buffers into fp32 reductions).
#include "sm100_ptx.cuh"
#include "fa2_params.h"
#include "fa2_launch.h"
#include "bwd_tile.cuh"

namespace fa2 {

namespace {

constexpr int kThreads = 512;
constexpr int kKeys = 64;  // keys of a CTA

struct WidePairCfg {
  static constexpr int kKAtom = kKeys * 128;                // 64 columns of a CTA's keys
  static constexpr int kKOff = 0;                           // own keys, whole head dim
  static constexpr int kKColOff = kKOff + 4 * kKAtom;       // 128 columns of all 128 keys: [2 halves of the keys][2][64][64]
  static constexpr int kVOff = kKColOff + 4 * kKAtom;
  // Q and dO go through a ring in the order in which the MMAs read them. A slot holds 128 columns of 64 rows, in two chunks of 64
  // columns: a half of the columns of the CTA's own query rows (S^T, dP^T), or its half of the columns of a half of the rows (dV, dK).
  static constexpr int kSlots = 4;
  static constexpr int kSlotBytes = 2 * kKAtom;
  static constexpr int kRingOff = kVOff + 4 * kKAtom;
  static constexpr int kPOff = kRingOff + kSlots * kSlotBytes;  // P^T, then dS^T: [2 halves of the queries][64 own keys][64]
  // dS^T [2][128 keys][32 own q] and, on its way, [2][64 own keys][32 q of the other CTA]: rows of 64 bytes, swizzled
  static constexpr int kDSQChunk = 2 * kKeys * 64;
  static constexpr int kSendChunk = kKeys * 64;
  static constexpr int kDSQOff = kPOff + 2 * kKAtom;
  static constexpr int kSendOff = kDSQOff + 2 * kDSQChunk;
  static constexpr int kPieceRows = 16;                     // dQ staging piece of a drain warp: [16 q][32 d] fp32
  static constexpr int kPieceBytes = kPieceRows * 128;
  static constexpr int kPieces = 3;
  static constexpr int kDQOff = kSendOff + 2 * kSendChunk;
  static constexpr int kBarOff = kDQOff + 4 * kPieces * kPieceBytes;
  static constexpr int kNumBars = 2 * kSlots + 22;
  static constexpr int kMiscOff = (kBarOff + kNumBars * 8 + 15) / 16 * 16;
  static constexpr int kStatOff = kMiscOff + 16;            // lse / delta: [2 buffers][2][128] fp32
  static constexpr int kSmemBytes = kStatOff + 2 * 2 * kBlk * 4;
  static_assert(kStatOff % 16 == 0 && kSmemBytes <= 227 * 1024, "shared memory");
  static constexpr uint32_t kTmemDK = 0, kTmemDV = 128, kTmemS = 256, kTmemDP = 320, kTmemDQ = 384;
};

__device__ __forceinline__ PairTile get_wide_pair_tile(const BwdParams& p, int t) {
  PairTile ti;
  const int first_bh = t / (p.head_group * p.num_nblk) * p.head_group;
  const int n_bh = min(p.head_group, p.batch * p.heads_k - first_bh);
  const int in_group = t - first_bh * p.num_nblk;
  const int nblk = in_group / n_bh;
  const int bh = first_bh + in_group - nblk * n_bh;
  ti.b = bh / p.heads_k;
  ti.hk = bh - ti.b * p.heads_k;
  ti.n0 = nblk * (2 * kKeys);
  q_block_range(p, p.seqlen_q, p.seqlen_k, ti.n0, 2 * kKeys, ti.m_start, ti.n_m);
  ti.n_iter = ti.n_m * p.group;
  return ti;
}

// FANCY: a soft cap or ALiBi is in use.
// ATOMS: 64-column atoms of the head dim; the fourth one is zeros at head dim 192 (the loads fill it), and only the contractions over the
// head dim leave it out.
template <int ATOMS, bool BF16, bool FANCY>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) bwd_wide_pair_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = WidePairCfg;
  constexpr int D = 256, kHalf = D / 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    early_wait();
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, kWaitNone + 1);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOff);
  // Barriers that both CTAs feed and the issuer waits for: only those of CTA 0 are used.
  uint64_t* ring_full = bars;                      // [kSlots]
  uint64_t* k_full = bars + 2 * Cfg::kSlots;
  uint64_t* kcol_full = k_full + 1;
  uint64_t* v_full = k_full + 2;
  uint64_t* p_full = k_full + 3;
  uint64_t* ds_full = k_full + 4;      // dS^T is where dK reads it
  uint64_t* dsq_full = k_full + 5;     // dS^T is where dQ reads it: what stays in its CTA, and what CTA 1 has received
  uint64_t* dq_free = k_full + 6;      // dQ^T has left TMEM
  // Barriers of each CTA; commits arrive at those of both.
  uint64_t* ring_empty = bars + Cfg::kSlots;       // [kSlots]
  uint64_t* s_full = k_full + 7;
  uint64_t* dp_full = k_full + 8;
  uint64_t* dv_read = k_full + 9;      // dV has read P^T, and dQ^T of the iteration before its dS^T
  uint64_t* dk_read = k_full + 10;     // dK has read dS^T
  uint64_t* dq_full = k_full + 11;
  uint64_t* dk_done = k_full + 12;
  uint64_t* stat_full = k_full + 13;   // [2]
  uint64_t* stat_empty = k_full + 15;  // [2]
  uint64_t* epi_full = k_full + 17;    // [2]
  uint64_t* received = k_full + 19;    // dS^T of the other CTA's keys has arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff + 8);
  float* s_stat = reinterpret_cast<float*>(smem + Cfg::kStatOff);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int rank = static_cast<int>(cluster_rank());
  const WaitCtl ctl{abort_flag};
  const PairTile ti = get_wide_pair_tile(p, blockIdx.x >> 1);
  const int n_iter = ti.n_iter;
  const int n0 = ti.n0 + rank * kKeys;  // first key of this CTA
  const int off = p.seqlen_k - p.seqlen_q;

  if (warp == 2 && lane == 0) {
    tma_prefetch_desc(&p.tm_k);
    tma_prefetch_desc(&p.tm_q);
    tma_prefetch_desc(&p.tm_v);
    tma_prefetch_desc(&p.tm_do);
    tma_prefetch_desc(&p.tm_dqa);
  }
  if (warp == 0) {
    for (int i = lane; i < Cfg::kNumBars; i += 32) {
      uint64_t* bar = bars + i;
      uint32_t count = 1;
      if (bar == p_full || bar == ds_full) count = 16;  // compute warps of both CTAs
      if (bar == dsq_full) count = 9;                   // four warps of each, and CTA 1's word that it has received
      if (bar == dq_free) count = 8;
      if (bar == stat_empty || bar == stat_empty + 1) count = 8;
      if (bar == epi_full || bar == epi_full + 1) count = 128;
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
  // CTA 0 announces the bytes of both.
  auto expect = [&](uint64_t* full, uint32_t bytes_each) {
    if (rank == 0) mbar_expect_tx(full, 2 * bytes_each);
  };
  // 64 rows of two 64-column atoms: [2][64][64]
  auto load = [&](int dst, const CUtensorMap* tm, uint64_t* full, int row, int atom, int head) {
    tma_load_5d_pair(smem + dst, tm, leader(full), 0, row, atom, head, ti.b);
  };
  if (tid == 0 && n_iter > 0) {
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      if (i == 0) expect(k_full, 4 * Cfg::kKAtom);
      load(Cfg::kKOff + i * (2 * Cfg::kKAtom), &p.tm_k, k_full, n0, 2 * i, ti.hk);
    }
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      if (i == 0) expect(v_full, 4 * Cfg::kKAtom);
      load(Cfg::kVOff + i * (2 * Cfg::kKAtom), &p.tm_v, v_full, n0, 2 * i, ti.hk);
    }
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
      if (i == 0) expect(kcol_full, 4 * Cfg::kKAtom);
      load(Cfg::kKColOff + i * (2 * Cfg::kKAtom), &p.tm_k, kcol_full, ti.n0 + i * kKeys, 2 * rank, ti.hk);
    }
  }
  __syncthreads();
  tc_fence_after();
  early_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    if (warp == 0 && elect_one()) {
      // ---------------------------------------------------------------- loader
      // The ring in the order of the MMAs, one load a slot (and one place in the code: the roles of the CTA share the SM's
      // instruction cache).
      uint32_t slot = 0, phase = 1;
      Walk w{0, -1}, next{0, 0};
      bool ok = true;
#pragma unroll 1
      for (int it = -1; it < n_iter && ok; ++it) {
#pragma unroll 1
        for (int i = 0; i < 8 && ok; ++i) {
          const bool rows = (i & 2) != 0;  // dO columns, the next Q rows, Q columns, the next dO rows: two slots each
          if (rows ? it + 1 >= n_iter : it < 0) continue;
          const bool is_q = i >= 2 && i < 6;
          const Walk& at = rows ? next : w;
          const int row = (ti.m_start + at.mi) * kBlk + (rows ? rank : i & 1) * 64, atom = 2 * (rows ? i & 1 : rank);
          ok = mbar_wait(&ring_empty[slot], phase, ctl, kWaitBwd + 1);
          if (!ok) break;
          expect(&ring_full[slot], Cfg::kSlotBytes);
          load(Cfg::kRingOff + slot * Cfg::kSlotBytes, is_q ? &p.tm_q : &p.tm_do, &ring_full[slot], row, atom, ti.hk * p.group + at.g);
          if (++slot == Cfg::kSlots) {
            slot = 0;
            phase ^= 1;
          }
        }
        w = next;
        next = walk_next(next, ti.n_m);
      }
    } else if (warp == 1 && rank == 0 && elect_one()) {
      // ---------------------------------------------------------------- mma issuer, for both CTAs
      constexpr uint32_t kBase = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10);
      constexpr uint32_t idesc_qk = kBase | (static_cast<uint32_t>(kBlk >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
      constexpr uint32_t idesc_dv = kBase | (static_cast<uint32_t>(D >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24) | (1u << 16);
      constexpr uint32_t idesc_dq = kBase | (static_cast<uint32_t>(kBlk >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24) | (1u << 15) | (1u << 16);
      const uint64_t base = make_smem_desc(smem_u32(smem), 16, 1024);
      // MN-major operands: bytes between chunks of 64 along M or N
      constexpr uint64_t kMn = static_cast<uint64_t>((Cfg::kKAtom >> 4) - 1) << 16;
      const uint64_t k_d = base + (Cfg::kKOff >> 4), v_d = base + (Cfg::kVOff >> 4), kcol_d = base + (Cfg::kKColOff >> 4) + kMn;
      const uint64_t ring_d = base + (Cfg::kRingOff >> 4), p_d = base + (Cfg::kPOff >> 4);
      const uint64_t dsq_d = make_smem_desc_64(smem_u32(smem) + Cfg::kDSQOff, Cfg::kDSQChunk, 512);
      uint32_t slot = 0, ring_phase = 0;
      auto ring_wait = [&]() -> bool {
        if (!mbar_wait(&ring_full[slot], ring_phase, ctl, kWaitBwd + 4)) return false;
        tc_fence_after();
        return true;
      };
      auto ring_next = [&]() {
        mma_pair_commit(&ring_empty[slot]);
        if (++slot == Cfg::kSlots) {
          slot = 0;
          ring_phase ^= 1;
        }
      };
      // [128 keys x 128 q] over d, 128 a slot
      auto kmajor = [&](uint32_t d_tmem, uint64_t a) -> bool {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          if (!ring_wait()) return false;
          const uint64_t b = ring_d + slot * (Cfg::kSlotBytes >> 4), aa = a + i * (2 * Cfg::kKAtom >> 4);
          auto steps = [&](auto atom) {
            static_for<4>([&](auto ks) {
              constexpr uint32_t o = atom.value * (Cfg::kKAtom >> 4) + ks.value * 2;
              mma_pair_ss_o<o, o>(d_tmem, aa, b, idesc_qk, i + atom.value + ks.value > 0 ? 1u : 0u);
            });
          };
          steps(std::integral_constant<int, 0>{});
          if (ATOMS == 4 || i == 0) steps(std::integral_constant<int, 1>{});
          ring_next();
        }
        return true;
      };
      // [128 keys x d] over 128 q, 64 a slot
      auto accumulate = [&](uint32_t d_tmem, uint32_t acc) -> bool {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          if (!ring_wait()) return false;
          const uint64_t b = ring_d + kMn + slot * (Cfg::kSlotBytes >> 4), a = p_d + i * (Cfg::kKAtom >> 4);
          static_for<4>([&](auto ks) {
            mma_pair_ss_o<ks.value * 2, ks.value * (2048 >> 4)>(d_tmem, a, b, idesc_dv, i + ks.value > 0 ? 1u : acc);
          });
          ring_next();
        }
        return true;
      };
      bool ok = n_iter > 0;
#pragma unroll 1
      for (int it = -1; it < n_iter && ok; ++it) {
        const uint32_t ph = it & 1;
        const uint32_t acc = it > 0 ? 1u : 0u;
        const bool has_next = it + 1 < n_iter;
        // dV += P^T dO
        if (it >= 0) {
          ok = mbar_wait(p_full, ph, ctl, kWaitBwd + 6) && accumulate(tmem + Cfg::kTmemDV, acc);
          if (!ok) break;
          mma_pair_commit(dv_read);
        }
        // the next S^T: these scores have become P^T
        if (has_next) {
          ok = (it >= 0 || mbar_wait(k_full, 0, ctl, kWaitBwd + 3)) && kmajor(tmem + Cfg::kTmemS, k_d);
          if (!ok) break;
          mma_pair_commit(s_full);
        }
        // dK += dS^T Q
        if (it >= 0) {
          ok = mbar_wait(ds_full, ph, ctl, kWaitBwd + 7) && accumulate(tmem + Cfg::kTmemDK, acc);
          if (!ok) break;
          mma_pair_commit(dk_read);
        }
        if (has_next) {
          ok = (it >= 0 || mbar_wait(v_full, 0, ctl, kWaitBwd + 3)) && kmajor(tmem + Cfg::kTmemDP, v_d);
          if (!ok) break;
          mma_pair_commit(dp_full);
        }
        if (it < 0) continue;
        // dQ^T = K^T dS^T
        mbar_expect_tx(received, 2 * Cfg::kSendChunk);
        ok = (it > 0 ? mbar_wait(dq_free, ph ^ 1, ctl, kWaitBwd + 10) : mbar_wait(kcol_full, 0, ctl, kWaitBwd + 3)) &&
             mbar_wait(received, ph, ctl, kWaitBwd + 19) && mbar_wait(dsq_full, ph, ctl, kWaitBwd + 8);
        if (!ok) break;
        tc_fence_after();
        static_for<2 * kKeys / 16>([&](auto ks) {
          mma_pair_ss_o<(ks.value / 4) * (2 * Cfg::kKAtom >> 4) + (ks.value % 4) * (2048 >> 4), ks.value * (1024 >> 4)>(
              tmem + Cfg::kTmemDQ, kcol_d, dsq_d, idesc_dq, ks.value > 0 ? 1u : 0u);
        });
        mma_pair_commit(dq_full);
      }
      // Only for who waits: an arrival that nobody waits for could land in the other CTA after its end.
      if (ok) mma_pair_commit(dk_done);
    } else if (warp == 2 && rank == 1 && elect_one()) {
      // ---------------------------------------------------------------- tells the issuer what this CTA has received
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        mbar_expect_tx(received, 2 * Cfg::kSendChunk);
        ok = mbar_wait(received, it & 1, ctl, kWaitBwd + 19);
        if (ok) mbar_arrive_cluster(leader(dsq_full));
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- -LSE (log2 domain) and -delta of a query block
      bool ok = pair_statistics(p, ti, s_stat, stat_full, stat_empty, lane, ctl);
      // The slots' last commits land before the CTA ends (eight loads an iteration, so all of them are in odd phases), and dK's.
#pragma unroll 1
      for (int i = 0; i < Cfg::kSlots && ok; ++i) ok = mbar_wait(&ring_empty[i], 1, ctl, kWaitBwd + 1);
      if (ok) ok = mbar_wait(dk_read, (n_iter - 1) & 1, ctl, kWaitBwd + 17);
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ compute: one key and 32 queries a thread
    const int wg = (warp - 4) >> 2;
    const int quad = warp & 3;
    const int key_in = (quad & 1) * 32 + lane;
    const int qh = quad >> 1;  // which 64 queries of the block: those of CTA qh's dQ. The warpgroup has 32 of them.
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + Cfg::kTmemS + wg * 32;
    const uint32_t t_dp = tmem + lane_addr + Cfg::kTmemDP + wg * 32;
    const uint32_t p_bar = leader(p_full), ds_bar = leader(ds_full), dsq_bar = leader(dsq_full);
    const bool keeps = qh == rank;
    const int swz = key_in & 7, dsq_swz = (key_in >> 1) & 3;
    uint8_t* p_row = smem + Cfg::kPOff + qh * Cfg::kKAtom + key_in * 128;
    const int dsq_off = Cfg::kDSQOff + wg * Cfg::kDSQChunk + rank * Cfg::kSendChunk, send_off = Cfg::kSendOff + wg * Cfg::kSendChunk;
    uint8_t* dsq_row = smem + (keeps ? dsq_off : send_off) + key_in * 64;
    const uint32_t send_from = smem_u32(smem) + send_off + (quad & 1) * 2048;
    const uint32_t send_to = peer_smem(smem_u32(smem) + dsq_off + (quad & 1) * 2048, qh);
    const uint32_t send_bar = peer_smem(smem_u32(received), qh);
    const int kpos = n0 + key_in;
    const float inv_cap = FANCY && p.softcap > 0.f ? p.scale / p.softcap : 0.f;
    const float cap_l2 = p.softcap * kLog2e;
    bool ok = true;
    Walk w{0, 0};
    for (int it = 0; it < n_iter; ++it) {
      const int m0 = (ti.m_start + w.mi) * kBlk;
      const int hq = ti.hk * p.group + w.g;
      w = walk_next(w, ti.n_m);
      const uint32_t par = it & 1;
      const float* stat = s_stat + par * (2 * kBlk) + qh * 64 + wg * 32;
      const bool stat_ok = mbar_wait(&stat_full[par], (it >> 1) & 1, ctl, kWaitBwd + 15);  // voted on with s_full below
      const float4* lse4 = reinterpret_cast<const float4*>(stat);
      const float4* dl4 = reinterpret_cast<const float4*>(stat + kBlk);

      // ---- P^T = exp2(S^T c - lse)
      if (!__all_sync(0xffffffffu, mbar_wait(s_full, par, ctl, kWaitBwd + 11) && stat_ok)) { ok = false; break; }
      tc_fence_after();
      uint32_t sr[32];
      tmem_ld32(t_s, sr);
      tmem_wait_ld();
      tc_fence_before();
      const int qbase = m0 + qh * 64 + wg * 32;
      bool need_mask = (n0 + kKeys > p.seqlen_k);
      if (p.window_right >= 0) need_mask |= (n0 + kKeys - 1 > m0 + off + p.window_right);
      if (p.window_left >= 0) need_mask |= (n0 < m0 + kBlk - 1 + off - p.window_left);
      int q_lo = 0, q_hi = 32;  // which of the thread's queries see its key
      if (need_mask) {
        if (p.window_right >= 0) q_lo = kpos - off - p.window_right - qbase;
        if (p.window_left >= 0) q_hi = kpos - off + p.window_left + 1 - qbase;
        if (kpos >= p.seqlen_k) q_hi = -1;
      }
      float pr[32];  // what dP^T - delta is multiplied by: P^T times the derivative of the score transform
      if constexpr (!FANCY) {
        const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l4 = lse4[i / 4];
          unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, pack_f32x2(l4.x, l4.y)), pr[i], pr[i + 1]);
          unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), c2, pack_f32x2(l4.z, l4.w)), pr[i + 2], pr[i + 3]);
#pragma unroll
          for (int e = 0; e < 4; ++e) pr[i + e] = ex2(pr[i + e]);
        }
        if (need_mask) fill_outside<32>(pr, q_lo, q_hi, 0.f);
#pragma unroll
        for (int i = 0; i < 16; ++i) sr[i] = pack2<BF16>(pr[2 * i], pr[2 * i + 1]);
      } else {
        const float slope = p.alibi != nullptr ? p.alibi[ti.b * p.alibi_batch_stride + hq] * kLog2e : 0.f;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float pp[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float raw = __uint_as_float(sr[i + e]);
            float x, deriv = 1.f;
            if (p.softcap > 0.f) {
              const float t = tanh_approx(raw * inv_cap);
              x = cap_l2 * t;
              deriv = fmaf(-t, t, 1.f);
            } else {
              x = raw * p.scale_log2;
            }
            if (p.alibi != nullptr)
              x += p.causal_alibi ? slope * static_cast<float>(kpos) : -slope * fabsf(static_cast<float>(qbase + i + e + off - kpos));
            float pv = ex2(x + reinterpret_cast<const float*>(lse4)[i + e]);
            if (need_mask && (i + e < q_lo || i + e >= q_hi)) pv = 0.f;
            pp[e] = pv;
            pr[i + e] = pv * deriv;
          }
          sr[i / 2] = pack2<BF16>(pp[0], pp[1]);
        }
      }
      auto store_half_row = [&]() {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(p_row + (((wg * 4 + c) ^ swz) << 4)) = make_uint4(sr[4 * c], sr[4 * c + 1], sr[4 * c + 2], sr[4 * c + 3]);
      };
      if (it > 0 && !warp_wait(dk_read, par ^ 1, ctl, kWaitBwd + 17)) { ok = false; break; }
      store_half_row();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(p_bar);

      // ---- dS^T = P^T (dP^T - delta)
      if (!warp_wait(dp_full, par, ctl, kWaitBwd + 12)) { ok = false; break; }
      tc_fence_after();
      tmem_ld32(t_dp, sr);
      tmem_wait_ld();
      tc_fence_before();
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 d = dl4[i / 4];
        float a, b;
        unpack_f32x2(mul2(pack_f32x2(pr[i], pr[i + 1]),
                          add2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), pack_f32x2(d.x, d.y))), a, b);
        sr[i / 2] = pack2<BF16>(a, b);
        unpack_f32x2(mul2(pack_f32x2(pr[i + 2], pr[i + 3]),
                          add2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), pack_f32x2(d.z, d.w))), a, b);
        sr[i / 2 + 1] = pack2<BF16>(a, b);
      }
      // Over P^T and, for dQ, over dS^T of the iteration before: what is sent comes first.
      if (!warp_wait(dv_read, par, ctl, kWaitBwd + 18)) { ok = false; break; }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(dsq_row + ((c ^ dsq_swz) << 4)) = make_uint4(sr[4 * c], sr[4 * c + 1], sr[4 * c + 2], sr[4 * c + 3]);
      store_half_row();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (keeps) mbar_arrive_cluster(dsq_bar);
        else bulk_copy_cluster(send_to, send_from, 2048, send_bar);
        mbar_arrive_cluster(ds_bar);
        mbar_arrive(&stat_empty[par]);
      }
      __syncwarp();
    }
    // ---- epilogue: warpgroup 0 writes dK (scaled), warpgroup 1 writes dV, through the K and V tiles. A thread has half a row.
    if (ok && n_iter > 0) ok = warp_wait(dk_done, 0, ctl, kWaitBwd + 13);
    if (ok && n0 < p.seqlen_k) {
      tc_fence_after();
      const uint32_t t_acc = tmem + lane_addr + (wg == 0 ? Cfg::kTmemDK : Cfg::kTmemDV);
      const float mul = (wg == 0) ? p.scale : 1.f;
      uint8_t* stage = smem + (wg == 0 ? Cfg::kKOff : Cfg::kVOff);
#pragma unroll 1
      for (int h = 0; h < kHalf; h += 32) {
        uint32_t acc[32];
        if (n_iter > 0) {
          tmem_ld32(t_acc + h, acc);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = 0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            o[q] = pack2<BF16>(__uint_as_float(acc[8 * c + 2 * q]) * mul, __uint_as_float(acc[8 * c + 2 * q + 1]) * mul);
          const int chunk = (qh * kHalf + h) / 8 + c;
          *reinterpret_cast<uint4*>(stage + (chunk >> 3) * Cfg::kKAtom + key_in * 128 + (((chunk & 7) ^ swz) << 4)) =
              make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(&epi_full[wg]);
      if ((tid & 127) == 0 && mbar_wait(&epi_full[wg], 0, ctl, kWaitBwd + 16)) {
#pragma unroll
        for (int a = 0; a < ATOMS; ++a)
          if (a * 64 < p.head_dim) tma_store_4d(wg == 0 ? &p.tm_dk : &p.tm_dv, stage + a * Cfg::kKAtom, a * 64, ti.hk, n0, ti.b);
        tma_commit_group();
        tma_wait_group_read<0>();
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ dQ drain: one column of the head dim a thread
    const int dw = warp & 3;
    const int col = rank * kHalf + dw * 32;  // of the warp's first lane
    const bool used = col < p.head_dim;
    const uint32_t t_dq = tmem + (static_cast<uint32_t>(dw * 32) << 16) + Cfg::kTmemDQ;
    const uint32_t free_bar = leader(dq_free);
    uint8_t* stage = smem + Cfg::kDQOff + dw * (Cfg::kPieces * Cfg::kPieceBytes);
    int piece = 0;
    Walk w{0, 0};
    bool ok = true;
    for (int it = 0; it < n_iter; ++it, w = walk_next(w, ti.n_m)) {
      const int hq = ti.hk * p.group + w.g;
      const int row = (ti.m_start + w.mi) * kBlk;
      ok = warp_wait(dq_full, it & 1, ctl, kWaitBwd + 14);
      if (!ok) break;
      tc_fence_after();
      // In two halves of 64 queries; pieces of 16 queries roll through the warp's staging buffers, each free once the reduction three
      // before has read it.
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        uint32_t acc[64];
        tmem_ld32(t_dq + half * 64, acc);
        tmem_ld32(t_dq + half * 64 + 32, acc + 32);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (half == 1 && lane == 0) mbar_arrive_cluster(free_bar);
        if (!used) continue;
#pragma unroll
        for (int k = 0; k < 64 / Cfg::kPieceRows; ++k) {
          if (lane == 0) tma_wait_group_read<Cfg::kPieces - 1>();
          __syncwarp();
          uint8_t* buf = stage + piece * Cfg::kPieceBytes;
          piece = piece + 1 == Cfg::kPieces ? 0 : piece + 1;
#pragma unroll
          for (int q = 0; q < Cfg::kPieceRows; ++q)
            *reinterpret_cast<uint32_t*>(buf + q * 128 + (((lane >> 2) ^ (q & 7)) << 4) + (lane & 3) * 4) = acc[k * Cfg::kPieceRows + q];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int r = row + half * 64 + k * Cfg::kPieceRows;
            if (r < p.seqlen_q) tma_reduce_add_4d(&p.tm_dqa, buf, col, hq, r, ti.b);
            tma_commit_group();
          }
        }
      }
    }
    if (lane == 0) tma_wait_group_read<0>();
  }
  end_pair(p, abort_flag, tid, warp, tmem);
}

template <int ATOMS, bool BF16, bool FANCY>
cudaError_t launch_one(const BwdParams& p, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(bwd_wide_pair_kernel<ATOMS, BF16, FANCY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         WidePairCfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int64_t blocks = 2LL * p.num_nblk * p.batch * p.heads_k;
  if (blocks <= 0) return cudaSuccess;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  return launch_grid(true, bwd_wide_pair_kernel<ATOMS, BF16, FANCY>, dim3(static_cast<unsigned>(blocks)), kThreads, WidePairCfg::kSmemBytes,
                     stream, p);
}

template <int ATOMS, bool BF16>
cudaError_t pick_mode(const BwdParams& p, cudaStream_t stream) {
  return p.softcap > 0.f || p.alibi != nullptr ? launch_one<ATOMS, BF16, true>(p, stream) : launch_one<ATOMS, BF16, false>(p, stream);
}

}  // namespace

cudaError_t launch_bwd_wide_pair(const BwdParams& p, bool bf16, cudaStream_t stream) {
  if (p.head_dim == 192) return bf16 ? pick_mode<3, true>(p, stream) : pick_mode<3, false>(p, stream);
  if (p.head_dim == 256) return bf16 ? pick_mode<4, true>(p, stream) : pick_mode<4, false>(p, stream);
  return cudaErrorInvalidValue;
}

}  // namespace fa2
