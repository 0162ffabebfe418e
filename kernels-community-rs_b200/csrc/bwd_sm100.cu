// FlashAttention-2 backward for sm_100a (B200): dQ, dK, dV in one kernel.
//
// One CTA owns 128 keys of one (batch, kv head) and walks every 128-row query block (and every
// query head of the GQA group) that can see those keys. Everything is computed transposed, keys
// on the TMEM lanes, so that P^T feeds the dV MMA straight from TMEM:
//
//   S^T  = K Q^T            smem x smem  -> TMEM [keys x q]
//   dP^T = V dO^T           smem x smem  -> TMEM [keys x q]
//   P^T  = exp2(S^T c - lse)             compute warps, written back over S^T as 16-bit
//   dV  += P^T dO           TMEM x smem (dO as MN-major operand)
//   dS^T = P^T (dP^T - delta)            compute warps -> swizzled smem [keys x q]
//   dK  += dS^T Q           smem (K-major view of dS^T) x smem (Q MN-major)
//   dQ   = dS K             smem (MN-major view of dS^T) x smem (K MN-major) -> TMEM, aliasing dP^T
//   dQ tile -> registers -> smem -> cp.reduce.async.bulk (fp32 add) into the dQ accumulator
//
// TMEM: dK [0,D) dV [D,2D) S^T/P^T [256,384) dP^T/dQ [384,512).
// Warps: 0 loader (TMA), 1 MMA issuer, 4-11 compute (two warpgroups, 64 query columns each),
// 12-15 dQ drain, 3 statistics (-LSE and -delta of the next query block into shared memory), 2 fixer (packed batches).
// dK and dV are accumulated over the whole loop in TMEM and written once, so they
// need no atomics; the GQA heads are walked serially like the reference kernel does.
//
// What bounds it: the compute warps. An iteration takes 3500-4000 cycles against 2560 of MMA at D = 128, 1450 of them P^T
// and 1000 dS^T. The warps used to fetch LSE and delta themselves, behind a barrier of both warpgroups, and to do that
// arithmetic one value at a time; with a warp for the statistics and packed instructions forward and backward of B4 H16/4
// S2048 D128 softcap take 316 instead of 329 us, B16 H16 S2048 causal 1145 instead of 1154.
//
// A CTA's start and end cost 9000 cycles, a third of its time where a head has four query blocks. At D = 64 there is shared
// memory for K and V of two tiles, so a CTA goes on with the tile of a CTA that has not started: K, V, Q and dO of the next
// tile are loaded beside the end of this one. B32 H12 S509 D64 fp16 223.6 -> 201.0 us, B2 H16 S4096 D64 causal 378 -> 358.
// That includes what it costs: with the tile carried through every role these instances spill 312-344 bytes of loads a thread. So
// calls in which no CTA takes a tile over have instances without it (launch_one).
// At D = 128 K has to wait for the last dQ and nothing is left to stage dK and dV in: B4 H16 S1000 112.8 -> 114.8 us,
// B4 H16/4 S2048 softcap 340 -> 345, so there a CTA has one tile. Packed batches have one tile per CTA too.
//
// Replaces the reference kernels `backward` (dQ) and `backward_kv`
// (flash-attn2-rs/src/device/backward/dq.rs:12-302,438-576, dkv.rs:15-266,865-1012,
//  common.rs:121-152) and their packed variants (src/device/varlen/backward.rs:134-648), with
// fp32 dQ accumulation in global memory as in the reference's fused kernel (common.rs:248-252).
#include "sm100_ptx.cuh"
#include "fa2_params.h"
#include "fa2_launch.h"
#include "bwd_tile.cuh"

namespace fa2 {

namespace {

constexpr int kThreads = 512;
constexpr int kComputeRegs = 152;
constexpr int kDrainRegs = 152;
constexpr int kMiscRegs = 56;
// setmaxnreg moves registers inside the CTA's own allocation (128 per thread at launch: 65536 / 512). What the
// compute and drain warps take must not exceed what warps 0-3 give back: an increase beyond it never returns.
static_assert(8 * (kComputeRegs - 128) + 4 * (kDrainRegs - 128) <= 4 * (128 - kMiscRegs), "setmaxnreg: more registers asked for than released");

template <int D>
struct BwdCfg {
  static constexpr int kAtoms = D / 64;
  static constexpr int kTileBytes = kBlk * D * 2;
  // K and V of the next tile are loaded beside the end of this one where there is room for two of each.
  static constexpr int kKVStages = D == 128 ? 1 : 2;
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kKVStages * kTileBytes;
  static constexpr int kQOff = 2 * kKVStages * kTileBytes;  // 2 stages
  // The dQ pieces have staging buffers of their own. While they went through the retired dO stage (two stages at either
  // head dim), dO came back to the loader only after the reductions had read it, two thirds of an iteration late. At
  // D = 128 the staging takes the place of the second dO stage: one is enough, because dV, its last reader, is issued
  // most of an iteration before the next dP^T. Forward and backward together, causal bf16: B16 H16 S2048 1413 -> 1392 us,
  // B1 H32 S16384 7933 -> 7742.
  static constexpr int kDOStages = D == 128 ? 1 : 2;
  static constexpr int kDOOff = kQOff + 2 * kTileBytes;
  static constexpr int kDSOff = kDOOff + kDOStages * kTileBytes;  // [128 keys x 128 q] 16-bit
  static constexpr int kDSBytes = kBlk * kBlk * 2;
  static constexpr int kPieceBytes = kBlk * 128;   // dQ staging piece: [128 rows x 32 fp32]
  static constexpr int kPieces = 2;                // staging buffers: 4 KB per drain warp and piece
  static constexpr int kDQOff = kDSOff + kDSBytes;
  static constexpr int kBarOff = kDQOff + kPieces * kPieceBytes;
  static constexpr int kNumBars = 40;
  static constexpr int kMiscOff = (kBarOff + kNumBars * 8 + 15) / 16 * 16;  // what follows is read as float4
  static constexpr int kAnswerOff = kMiscOff + 16;     // what the scheduler answered
  static constexpr int kNextOff = kMiscOff + 32;       // [2] the CTA's next tile: twelve words
  static constexpr int kStatOff = kNextOff + 96;       // lse / delta: [2 buffers][2][128] fp32
  static constexpr int kSmemBytes = kStatOff + 2 * 2 * kBlk * 4;  // the dynamic window must start 1024-aligned
  static_assert(kStatOff % 16 == 0, "lse / delta are read as float4");
  static constexpr uint32_t kTmemDK = 0, kTmemDV = D, kTmemS = 256, kTmemDP = 384;
};

struct KvTile {
  int b, hk, n0;
  int sq, sk, q_row0, k_row0, bq, off;
  int m_start, n_m, n_iter;
  int g0, mi0;         // where the walk over (query head, query block) starts
  int part, parts;     // which part of a split key block this CTA is
  bool valid;
};

template <bool PACKED>
__device__ __forceinline__ KvTile get_kv_tile(const BwdParams& p, int t) {
  KvTile ti;
  // The key blocks of a group of heads are listed together, the first block of every head, then the second ...: with a
  // causal mask the first ones see the most query rows, so each group starts with its heaviest CTAs and ends with its
  // lightest (bwd_head_group: how many heads, and what it gives).
  const int per_head = !PACKED && p.dk_part != nullptr ? p.items_per_head : p.num_nblk;
  const int first_bh = t / (p.head_group * per_head) * p.head_group;
  const int n_bh = min(p.head_group, p.batch * p.heads_k - first_bh);
  const int in_group = t - first_bh * per_head;
  const int i = in_group / n_bh;
  const int bh = first_bh + in_group - i * n_bh;
  int nblk = i;
  ti.part = 0;
  ti.parts = 1;
  if (!PACKED && p.dk_part != nullptr) {
    // The parts of all key blocks of a head, block by block.
    int lo = 0, hi = p.num_nblk;  // part_start[lo] <= i < part_start[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (p.part_start[mid] <= i) lo = mid;
      else hi = mid;
    }
    nblk = lo;
    ti.part = i - p.part_start[lo];
    ti.parts = p.part_start[lo + 1] - p.part_start[lo];
  }
  // Ordered dQ accumulation waits for the higher key blocks of the same head. CTAs start in grid order, so
  // there the highest key block comes first: a CTA only ever waits for CTAs that were started before it,
  // whatever the number of key blocks and of resident CTAs.
  if (PACKED && p.dq_turn != nullptr) nblk = p.num_nblk - 1 - nblk;
  ti.b = bh / p.heads_k;
  ti.hk = bh - ti.b * p.heads_k;
  ti.n0 = nblk * kBlk;
  if (PACKED) {
    ti.q_row0 = p.cu_q[ti.b];
    ti.sq = p.cu_q[ti.b + 1] - ti.q_row0;
    ti.k_row0 = p.cu_k[ti.b];
    ti.sk = p.cu_k[ti.b + 1] - ti.k_row0;
    ti.bq = 0;
    if (ti.sq < 0 || ti.sk < 0 || ti.sq > p.seqlen_q || ti.sk > p.seqlen_k) ti.sk = 0;
  } else {
    ti.q_row0 = 0;
    ti.k_row0 = 0;
    ti.sq = p.seqlen_q;
    ti.sk = p.seqlen_k;
    ti.bq = ti.b;
  }
  ti.off = ti.sk - ti.sq;
  ti.valid = ti.n0 < ti.sk;
  q_block_range(p, ti.sq, ti.sk, ti.n0, kBlk, ti.m_start, ti.n_m);
  ti.n_iter = ti.n_m * p.group;
  ti.g0 = ti.mi0 = 0;
  if (ti.parts > 1) {
    const int first = ti.n_iter * ti.part / ti.parts;
    ti.n_iter = ti.n_iter * (ti.part + 1) / ti.parts - first;
    ti.g0 = first / ti.n_m;
    ti.mi0 = first - ti.g0 * ti.n_m;
  }
  return ti;
}

// MODE: what is done to the scores; PACKED: cu_seqlens batches. Both are compile-time so that the plain dense
// kernel carries none of their code: at 156 KB the all-in-one kernel missed the SM's instruction cache on a
// quarter of its fetches and ran 6-9 % slower than the 62 KB one.
// TAKE_OVER: a CTA goes on with tiles of CTAs that have not started. Calls in which no CTA does have instances without the code.
template <int D, bool BF16, int MODE, bool PACKED, bool TAKE_OVER>
__global__ void __launch_bounds__(kThreads, 1) bwd_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = BwdCfg<D>;
  static_assert(!TAKE_OVER || (Cfg::kKVStages == 2 && !PACKED), "the next tile needs K and V stages of its own");
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    early_wait();
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, kWaitNone + 1);
    return;
  }
  uint8_t* s_k = smem + Cfg::kKOff;
  uint8_t* s_v = smem + Cfg::kVOff;
  uint8_t* s_q = smem + Cfg::kQOff;
  uint8_t* s_do = smem + Cfg::kDOOff;
  uint8_t* s_ds = smem + Cfg::kDSOff;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOff);
  uint64_t* k_full = bars + 0;     // [2] K has landed (V has a barrier of its own: the first S^T needs only K and Q)
  uint64_t* v_full = bars + 2;     // [2]
  uint64_t* k_empty = bars + 4;    // [2] the tile's last dQ has read K
  uint64_t* v_empty = bars + 6;    // [2] its last dP^T has read V
  uint64_t* q_full = bars + 8;     // [2]
  uint64_t* q_empty = bars + 10;   // [2] dK has read the stage (and, in packed batches, the fixer has seen it)
  uint64_t* do_full = bars + 12;   // [2]
  uint64_t* do_empty = bars + 14;  // [2] dV has read the stage (and, in packed batches, the fixer has seen it)
  uint64_t* s_full = bars + 16;
  uint64_t* p_full = bars + 17;
  uint64_t* dp_full = bars + 18;
  uint64_t* ds_full = bars + 19;
  uint64_t* dq_full = bars + 20;
  uint64_t* dq_free = bars + 21;
  uint64_t* dkv_done = bars + 22;
  uint64_t* dv_done = bars + 23;   // the last dV MMA has completed (dK still has one GEMM to go)
  uint64_t* stat_full = bars + 24;   // [2]
  uint64_t* stat_empty = bars + 26;  // [2]
  uint64_t* next_full = bars + 28;   // [2] the loader has written down the next tile
  uint64_t* next_empty = bars + 30;  // [2] every role has read it
  uint64_t* kv_fixed = bars + 32;  // packed batches: the fixer warp has cleared the rows past the sequence
  uint64_t* q_fixed = bars + 33;   // [2]
  uint64_t* do_fixed = bars + 35;  // [2]
  uint64_t* epi_full = bars + 37;  // [2] packed batches: dK, dV are staged for their bulk store
  uint64_t* answered = bars + 39;  // the scheduler has answered
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff + 8);
  float* s_stat = reinterpret_cast<float*>(smem + Cfg::kStatOff);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const WaitCtl ctl{abort_flag};
  const KvTile first_tile = get_kv_tile<PACKED>(p, blockIdx.x);
  if (!first_tile.valid) return;
  const bool want_dq = (p.which & 1) != 0;
  // A dQ-only call skips the dV and dK GEMMs (their commits still hand the stages back). Only packed ones come here: dense
  // ones have bwd_dq_sm100.cu.
  const bool want_dkv = !PACKED || (p.which & 2) != 0;

  // Descriptor fetches start first: they are the head of the latency chain of the first loads.
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
      if (bar == p_full || bar == ds_full) count = 256;
      if (bar == dq_free || bar == epi_full || bar == epi_full + 1) count = kBlk;
      if (bar == stat_empty || bar == stat_empty + 1) count = 8;    // compute warps
      if (bar == next_empty || bar == next_empty + 1) count = want_dq ? 14 : 10;  // issuer, statistics, compute, drain warps
      if (PACKED && (bar == q_empty || bar == q_empty + 1 || bar == do_empty || bar == do_empty + 1)) count = 2;  // the commit and the fixer
      mbar_init(bar, count);
    }
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
    __syncwarp();
  }
  if (tid == 0) {
    // The first loads go out before the rest of the CTA is set up (TMEM allocation, the block-wide
    // barrier): their latency is the longest item of a CTA's start.
    early_wait();
    const KvTile& ti = first_tile;
    if (ti.n_iter > 0) {
      const int hq0 = ti.hk * p.group + ti.g0;
      const int m00 = (ti.m_start + ti.mi0) * kBlk;
      mbar_expect_tx(k_full, Cfg::kTileBytes);
      mbar_expect_tx(v_full, Cfg::kTileBytes);
      mbar_expect_tx(q_full, Cfg::kTileBytes);
      mbar_expect_tx(do_full, Cfg::kTileBytes);
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a) {
        tma_load_4d(s_k + a * (kBlk * 128), &p.tm_k, k_full, a * 64, ti.hk, ti.k_row0 + ti.n0, ti.bq);
        tma_load_4d(s_q + a * (kBlk * 128), &p.tm_q, q_full, a * 64, hq0, ti.q_row0 + m00, ti.bq);
      }
#pragma unroll
      for (int a = 0; a < Cfg::kAtoms; ++a) {
        tma_load_4d(s_v + a * (kBlk * 128), &p.tm_v, v_full, a * 64, ti.hk, ti.k_row0 + ti.n0, ti.bq);
        tma_load_4d(s_do + a * (kBlk * 128), &p.tm_do, do_full, a * 64, hq0, ti.q_row0 + m00, ti.bq);
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  early_wait();
  __syncthreads();
  tc_fence_after();
  if (!PACKED) early_trigger();
  const uint32_t tmem = *tmem_slot;

  // Dense calls: a CTA that has finished a tile goes on with one that has not started yet (the scheduler hands it the
  // grid index of a CTA that it then leaves out). The loader asks and writes the tile down, every role reads it. Barriers,
  // stages and TMEM carry on: the counters of a role, iterations, tiles with iterations and tiles, run through all its tiles.
  struct Pos {
    uint32_t it0 = 0, kv = 0, n = 0;
  };
  volatile int4* s_next = reinterpret_cast<volatile int4*>(smem + Cfg::kNextOff);
  // false: no more tiles, or a wait ran out
  auto next_tile = [&](KvTile& ti, Pos& pos) -> bool {
    pos.it0 += ti.n_iter;
    pos.kv += ti.n_iter > 0 ? 1 : 0;
    const uint32_t slot = pos.n & 1;
    if (!mbar_wait(&next_full[slot], (pos.n >> 1) & 1, ctl, kWaitBwd + 24)) return false;
    ++pos.n;
    const volatile int4* a = s_next + slot * 3;
    ti.b = ti.bq = a[0].x;
    ti.hk = a[0].y;
    ti.n0 = a[0].z;
    ti.n_iter = a[0].w;
    ti.m_start = a[1].x;
    ti.n_m = a[1].y;
    ti.g0 = a[1].z;
    ti.mi0 = a[1].w;
    ti.part = a[2].x;
    ti.parts = a[2].y;
    return ti.n_iter >= 0;
  };
  auto next_tile_warp = [&](KvTile& ti, Pos& pos) -> bool {
    const uint32_t slot = pos.n & 1;
    const bool more = next_tile(ti, pos);
    __syncwarp();
    if (lane == 0) mbar_arrive(&next_empty[slot]);
    return __all_sync(0xffffffffu, more);
  };

  if (warp < 4) {
    reg_dealloc<kMiscRegs>();
    if (warp == 0 && elect_one()) {
      // ---------------------------------------------------------------- loader
      // K, V and the first Q / dO tiles of the first tile were requested during set-up.
      bool ok = true;
      KvTile ti = first_tile;
      Pos pos;
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* full, int head, int row) {
        mbar_expect_tx(full, Cfg::kTileBytes);
#pragma unroll
        for (int a = 0; a < Cfg::kAtoms; ++a) tma_load_4d(dst + a * (kBlk * 128), tm, full, a * 64, head, row, ti.bq);
      };
      do {
        const uint32_t ks = pos.kv % Cfg::kKVStages, kph = (pos.kv / Cfg::kKVStages) & 1;
        Walk w{ti.g0, ti.mi0};
        for (int it = 0; it < ti.n_iter || it == 0; ++it) {
          if (TAKE_OVER && it + 1 >= ti.n_iter) {
            mbar_expect_tx(answered, 16);
            ask_next_cta(smem_u32(smem + Cfg::kAnswerOff), answered);
          }
          if (ti.n_iter == 0) break;
          if (it > 0) w = walk_next(w, ti.n_m);
          else if (pos.n == 0) continue;
          const int hq = ti.hk * p.group + w.g;
          const int row = ti.q_row0 + (ti.m_start + w.mi) * kBlk;
          const uint32_t gi = pos.it0 + it;
          const uint32_t st = gi & 1, dst = gi % Cfg::kDOStages;
          ok = mbar_wait(&q_empty[st], ((gi >> 1) & 1) ^ 1, ctl, kWaitBwd + 1);
          if (!ok) break;
          load(s_q + st * Cfg::kTileBytes, &p.tm_q, &q_full[st], hq, row);
          if (it == 0) {
            ok = mbar_wait(&v_empty[ks], kph ^ 1, ctl, kWaitBwd + 26);
            if (!ok) break;
            load(s_v + ks * Cfg::kTileBytes, &p.tm_v, &v_full[ks], ti.hk, ti.k_row0 + ti.n0);
          }
          ok = mbar_wait(&do_empty[dst], ((gi / Cfg::kDOStages) & 1) ^ 1, ctl, kWaitBwd + 2);
          if (!ok) break;
          load(s_do + dst * Cfg::kTileBytes, &p.tm_do, &do_full[dst], hq, row);
          if (it == 0) {
            ok = mbar_wait(&k_empty[ks], kph ^ 1, ctl, kWaitBwd + 27);
            if (!ok) break;
            load(s_k + ks * Cfg::kTileBytes, &p.tm_k, &k_full[ks], ti.hk, ti.k_row0 + ti.n0);
          }
        }
        if (!TAKE_OVER || !ok) break;
        // The tile after this one.
        const uint32_t slot = pos.n & 1;
        ok = mbar_wait(answered, pos.n & 1, ctl, kWaitBwd + 24) &&
             mbar_wait(&next_empty[slot], ((pos.n >> 1) & 1) ^ 1, ctl, kWaitBwd + 25);
        if (!ok) break;
        ++pos.n;
        pos.it0 += ti.n_iter;
        pos.kv += ti.n_iter > 0 ? 1 : 0;
        const int t = next_cta(smem_u32(smem + Cfg::kAnswerOff));
        if (t >= 0) ti = get_kv_tile<PACKED>(p, t);
        else ti.n_iter = -1;
        volatile int* a = reinterpret_cast<volatile int*>(s_next + slot * 3);
        a[0] = ti.b;
        a[1] = ti.hk;
        a[2] = ti.n0;
        a[3] = ti.n_iter;
        a[4] = ti.m_start;
        a[5] = ti.n_m;
        a[6] = ti.g0;
        a[7] = ti.mi0;
        a[8] = ti.part;
        a[9] = ti.parts;
        mbar_arrive(&next_full[slot]);
      } while (ti.n_iter >= 0);
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
      }
    } else if (warp == 1 && elect_one()) {
      // ---------------------------------------------------------------- mma issuer
      // Descriptors are built once; in the loops an operand address is one 64-bit add of a constant
      // (the descriptor's address field counts 16-byte units).
      constexpr uint32_t kBase = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) |
                                 (static_cast<uint32_t>(kBlk >> 4) << 24);
      constexpr uint32_t idesc_qk = kBase | (static_cast<uint32_t>(kBlk >> 3) << 17);             // S^T, dP^T
      constexpr uint32_t idesc_dv = kBase | (static_cast<uint32_t>(D >> 3) << 17) | (1u << 16);   // dV, dK: B MN-major
      constexpr uint32_t idesc_dq = idesc_dv | (1u << 15);                                        // dQ: A and B MN-major
      constexpr uint32_t kTile16 = Cfg::kTileBytes >> 4;
      constexpr uint32_t kAtom16 = (kBlk * 128) >> 4;
      // One base descriptor (K-major view of the start of shared memory); every operand is that
      // plus a constant: its byte offset / 16, and for the MN-major views the larger leading offset.
      const uint64_t base = make_smem_desc(smem_u32(smem), 16, 1024);
      constexpr uint64_t kMn = static_cast<uint64_t>(((kBlk * 128) >> 4) - 1) << 16;
      const uint64_t k0_kmaj = base + (Cfg::kKOff >> 4), v0_kmaj = base + (Cfg::kVOff >> 4);
      const uint64_t q_kmaj = base + (Cfg::kQOff >> 4), q_mn = q_kmaj + kMn;
      const uint64_t do_kmaj = base + (Cfg::kDOOff >> 4), do_mn = do_kmaj + kMn;
      const uint64_t ds_kmaj = base + (Cfg::kDSOff >> 4), ds_mn = ds_kmaj + kMn;
      // [keys x q] = A[keys x d] B[q x d]^T, both K-major, over d in steps of 16
      auto kmajor_pair = [&](uint32_t d_tmem, uint64_t a, uint64_t b) {
        static_for<D / 16>([&](auto ks) {
          constexpr uint32_t o = (ks.value / 4) * kAtom16 + (ks.value % 4) * 2;
          mma_ss_o<o, o>(d_tmem, a, b, idesc_qk, ks.value > 0 ? 1u : 0u);
        });
      };
      // Packed batches: a tile that reaches past the end of its sequence holds rows of the next sequence; it
      // is usable once the fixer warp has cleared them. bit st of *_par: parity of the stage's next fix.
      constexpr bool packed = PACKED;
      KvTile ti = first_tile;
      Pos pos;
      uint32_t qfix_par = 0, dofix_par = 0;
      auto ragged_q = [&](int mi) { return packed && (ti.m_start + mi) * kBlk + kBlk > ti.sq; };
      auto q_ready = [&](int mi, uint32_t st, uint32_t ph, int code) -> bool {
        if (!mbar_wait(&q_full[st], ph, ctl, code)) return false;
        if (!ragged_q(mi)) return true;
        const uint32_t par = (qfix_par >> st) & 1;
        qfix_par ^= 1u << st;
        return mbar_wait(&q_fixed[st], par, ctl, kWaitBwd + 21);
      };
      auto do_ready = [&](int mi, uint32_t st, uint32_t ph, int code) -> bool {
        if (!mbar_wait(&do_full[st], ph, ctl, code)) return false;
        if (!ragged_q(mi)) return true;
        const uint32_t par = (dofix_par >> st) & 1;
        dofix_par ^= 1u << st;
        return mbar_wait(&do_fixed[st], par, ctl, kWaitBwd + 22);
      };
      bool ok = true;
      do {
        const int n_iter = ti.n_iter;
        const uint32_t ks = pos.kv % Cfg::kKVStages, kph = (pos.kv / Cfg::kKVStages) & 1;
        const uint64_t k_kmaj = k0_kmaj + ks * kTile16, k_mn = k_kmaj + kMn, v_kmaj = v0_kmaj + ks * kTile16;
        // From one iteration before the first, of which only the next S^T and dP^T exist: the steps have one place in the code.
        Walk wn{ti.g0, ti.mi0};  // position of iteration it + 1
#pragma unroll 1
        for (int it = -1; it < n_iter && ok; ++it) {
          if (it >= 0) wn = walk_next(wn, ti.n_m);
          const uint32_t gi = pos.it0 + it;
          const uint32_t st = gi & 1;
          const uint32_t nph = ((gi + 1) >> 1) & 1;  // phase of the Q stage barriers of the next iteration
          const uint32_t dst = gi % Cfg::kDOStages, ndst = (gi + 1) % Cfg::kDOStages;
          const uint32_t ndph = ((gi + 1) / Cfg::kDOStages) & 1;
          const bool has_next = it + 1 < n_iter;
          const uint32_t acc = it > 0 ? 1u : 0u;
          // dV += P^T dO   (P^T: two 32-column halves at S + 0 and S + 64)
          if (it >= 0) {
            ok = mbar_wait(p_full, gi & 1, ctl, kWaitBwd + 6);
            if (!ok) break;
            tc_fence_after();
            if (want_dkv) {
              const uint64_t b = do_mn + dst * kTile16;
              static_for<kBlk / 16>([&](auto ks) {
                mma_ts_o<(ks.value / 4) * 64 + (ks.value % 4) * 8, ks.value * (2048 >> 4)>(
                    tmem + Cfg::kTmemDV, tmem + Cfg::kTmemS, b, idesc_dv, ks.value > 0 ? 1u : acc);
              });
            }
            mma_commit(&do_empty[dst]);
            if (!has_next) {
              mma_commit(dv_done);  // dV is final: its epilogue runs beside the last dQ and dK GEMMs
              mma_commit(&v_empty[ks]);
            }
          } else if (has_next) {
            ok = mbar_wait(&k_full[ks], kph, ctl, kWaitBwd + 3);
            if (ok && packed && ti.n0 + kBlk > ti.sk) ok = mbar_wait(kv_fixed, 0, ctl, kWaitBwd + 20);
            if (!ok) break;
          }
          // S^T of the next iteration right behind dV, the last reader of P^T: the scores are there when the
          // compute warps come out of phase B.
          if (has_next) {
            ok = q_ready(wn.mi, st ^ 1, nph, kWaitBwd + 8);
            if (!ok) break;
            tc_fence_after();
            kmajor_pair(tmem + Cfg::kTmemS, k_kmaj, q_kmaj + (st ^ 1) * kTile16);
            mma_commit(s_full);
          }
          // dQ = dS K   (into the dP^T columns, which the compute warps have drained)
          if (it >= 0) {
            ok = mbar_wait(ds_full, gi & 1, ctl, kWaitBwd + 7);
            if (!ok) break;
            tc_fence_after();
            if (want_dq) {
              static_for<kBlk / 16>([&](auto ks) {
                mma_ss_o<ks.value * (2048 >> 4), ks.value * (2048 >> 4)>(tmem + Cfg::kTmemDP, ds_mn, k_mn, idesc_dq,
                                                                          ks.value > 0 ? 1u : 0u);
              });
              mma_commit(dq_full);
            }
            if (!has_next) mma_commit(&k_empty[ks]);
            // dK += dS^T Q
            if (want_dkv) {
              const uint64_t b = q_mn + st * kTile16;
              static_for<kBlk / 16>([&](auto ks) {
                mma_ss_o<(ks.value / 4) * kAtom16 + (ks.value % 4) * 2, ks.value * (2048 >> 4)>(
                    tmem + Cfg::kTmemDK, ds_kmaj, b, idesc_dv, ks.value > 0 ? 1u : acc);
              });
            }
            mma_commit(&q_empty[st]);
          }
          // dP^T of the next iteration, once the dQ tile, or the last one of the tile before, has left TMEM
          if (has_next) {
            ok = do_ready(wn.mi, ndst, ndph, kWaitBwd + 9);
            if (ok && it < 0) ok = mbar_wait(&v_full[ks], kph, ctl, kWaitBwd + 3);
            if (ok && want_dq && gi + 1 > 0) ok = mbar_wait(dq_free, gi & 1, ctl, kWaitBwd + 10);
            if (!ok) break;
            tc_fence_after();
            kmajor_pair(tmem + Cfg::kTmemDP, v_kmaj, do_kmaj + ndst * kTile16);
            mma_commit(dp_full);
          }
        }
        if (ok && n_iter > 0) mma_commit(dkv_done);
        if (!ok || !TAKE_OVER) break;
        const uint32_t slot = pos.n & 1;
        ok = next_tile(ti, pos);
        mbar_arrive(&next_empty[slot]);
      } while (ok);
    } else if (PACKED && warp == 2 && first_tile.n_iter > 0) {
      const KvTile& ti = first_tile;
      const int n_iter = ti.n_iter;
      // ---------------------------------------------------------------- fixer (packed batches)
      // The reference zero-fills the rows of a tile that lie past the end of the sequence while staging it
      // (flash-attn2-rs/src/device/varlen/backward.rs:134-648 through the zfill copies of
      // src/device/forward/mod.rs:171-175); the TMA boxes here carry the next sequence's rows instead, and
      // a zero probability times a NaN or Inf of a neighbour would still poison dK, dV and dQ. This warp
      // waits for every Q and dO tile (which keeps it in step with the loader) and clears the stray rows
      // of those that need it, and of K and V once.
      auto clear_rows = [&](uint8_t* tile, int first) {
        for (int r = first + (lane >> 3); r < kBlk; r += 4)
#pragma unroll
          for (int a = 0; a < Cfg::kAtoms; ++a)
            *reinterpret_cast<uint4*>(tile + a * (kBlk * 128) + r * 128 + (lane & 7) * 16) = make_uint4(0, 0, 0, 0);
      };
      auto publish = [&](uint64_t* bar) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
        __syncwarp();
      };
      bool ok = true;
      const int kv_first = ti.sk - ti.n0;
      if (kv_first < kBlk) {
        ok = __all_sync(0xffffffffu, mbar_wait(k_full, 0, ctl, kWaitBwd + 3) && mbar_wait(v_full, 0, ctl, kWaitBwd + 3));
        if (ok) {
          clear_rows(s_k, kv_first);
          clear_rows(s_v, kv_first);
          publish(kv_fixed);
        }
      }
      Walk w{ti.g0, ti.mi0};
      for (int it = 0; it < n_iter && ok; ++it, w = walk_next(w, ti.n_m)) {
        const int first = ti.sq - (ti.m_start + w.mi) * kBlk;
        const uint32_t st = it & 1, ph = (it >> 1) & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&q_full[st], ph, ctl, kWaitBwd + 4));
        if (ok && first < kBlk) {
          clear_rows(s_q + st * Cfg::kTileBytes, first);
          publish(&q_fixed[st]);
        }
        // No stage is refilled before this warp has seen it: its waits go by phase parity.
        if (ok && lane == 0) mbar_arrive(&q_empty[st]);
        __syncwarp();
        const uint32_t dst = it % Cfg::kDOStages;
        ok = ok && __all_sync(0xffffffffu, mbar_wait(&do_full[dst], (it / Cfg::kDOStages) & 1, ctl, kWaitBwd + 5));
        if (ok && first < kBlk) {
          clear_rows(s_do + dst * Cfg::kTileBytes, first);
          publish(&do_fixed[dst]);
        }
        if (ok && lane == 0) mbar_arrive(&do_empty[dst]);
        __syncwarp();
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- -LSE (log2 domain) and -delta of a query block
      // Rows past the sequence give P = 0. Two buffers: the values of the next iteration, and of the next tile, are in
      // shared memory before the compute warps ask for them.
      KvTile ti = first_tile;
      Pos pos;
      bool ok = true;
      do {
        Walk w{ti.g0, ti.mi0};
        for (int it = 0; it < ti.n_iter && ok; ++it, w = walk_next(w, ti.n_m)) {
          const int hq = ti.hk * p.group + w.g, q0 = (ti.m_start + w.mi) * kBlk + lane;
          const float* lse = p.lse + ti.bq * p.lse_batch_stride + hq * p.lse_head_stride + ti.q_row0;
          const float* delta = p.delta + ti.bq * p.delta_batch_stride + hq * p.delta_head_stride + ti.q_row0 + ti.b * p.delta_seq_pad;
          float v[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int q = q0 + 32 * i;
            v[i] = q < ti.sq ? lse[q] * -kLog2e : -INFINITY;
            v[4 + i] = q < ti.sq ? -delta[q] : 0.f;
          }
          const uint32_t gi = pos.it0 + it, buf = gi & 1;
          ok = warp_wait(&stat_empty[buf], ((gi >> 1) & 1) ^ 1, ctl, kWaitBwd + 15);
          float* stat = s_stat + buf * (2 * kBlk) + lane;
#pragma unroll
          for (int i = 0; i < 8; ++i) stat[32 * i] = v[i];
          __syncwarp();
          if (lane == 0) mbar_arrive(&stat_full[buf]);
        }
      } while (TAKE_OVER && ok && next_tile_warp(ti, pos));
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ compute
    reg_alloc<kComputeRegs>();
    const int cw = warp - 4;
    const int wg = cw >> 2;                 // which 64 query columns
    const int key_in = (cw & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((cw & 3) * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + Cfg::kTmemS + wg * 64;
    const uint32_t t_dp = tmem + lane_addr + Cfg::kTmemDP + wg * 64;
    bool ok = true;
    constexpr bool fancy = MODE == kScoreAny;
    const float inv_cap1 = MODE == kScoreSoftcap ? p.scale / p.softcap : 0.f;
    const float cap1 = p.softcap * kLog2e;
    KvTile ti = first_tile;
    Pos pos;
    do {
      const int n_iter = ti.n_iter;
      const int kpos = ti.n0 + key_in;
      Walk w{ti.g0, ti.mi0};
      for (int it = 0; it < n_iter; ++it) {
        const int m0 = (ti.m_start + w.mi) * kBlk;
        const int g_cur = w.g;
        w = walk_next(w, ti.n_m);
        const uint32_t gi = pos.it0 + it, par = gi & 1;
        const float* stat = s_stat + par * (2 * kBlk);
        const bool stat_ok = mbar_wait(&stat_full[par], (gi >> 1) & 1, ctl, kWaitBwd + 15);  // voted on with s_full below
        const float4* lse4 = reinterpret_cast<const float4*>(stat + wg * 64);
        const float4* dl4 = reinterpret_cast<const float4*>(stat + kBlk + wg * 64);

        // ---- phase A: P^T = exp2(S^T c - lse)
        if (!__all_sync(0xffffffffu, mbar_wait(s_full, par, ctl, kWaitBwd + 11) && stat_ok)) { ok = false; break; }
        tc_fence_after();
        uint32_t sr[64];
        tmem_ld32(t_s, sr);
        tmem_ld32(t_s + 32, sr + 32);
        tmem_wait_ld();
        const int qbase = m0 + wg * 64;
        bool need_mask = (ti.n0 + kBlk > ti.sk);
        if (p.window_right >= 0) need_mask |= (ti.n0 + kBlk - 1 > m0 + ti.off + p.window_right);
        if (p.window_left >= 0) need_mask |= (ti.n0 < m0 + kBlk - 1 + ti.off - p.window_left);
        int c_lo = 0, c_hi = 64;
        if (need_mask) {
          if (p.window_right >= 0) c_lo = kpos - ti.off - p.window_right - qbase;
          if (p.window_left >= 0) c_hi = kpos - ti.off + p.window_left + 1 - qbase;
          if (kpos >= ti.sk) c_hi = -1;
        }
        float pr[64];
        if constexpr (MODE == kScoreSoftcap) {
          // P = exp2(cap tanh - lse); dS takes P times the derivative of the cap, 1 - tanh^2.
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const float4 l4 = lse4[i / 4];
            const float l[4] = {l4.x, l4.y, l4.z, l4.w};
            float pp[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float t = tanh_approx(__uint_as_float(sr[i + e]) * inv_cap1);
              pp[e] = ex2(fmaf(t, cap1, l[e]));
              if (need_mask && (i + e < c_lo || i + e >= c_hi)) pp[e] = 0.f;
              pr[i + e] = pp[e] * fmaf(-t, t, 1.f);
            }
            sr[i / 2] = pack2<BF16>(pp[0], pp[1]);
            sr[i / 2 + 1] = pack2<BF16>(pp[2], pp[3]);
          }
        } else if (!fancy) {
          // The bias of a key is the same for all queries in the causal form of ALiBi.
          float slope1 = 0.f, bias1 = 0.f;
          if constexpr (MODE == kScoreAlibi) {
            slope1 = p.alibi[ti.b * p.alibi_batch_stride + ti.hk * p.group + g_cur] * kLog2e;
            bias1 = slope1 * static_cast<float>(kpos);
            if (!p.causal_alibi) {
              const float dist = static_cast<float>(qbase + ti.off - kpos);
              bias1 = 0.f;
#pragma unroll
              for (int i = 0; i < 64; ++i)
                sr[i] = __float_as_uint(fmaf(-slope1, fabsf(dist + static_cast<float>(i)), __uint_as_float(sr[i]) * p.scale_log2));
            }
          }
          const float mul1 = MODE == kScoreAlibi && !p.causal_alibi ? 1.f : p.scale_log2;
          const uint64_t c2 = pack_f32x2(mul1, mul1), bias2 = pack_f32x2(bias1, bias1);
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const float4 l4 = lse4[i / 4];
            uint64_t n0 = pack_f32x2(l4.x, l4.y), n1 = pack_f32x2(l4.z, l4.w);
            if constexpr (MODE == kScoreAlibi) {
              n0 = add2(n0, bias2);
              n1 = add2(n1, bias2);
            }
            unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, n0), pr[i], pr[i + 1]);
            unpack_f32x2(fma2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), c2, n1), pr[i + 2], pr[i + 3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) pr[i + e] = ex2(pr[i + e]);
          }
          if (need_mask) {
            fill_outside<64>(pr, c_lo, c_hi, 0.f);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) sr[i] = pack2<BF16>(pr[2 * i], pr[2 * i + 1]);
        } else {
          // softcap / ALiBi: P follows the transformed scores of the forward; what goes on to dS is
          // P times the derivative of the transform, 1 - tanh^2 (the ALiBi bias is a constant).
          const int hq = ti.hk * p.group + g_cur;
          const float slope = (p.alibi != nullptr) ? p.alibi[ti.b * p.alibi_batch_stride + hq] * kLog2e : 0.f;
          const float inv_cap = (p.softcap > 0.f) ? p.scale / p.softcap : 0.f;
          const float cap_l2 = p.softcap * kLog2e;
#pragma unroll
          for (int i = 0; i < 64; i += 2) {
            float pp[2], dd[2];
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
                x += p.causal_alibi ? slope * static_cast<float>(kpos)
                                    : -slope * fabsf(static_cast<float>(qbase + i + e + ti.off - kpos));
              const float l = reinterpret_cast<const float*>(lse4)[i + e];
              float pv = ex2(x + l);
              if (need_mask && (i + e < c_lo || i + e >= c_hi)) pv = 0.f;
              pp[e] = pv;
              dd[e] = pv * deriv;
            }
            sr[i / 2] = pack2<BF16>(pp[0], pp[1]);
            pr[i] = dd[0];
            pr[i + 1] = dd[1];
          }
        }
        tmem_st32(t_s, sr);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(p_full);

        // ---- phase B: dS^T = P^T (dP^T - delta)
        if (!warp_wait(dp_full, par, ctl, kWaitBwd + 12)) { ok = false; break; }
        tc_fence_after();
        tmem_ld32(t_dp, sr);
        tmem_ld32(t_dp + 32, sr + 32);
        tmem_wait_ld();
        tc_fence_before();
        uint8_t* ds_row = s_ds + wg * (kBlk * 128) + key_in * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 d0 = dl4[2 * c], d1 = dl4[2 * c + 1];
          const int i = c * 8;
          const float d[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
          uint32_t ds[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int e = i + 2 * q;
            const uint64_t dp = add2(pack_f32x2(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), pack_f32x2(d[2 * q], d[2 * q + 1]));
            float a, b;
            unpack_f32x2(mul2(pack_f32x2(pr[e], pr[e + 1]), dp), a, b);
            ds[q] = pack2<BF16>(a, b);
          }
          const uint4 w = make_uint4(ds[0], ds[1], ds[2], ds[3]);
          *reinterpret_cast<uint4*>(ds_row + ((c ^ (key_in & 7)) << 4)) = w;
        }
        fence_proxy_async_smem();
        mbar_arrive(ds_full);
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_empty[par]);
      }
      // ---- epilogue: warpgroup 0 writes dK (scaled), warpgroup 1 writes dV
      if (ok) {
        const uint32_t t_acc = tmem + lane_addr + (wg == 0 ? Cfg::kTmemDK : Cfg::kTmemDV);
        const float mul = (wg == 0) ? p.scale : 1.f;
        uint16_t* gptr = reinterpret_cast<uint16_t*>(wg == 0 ? p.dk_ptr : p.dv_ptr);
        const bool store = (p.which & 2) != 0;
        if (n_iter > 0) ok = warp_wait(wg == 0 ? dkv_done : dv_done, pos.kv & 1, ctl, kWaitBwd + 13);
        if (ok && store) {
          tc_fence_after();
          uint16_t* grow = gptr + ti.bq * p.dkv_batch_stride + static_cast<int64_t>(ti.k_row0 + kpos) * p.dkv_row_stride +
                           ti.hk * p.dkv_head_stride;
          uint32_t acc[D];
          if (n_iter > 0) {
#pragma unroll
            for (int c = 0; c < D / 32; ++c) tmem_ld32(t_acc + c * 32, acc + c * 32);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < D; ++i) acc[i] = 0;
          }
          if (!PACKED && ti.parts > 1) {
            // A part of a split key block: fp32, 32 bytes (a whole sector) per store.
            if (kpos < ti.sk) {
              float* row = (wg == 0 ? p.dk_part : p.dv_part) + ti.part * p.part_stride + ti.bq * p.dkv_batch_stride +
                           static_cast<int64_t>(kpos) * p.dkv_row_stride + ti.hk * p.dkv_head_stride;
#pragma unroll
              for (int c = 0; c < D / 8; ++c)
                if (c * 8 < p.head_dim)
                  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row + 8 * c), "r"(acc[8 * c]),
                               "r"(acc[8 * c + 1]), "r"(acc[8 * c + 2]), "r"(acc[8 * c + 3]), "r"(acc[8 * c + 4]),
                               "r"(acc[8 * c + 5]), "r"(acc[8 * c + 6]), "r"(acc[8 * c + 7])
                               : "memory");
            }
          } else if (TAKE_OVER) {
            // Straight to memory, 32 bytes (a whole sector) per store where the rows allow.
            const bool sectors = (reinterpret_cast<uintptr_t>(gptr) & 31) == 0 && (p.head_dim & 15) == 0;
            if (kpos < ti.sk) {
#pragma unroll
              for (int c = 0; c < D / 16; ++c) {
                if (c * 16 >= p.head_dim) break;
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  w[i] = pack2<BF16>(__uint_as_float(acc[16 * c + 2 * i]) * mul, __uint_as_float(acc[16 * c + 2 * i + 1]) * mul);
                if (sectors) {
                  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(grow + 16 * c), "r"(w[0]), "r"(w[1]),
                               "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                               : "memory");
                } else {
                  *reinterpret_cast<uint4*>(grow + 16 * c) = make_uint4(w[0], w[1], w[2], w[3]);
                  if (c * 16 + 8 < p.head_dim) *reinterpret_cast<uint4*>(grow + 16 * c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
                }
              }
            }
          } else {
            // Staging tile of the bulk store: the K tile for dK, the V tile for dV (their last readers have completed
            // with dkv_done).
            const bool tma_store = !PACKED || ti.n0 + kBlk <= ti.sk;
            const CUtensorMap* tm = (wg == 0) ? &p.tm_dk : &p.tm_dv;
            uint8_t* stage = (wg == 0) ? s_k : s_v;
#pragma unroll
            for (int c = 0; c < D / 8; ++c) {  // 16-byte chunks of the row
              uint4 w;
              w.x = pack2<BF16>(__uint_as_float(acc[8 * c]) * mul, __uint_as_float(acc[8 * c + 1]) * mul);
              w.y = pack2<BF16>(__uint_as_float(acc[8 * c + 2]) * mul, __uint_as_float(acc[8 * c + 3]) * mul);
              w.z = pack2<BF16>(__uint_as_float(acc[8 * c + 4]) * mul, __uint_as_float(acc[8 * c + 5]) * mul);
              w.w = pack2<BF16>(__uint_as_float(acc[8 * c + 6]) * mul, __uint_as_float(acc[8 * c + 7]) * mul);
              if (tma_store) {
                *reinterpret_cast<uint4*>(stage + (c / 8) * (kBlk * 128) + key_in * 128 + (((c & 7) ^ (key_in & 7)) << 4)) = w;
              } else if (kpos < ti.sk && c * 8 < p.head_dim) {
                *reinterpret_cast<uint4*>(grow + c * 8) = w;
              }
            }
            if (tma_store) {
              fence_proxy_async_smem();
              mbar_arrive(&epi_full[wg]);
              if (key_in == 0 && mbar_wait(&epi_full[wg], 0, ctl, kWaitBwd + 16)) {
#pragma unroll
                for (int a = 0; a < Cfg::kAtoms; ++a)
                  if (a * 64 < p.head_dim) tma_store_4d(tm, stage + a * (kBlk * 128), a * 64, ti.hk, ti.k_row0 + ti.n0, ti.bq);
                tma_commit_group();
                tma_wait_group_read<0>();  // the staging tile must outlive the copy's reads, not its writes
              }
            }
          }
          tc_fence_before();  // the next tile's dV and dK overwrite the accumulators behind its P^T
        }
      }
      __syncwarp();
    } while (TAKE_OVER && ok && next_tile_warp(ti, pos));
  } else {
    // ------------------------------------------------------------------ dQ drain
    // The whole 128 x D fp32 tile goes to registers at once so that the dP^T / dQ columns are free
    // for the next iteration right away; it then leaves through a staging area of the drain's own
    // as cp.reduce.async.bulk adds into the accumulator.
    reg_alloc<kDrainRegs>();
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_dq = tmem + lane_addr + Cfg::kTmemDP;
    if (want_dq) {
      bool ok = true;
      KvTile ti = first_tile;
      Pos pos;
      do {
        Walk w{ti.g0, ti.mi0};
        for (int it = 0; it < ti.n_iter && ok; ++it, w = walk_next(w, ti.n_m)) {
          const int hq = ti.hk * p.group + w.g;
          const int m0 = (ti.m_start + w.mi) * kBlk;
          ok = warp_wait(dq_full, (pos.it0 + it) & 1, ctl, kWaitBwd + 14);
          if (!ok) break;
          tc_fence_after();
          uint32_t acc[D];
#pragma unroll
          for (int c = 0; c < D / 32; ++c) tmem_ld32(t_dq + c * 32, acc + c * 32);
          tmem_wait_ld();
          tc_fence_before();
          mbar_arrive(dq_free);
          // Packed batches: the 32-row boxes of the reduce-adds below reach past the end of the sequence into
          // the next sequence's rows. Rows past the end hold nothing of this sequence (and possibly NaN, when this
          // sequence's own data is not finite): they add exact zeros.
          if (PACKED && m0 + (warp & 3) * 32 + lane >= ti.sq) {
#pragma unroll
            for (int i = 0; i < D; ++i) acc[i] = 0u;
          }
          // Each warp drains its own 32 rows in pieces of 32 fp32 columns (4 KB) that roll through two buffers of its
          // own, also from one tile to the next. Nothing but the warp itself has to be synchronised.
          constexpr int kWarpPiece = Cfg::kPieceBytes / 4;
          uint8_t* stage = smem + Cfg::kDQOff + (warp & 3) * (Cfg::kPieces * kWarpPiece);
          int* turn = nullptr;
          if (PACKED && p.dq_turn != nullptr) {
            // Ordered mode: the key blocks that add into these rows take their turns in descending order,
            // which is the order in which they get there under a causal or sliding-window mask (a higher key
            // block starts at a later query block). This block's turn is the number of higher key blocks
            // that cover the rows; a bounded wait for the slab's counter to reach it follows. In this mode the
            // grid lists a head's key blocks highest first (get_kv_tile), so the blocks waited for started earlier.
            const int mq = m0 / kBlk;
            int rank = 0;
            for (int nb = ti.n0 / kBlk + 1; nb < p.num_nblk; nb += 32) {
              const int n = nb + lane;
              bool covers = false;
              if (n < p.num_nblk && n * kBlk < ti.sk) {
                int ms, nm;
                q_block_range(p, ti.sq, ti.sk, n * kBlk, kBlk, ms, nm);
                covers = (mq >= ms) && (mq < ms + nm);
              }
              rank += __popc(__ballot_sync(0xffffffffu, covers));
            }
            turn = p.dq_turn + ((static_cast<int64_t>(ti.b) * p.heads + hq) * p.num_mblk_q + mq) * 4 + (warp & 3);
            if (lane == 0) {
              const long long t0 = clock64();
              while (*reinterpret_cast<volatile int*>(turn) != rank) {
                __nanosleep(200);
                if (*abort_flag || clock64() - t0 > FA2_WAIT_LIMIT_CYCLES) {
                  if (!*abort_flag) *abort_flag = kWaitBwd + 19;
                  ok = false;
                  break;
                }
              }
              __threadfence();
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
          }
#pragma unroll
          for (int k = 0; k < D / 32; ++k) {
            // The buffer is free once the reduce of the piece two before this one has read it.
            if (lane == 0) tma_wait_group_read<Cfg::kPieces - 1>();
            __syncwarp();
            uint8_t* buf = stage + (k % Cfg::kPieces) * kWarpPiece;
            uint8_t* rowp = buf + lane * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<uint4*>(rowp + ((c ^ (lane & 7)) << 4)) =
                  make_uint4(acc[k * 32 + 4 * c], acc[k * 32 + 4 * c + 1], acc[k * 32 + 4 * c + 2], acc[k * 32 + 4 * c + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (k * 32 < p.head_dim) tma_reduce_add_4d(&p.tm_dqa, buf, k * 32, hq, ti.q_row0 + m0 + (warp & 3) * 32, ti.bq);
              tma_commit_group();
            }
          }
          if (!ok) break;
          if (turn != nullptr && lane == 0) {
            // The adds have to be in memory before the next key block may start on these rows.
            tma_wait_group<0>();
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __threadfence();
            atomicAdd(turn, 1);
          }
        }
      } while (TAKE_OVER && ok && next_tile_warp(ti, pos));
      if (lane == 0) tma_wait_group_read<0>();
    }
  }
  __syncwarp();
  if (*abort_flag) {
    // A wait ran out somewhere in this CTA. MMAs, commits and copies may still be in flight: give them
    // about a millisecond to land before the barriers' memory and the TMEM columns are given back.
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {  // its index lives to the end anyway; the thread's (tid == 0) was spilled for it
    if (elect_one()) report_abort(abort_flag, p.status);
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

template <int D, bool BF16, int MODE, bool PACKED, bool TAKE_OVER>
cudaError_t launch_tiles(const BwdParams& p, int num_ctas, cudaStream_t stream) {
  using Cfg = BwdCfg<D>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(bwd_kernel<D, BF16, MODE, PACKED, TAKE_OVER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_grid(!PACKED, bwd_kernel<D, BF16, MODE, PACKED, TAKE_OVER>, dim3(num_ctas), kThreads, Cfg::kSmemBytes, stream, p);
}

template <int D, bool BF16, int MODE, bool PACKED>
cudaError_t launch_one(const BwdParams& p, int num_ctas, int num_sms, cudaStream_t stream) {
  // A CTA asks for its next tile before it has finished this one; in a call of a wave or two that takes tiles away from SMs
  // that are about to be free (B1 H8/2 S1500 D64, bit-reproducible: 57.7 -> 59.5 us). Below the line the code alone costs 1-4 us;
  // forward and backward (graph replay) with it and without: 288 CTAs, B2 H16 S1100 causal, 55.8, 52.0 us, 144 CTAs, B1 H12 S1500,
  // 61.1, 59.6. Above it: 416 CTAs, B26 H8 S256, 45.0, 46.7, 1536 CTAs, B32 H12 S509 fp16, 207, 222.
  if constexpr (D == 64 && !PACKED) {
    if (num_ctas > 2 * num_sms) return launch_tiles<D, BF16, MODE, PACKED, true>(p, num_ctas, stream);
  }
  return launch_tiles<D, BF16, MODE, PACKED, false>(p, num_ctas, stream);
}

template <int D, bool BF16>
cudaError_t pick_features(const BwdParams& p, int mode, bool packed, int num_ctas, int num_sms, cudaStream_t stream) {
  if (packed) {
    return mode != kScorePlain ? launch_one<D, BF16, kScoreAny, true>(p, num_ctas, num_sms, stream)
                               : launch_one<D, BF16, kScorePlain, true>(p, num_ctas, num_sms, stream);
  }
  switch (mode) {
    case kScorePlain: return launch_one<D, BF16, kScorePlain, false>(p, num_ctas, num_sms, stream);
    case kScoreSoftcap: return launch_one<D, BF16, kScoreSoftcap, false>(p, num_ctas, num_sms, stream);
    case kScoreAlibi: return launch_one<D, BF16, kScoreAlibi, false>(p, num_ctas, num_sms, stream);
    default: return launch_one<D, BF16, kScoreAny, false>(p, num_ctas, num_sms, stream);
  }
}

template <int D>
cudaError_t pick_dtype(const BwdParams& p, bool bf16, int mode, bool packed, int num_ctas, int num_sms, cudaStream_t stream) {
  return bf16 ? pick_features<D, true>(p, mode, packed, num_ctas, num_sms, stream)
              : pick_features<D, false>(p, mode, packed, num_ctas, num_sms, stream);
}

}  // namespace

cudaError_t launch_bwd(const BwdParams& p, int head_dim, bool bf16, int num_sms, cudaStream_t stream) {
  const int num_ctas = (p.dk_part != nullptr ? p.items_per_head : p.num_nblk) * p.batch * p.heads_k;
  if (num_ctas <= 0) return cudaSuccess;
  if (head_dim <= 0 || head_dim > 128) return cudaErrorInvalidValue;
  const int mode = (p.softcap > 0.f ? kScoreSoftcap : 0) | (p.alibi != nullptr ? kScoreAlibi : 0);
  const bool packed = p.cu_q != nullptr;
  return head_dim > 64 ? pick_dtype<128>(p, bf16, mode, packed, num_ctas, num_sms, stream)
                       : pick_dtype<64>(p, bf16, mode, packed, num_ctas, num_sms, stream);
}

}  // namespace fa2
