// Forward for few query rows against many keys (decoding, speculative decoding) for sm_100a (B200).
//
// What bounds it: reading K and V once. With at most 64 query rows per kv head the products are a few percent of
// the chip's tensor rate, so the design is about keeping every SM's share of HBM busy:
//
//   * The query heads of a GQA group share their kv head's K and V: the group's rows (row r = query r / group,
//     head r % group) are the M dimension of one problem, and K and V cross the memory system once per kv head.
//   * The key tiles of all (batch, kv head) units form one list that is cut into equal contiguous shares, one per
//     CTA, one CTA per SM. A share may end in the middle of a unit; the CTA then leaves a partial result (fp32 O, row
//     maximum, row sum) in the workspace and the CTA that finishes a unit last adds the partials up. Which CTA that is
//     is seen from a flag per part that holds the launch's number, so the workspace needs no clearing.
//   * One warp keeps a ring of 196 KB of K and V tiles filled by TMA (23 B/clk per SM is an SM's share of HBM; a
//     round trip of about 2000 cycles needs 46 KB in flight), eight warps consume it. Each consumer owns 16 x MT keys
//     of a 128-key tile and 16 query rows and never waits for another consumer until the share's unit ends.
//   * The products are m16n8k16 mma.sync: 16 rows are exactly one M tile, the scores come back in registers in the
//     layout that the second product takes, and a tile needs about 600 of the 2800 cycles its bytes take to arrive.
//     tcgen05 has M = 128 at least: it would need the transposed problem with the row maxima across TMEM lanes.
//
// Stands in for the reference's split-KV forward and its combine kernel
// (flash-attn2-rs/src/host/forward/dispatch.rs:63-437, src/device/forward/mod.rs:1162-1407).
#include "sm100_ptx.cuh"
#include "fa2_params.h"
#include "fa2_launch.h"

namespace fa2 {

namespace {

constexpr int kTile = 128;           // keys per tile
constexpr int kConsumers = 8;        // warps
constexpr int kThreads = 384;         // two warpgroups of consumers, one that holds the loader warp
constexpr int kConsumerRegs = 232;    // the output accumulators alone take D / 2 registers
constexpr int kLoaderRegs = 40;
// setmaxnreg moves registers inside the CTA's own allocation (168 per thread at launch: 65536 / 384 rounded down).
static_assert(8 * (kConsumerRegs - 168) <= 4 * (168 - kLoaderRegs), "setmaxnreg: the consumers ask for more than the loader's group releases");
constexpr int kMaxSlots = 12;

template <int A, int MT>  // A: 64-column atoms of the head dim; MT: 16-row tiles
struct DecCfg {
  static constexpr int D = A * 64;
  static constexpr int kSlotBytes = kTile * D * 2;
  static constexpr int kSlots = kMaxSlots / A;
  static constexpr int kRows = 16 * MT;
  static constexpr int kQOff = kSlots * kSlotBytes;
  static constexpr int kQBytes = kRows * D * 2;
  static constexpr int kStatOff = kQOff + kQBytes;                 // m, l of every consumer warp: [8][16][2] fp32
  static constexpr int kBarOff = kStatOff + kConsumers * 16 * 2 * 4;
  static constexpr int kMiscOff = kBarOff + 2 * kMaxSlots * 8;
  static constexpr int kSmemBytes = kMiscOff + 16;
  // Does the merge load twelve parts at a time, the first ones before the rows' maxima, or eight behind them? Eight, then twelve,
  // us a call: B1 H32/8 Sk 8192 D64 11.7, 11.1 and D128 13.1, 12.7; B1 H64/8 Sq 3 Sk 8192 D64 15.9, 15.5, D128 22.0, 20.9 and
  // D192 30.0, 29.1. Elsewhere the registers that it takes cost the loop over the key tiles more: spills at D192 with up to 16
  // rows and with more than 32; B4 H16/2 Sk 5000 D256 19.5, 20.5; B4 H64/8 Sq 8 Sk 2000 D256 45.0, 48.7.
  static constexpr bool kMergeAhead = A < 4 && MT < 4 && !(A == 3 && MT == 1);
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if constexpr (BF16) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers * 32) : "memory"); }

// exp2(m - m_tot) with m = -inf (a part that saw no key) giving 0 also when m_tot = -inf.
__device__ __forceinline__ float part_scale(float m, float m_tot) { return m == -INFINITY ? 0.f : ex2(m - m_tot); }

// PARTS: units may be shared by CTAs. Calls without parts have instances of their own: the merge, although they never reach it,
// changes how the compiler lays out the loop over the key tiles: B10 H32/8 Sk 4000 D128 34.8 us a call with it, 30.8 without,
// D64 25.3 and 22.6. With more than 32 rows the loop is the better one with it (B16 H64/8 Sq 8 Sk 4096 D128 72.0, without 73.8),
// so there one instance takes both.
template <int A, int MT, bool BF16, bool PARTS>
__global__ void __launch_bounds__(kThreads, 1) fwd_decode_kernel(const __grid_constant__ DecodeParams p) {
  using Cfg = DecCfg<A, MT>;
  constexpr int D = Cfg::D;
  constexpr int kGroups = kConsumers / MT;      // key groups
  constexpr int kKeys = kTile / kGroups;        // keys of a tile per warp
  constexpr int kNT = kKeys / 8;                // score n-tiles per warp
  constexpr int kOT = D / 8;                    // output n-tiles
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kBarOff);
  uint64_t* empty = full + kMaxSlots;
  float* s_stat = reinterpret_cast<float*>(smem + Cfg::kStatOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff);
  volatile int* s_last = reinterpret_cast<volatile int*>(smem + Cfg::kMiscOff + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const WaitCtl ctl{abort_flag};
  // this CTA's share of the tile list; without parts (no workspace for them) it is whole units
  const int64_t n_tiles = static_cast<int64_t>(p.units) * p.tiles_per_unit;
  int lo, hi;
  if (PARTS && p.partials != nullptr) {
    lo = static_cast<int>(blockIdx.x * n_tiles / gridDim.x);
    hi = static_cast<int>((blockIdx.x + 1) * n_tiles / gridDim.x);
  } else {
    lo = static_cast<int>(static_cast<int64_t>(blockIdx.x) * p.units / gridDim.x) * p.tiles_per_unit;
    hi = static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * p.units / gridDim.x) * p.tiles_per_unit;
  }

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < Cfg::kSlots; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], kConsumers);
    }
    mbar_fence_init();
  }
  if (warp == kConsumers && lane == 0) {
    tma_prefetch_desc(&p.tm_k);
    tma_prefetch_desc(&p.tm_v);
  }
  early_wait();
  __syncthreads();
  early_trigger();

  if (warp >= kConsumers) {
    // ---------------------------------------------------------------- loader
    reg_dealloc<kLoaderRegs>();
    if (warp == kConsumers && elect_one()) {
      uint32_t slot = 0, phase = 0;
      bool ok = true;
      int u = lo / p.tiles_per_unit, j = lo - u * p.tiles_per_unit;
      for (int x = lo; x < hi && ok; ++x) {
        const int b = u / p.heads_k, hk = u - b * p.heads_k;
        const int row = (p.tile_lo + j) * kTile;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          ok = ok && mbar_wait(&empty[slot], phase ^ 1, ctl, kWaitDecode + 1);
          if (!ok) break;
          mbar_expect_tx(&full[slot], Cfg::kSlotBytes);
#pragma unroll
          for (int a = 0; a < A; ++a)
            tma_load_4d(smem + slot * Cfg::kSlotBytes + a * (kTile * 128), which ? &p.tm_v : &p.tm_k, &full[slot], a * 64, hk, row, b);
          if (++slot == Cfg::kSlots) {
            slot = 0;
            phase ^= 1;
          }
        }
        if (++j == p.tiles_per_unit) {
          j = 0;
          ++u;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- consumers
    reg_alloc<kConsumerRegs>();
    const int mt = warp % MT, kg = warp / MT;
    const int g = lane >> 2, t4 = lane & 3;      // fragment coordinates: rows g and g + 8, columns 2 t4 and 2 t4 + 1
    const int lm = lane >> 3, lr = lane & 7;     // ldmatrix: matrix and row this lane addresses
    const uint32_t s_base = smem_u32(smem);
    // Byte offsets of this lane's ldmatrix row inside a tile. The row's index within 8 is lr everywhere, so the
    // swizzle is one XOR with lr of the 16-byte chunk index.
    const uint32_t k_row = (kg * kKeys + (lm >> 1) * 8 + lr) * 128;  // K: matrices (keys 0-7, chunk 0), (0-7, 1), (8-15, 0), (8-15, 1)
    const uint32_t v_row = (kg * kKeys + (lm & 1) * 8 + lr) * 128;   // V, transposed: (keys 0-7, chunk 0), (8-15, 0), (0-7, 1), (8-15, 1)
    const uint32_t q_addr = s_base + Cfg::kQOff + (mt * 16 + (lm & 1) * 8 + lr) * 128;
    auto q_frag = [&](int ks, uint32_t* r) {
      ldsm4(q_addr + (ks / 4) * (Cfg::kRows * 128) + ((((ks % 4) * 2 + (lm >> 1)) ^ lr) << 4), r);
    };
    // The rows of this thread: query index and head within the group.
    const int r0 = mt * 16 + g, r1 = r0 + 8;
    const int q0 = r0 / p.group, q1 = r1 / p.group;
    const bool has_alibi = p.alibi != nullptr;
    const float inv_cap = p.softcap > 0.f ? p.scale / p.softcap : 0.f;
    const float cap_l2 = p.softcap * 1.4426950408889634f;
    uint32_t slot = 0, phase = 0;
    auto next_slot = [&]() {
      if (++slot == Cfg::kSlots) {
        slot = 0;
        phase ^= 1;
      }
    };
    int u = lo / p.tiles_per_unit, j = lo - u * p.tiles_per_unit;
    // A segment: the share's part of one unit, tiles [seg_first, seg_end) of it.
    for (int x = lo; x < hi;) {
      const int b = u / p.heads_k, hk = u - b * p.heads_k;
      const int seg_first = j, seg_end = min(p.tiles_per_unit, j + hi - x);
      x += seg_end - seg_first;
      // Q rows of the unit -> swizzled shared memory; rows past the last one are zero.
      consumers_sync();  // the previous unit's Q has been read
      for (int c = tid; c < Cfg::kRows * A * 8; c += kConsumers * 32) {
        const int r = c / (A * 8), ch = c - r * (A * 8);
        uint4 w = make_uint4(0, 0, 0, 0);
        if (r < p.rows && ch * 8 < p.head_dim) {
          const int q = r / p.group, h = hk * p.group + (r - q * p.group);
          w = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.q_ptr) + b * p.q_batch_stride +
                                              q * p.q_row_stride + h * p.q_head_stride + ch * 8);
        }
        *reinterpret_cast<uint4*>(smem + Cfg::kQOff + (ch / 8) * (Cfg::kRows * 128) + r * 128 + (((ch & 7) ^ (r & 7)) << 4)) = w;
      }
      consumers_sync();
      uint32_t qf[A <= 2 ? D / 16 : 1][4];  // Q fragments stay in registers up to head dim 128
      if constexpr (A <= 2) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) q_frag(ks, qf[ks]);
      }
      float slope0 = 0.f, slope1 = 0.f;
      if (has_alibi) {
        const float* al = p.alibi + b * p.alibi_batch_stride + hk * p.group;
        slope0 = r0 < p.rows ? al[r0 - q0 * p.group] * 1.4426950408889634f : 0.f;
        slope1 = r1 < p.rows ? al[r1 - q1 * p.group] * 1.4426950408889634f : 0.f;
      }
      float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
      float o[kOT][4];
#pragma unroll
      for (int i = 0; i < kOT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
      for (; j < seg_end; ++j) {
        // ---- scores of this warp's keys
        float s[kNT][4];
#pragma unroll
        for (int i = 0; i < kNT; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
        mbar_wait(&full[slot], phase, ctl, kWaitDecode + 2);
        __syncwarp();
        {
          const uint32_t kb = s_base + slot * Cfg::kSlotBytes + k_row;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t qa[4];
            if constexpr (A <= 2) {
#pragma unroll
              for (int e = 0; e < 4; ++e) qa[e] = qf[ks][e];
            } else {
              q_frag(ks, qa);
            }
#pragma unroll
            for (int i = 0; i < kNT; i += 2) {
              uint32_t kf[4];
              ldsm4(kb + (ks / 4) * (kTile * 128) + i * (8 * 128) + ((((ks % 4) * 2 + (lm & 1)) ^ lr) << 4), kf);
              mma16816<BF16>(s[i], qa, kf[0], kf[1]);
              mma16816<BF16>(s[i + 1], qa, kf[2], kf[3]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        next_slot();
        // ---- transform and mask: scores into the log2 domain
        const int col0 = (p.tile_lo + j) * kTile + kg * kKeys + 2 * t4;
        if (p.softcap > 0.f) {
#pragma unroll
          for (int i = 0; i < kNT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] = cap_l2 * tanh_approx(s[i][e] * inv_cap);
        } else {
#pragma unroll
          for (int i = 0; i < kNT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] *= p.scale_log2;
        }
        if (has_alibi) {
#pragma unroll
          for (int i = 0; i < kNT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int col = col0 + i * 8 + (e & 1);
              const float sl = (e & 2) ? slope1 : slope0;
              s[i][e] += p.causal_alibi ? sl * static_cast<float>(col)
                                        : -sl * fabsf(static_cast<float>(((e & 2) ? q1 : q0) + p.off - col));
            }
        }
        const int tile_col = (p.tile_lo + j) * kTile;
        // Only the tiles at the ends of the rows' key ranges have anything to mask.
        if (tile_col + kTile > p.full_hi || tile_col < p.full_lo) {
          int hi0 = p.seqlen_k, hi1 = p.seqlen_k, lo0 = 0, lo1 = 0;
          if (p.window_right >= 0) {
            hi0 = min(hi0, q0 + p.off + p.window_right + 1);
            hi1 = min(hi1, q1 + p.off + p.window_right + 1);
          }
          if (p.window_left >= 0) {
            lo0 = q0 + p.off - p.window_left;
            lo1 = q1 + p.off - p.window_left;
          }
#pragma unroll
          for (int i = 0; i < kNT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int col = col0 + i * 8 + (e & 1);
              if (col >= ((e & 2) ? hi1 : hi0) || col < ((e & 2) ? lo1 : lo0)) s[i][e] = -INFINITY;
            }
        }
        // ---- row maxima over the four lanes of a row, rescale
        float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < kNT; ++i) {
          x0 = max3(x0, s[i][0], s[i][1]);
          x1 = max3(x1, s[i][2], s[i][3]);
        }
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {
          x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, d));
          x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, d));
        }
        const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
        if (__any_sync(0xffffffffu, n0 > m0 || n1 > m1)) {
          const float a0 = part_scale(m0, n0), a1 = part_scale(m1, n1);
          l0 *= a0;
          l1 *= a1;
#pragma unroll
          for (int i = 0; i < kOT; ++i) {
            o[i][0] *= a0;
            o[i][1] *= a0;
            o[i][2] *= a1;
            o[i][3] *= a1;
          }
          m0 = n0;
          m1 = n1;
        }
        const float b0 = m0 == -INFINITY ? 0.f : m0, b1 = m1 == -INFINITY ? 0.f : m1;
        uint32_t pf[kNT][2];
#pragma unroll
        for (int i = 0; i < kNT; ++i) {
          const float e0 = ex2(s[i][0] - b0), e1 = ex2(s[i][1] - b0), e2 = ex2(s[i][2] - b1), e3 = ex2(s[i][3] - b1);
          l0 += e0 + e1;
          l1 += e2 + e3;
          pf[i][0] = pack2<BF16>(e0, e1);
          pf[i][1] = pack2<BF16>(e2, e3);
        }
        // ---- O += P V
        mbar_wait(&full[slot], phase, ctl, kWaitDecode + 3);
        __syncwarp();
        {
          const uint32_t vb = s_base + slot * Cfg::kSlotBytes + v_row;
#pragma unroll
          for (int kk = 0; kk < kNT / 2; ++kk) {
            const uint32_t pa[4] = {pf[2 * kk][0], pf[2 * kk][1], pf[2 * kk + 1][0], pf[2 * kk + 1][1]};
#pragma unroll
            for (int i = 0; i < kOT; i += 2) {
              uint32_t vf[4];
              ldsm4_trans(vb + (i / 8) * (kTile * 128) + kk * (16 * 128) + ((((i % 8) + (lm >> 1)) ^ lr) << 4), vf);
              mma16816<BF16>(o[i], pa, vf[0], vf[1]);
              mma16816<BF16>(o[i + 1], pa, vf[2], vf[3]);
            }
          }
        }
        __syncwarp();
        if (j + 1 < seg_end) {  // the last V slot stays held
          if (lane == 0) mbar_arrive(&empty[slot]);
          next_slot();
        }
      }
      // ---- the consumers' parts of this segment become one: the last V slot, still held, is the scratch space.
      l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
      l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
      l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
      l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
      if (t4 == 0) {
        float* st = s_stat + warp * 32;
        st[g] = m0;
        st[8 + g] = m1;
        st[16 + g] = l0;
        st[24 + g] = l1;
      }
      consumers_sync();
      float t0 = -INFINITY, t1 = -INFINITY;
#pragma unroll
      for (int w = 0; w < kGroups; ++w) {
        t0 = fmaxf(t0, s_stat[(w * MT + mt) * 32 + g]);
        t1 = fmaxf(t1, s_stat[(w * MT + mt) * 32 + 8 + g]);
      }
      float ls0 = 0.f, ls1 = 0.f;
#pragma unroll
      for (int w = 0; w < kGroups; ++w) {
        const float* st = s_stat + (w * MT + mt) * 32;
        ls0 += st[16 + g] * part_scale(st[g], t0);
        ls1 += st[24 + g] * part_scale(st[8 + g], t1);
      }
      {
        const float a0 = part_scale(m0, t0), a1 = part_scale(m1, t1);
#pragma unroll
        for (int i = 0; i < kOT; ++i) {
          o[i][0] *= a0;
          o[i][1] *= a0;
          o[i][2] *= a1;
          o[i][3] *= a1;
        }
      }
      // Half of the key groups leave their fragments, the other half adds its own on top, then every warp sums its
      // share of the columns over what is left: two barriers, and the rest of the segment's end is spread over
      // all warps. 4 x 16 rows x D fp32 = one slot.
      float4* scratch = reinterpret_cast<float4*>(smem + slot * Cfg::kSlotBytes);
      constexpr int kHalf = kGroups / 2;
      float4* mine = scratch + ((kg % kHalf) * MT + mt) * (kOT * 32) + lane;
      if (kg >= kHalf) {
#pragma unroll
        for (int i = 0; i < kOT; ++i) mine[i * 32] = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
      }
      consumers_sync();
      if (kg < kHalf) {
#pragma unroll
        for (int i = 0; i < kOT; ++i) {
          const float4 w = mine[i * 32];
          mine[i * 32] = make_float4(o[i][0] + w.x, o[i][1] + w.y, o[i][2] + w.z, o[i][3] + w.w);
        }
      }
      consumers_sync();
      constexpr int kMine = kOT / kGroups;  // column tiles of this warp: kg * kMine + i
      float4 part_o[kMine];
#pragma unroll
      for (int i = 0; i < kMine; ++i) {
        const float4* src = scratch + mt * (kOT * 32) + (kg * kMine + i) * 32 + lane;
        part_o[i] = src[0];
#pragma unroll
        for (int w = 1; w < kHalf; ++w) {
          const float4 t = src[w * MT * (kOT * 32)];
          part_o[i].x += t.x;
          part_o[i].y += t.y;
          part_o[i].z += t.z;
          part_o[i].w += t.w;
        }
      }
      // ---- out, or a partial result
      auto store_pair = [&](int r, int i, float a, float c) {
        if (r < p.rows && i * 8 < p.head_dim) {
          const int q = r / p.group, h = hk * p.group + (r - q * p.group);
          *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.o_ptr) + b * p.o_batch_stride + q * p.o_row_stride +
                                       h * p.o_head_stride + i * 8 + 2 * t4) = pack2<BF16>(a, c);
        }
      };
      auto store_lse = [&](int r, float m, float l) {
        if (r < p.rows) {
          const int q = r / p.group, h = hk * p.group + (r - q * p.group);
          p.lse_ptr[b * p.lse_batch_stride + h * p.lse_head_stride + q] = l > 0.f ? (m + lg2(l)) * 0.6931471805599453f : INFINITY;
        }
      };
      const bool whole = !PARTS || (seg_first == 0 && seg_end == p.tiles_per_unit);
      if (whole) {
        const float i0 = ls0 > 0.f ? 1.f / ls0 : 0.f, i1 = ls1 > 0.f ? 1.f / ls1 : 0.f;
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
          store_pair(r0, kg * kMine + i, part_o[i].x * i0, part_o[i].y * i0);
          store_pair(r1, kg * kMine + i, part_o[i].z * i1, part_o[i].w * i1);
        }
        if (kg == 0 && t4 == 0) {
          store_lse(r0, t0, ls0);
          store_lse(r1, t1, ls1);
        }
      } else if constexpr (PARTS) {
        // Slot 2c holds a segment that began before this share, 2c + 1 one that began in it. Layout of a slot: O
        // [row][column], then m and l of the rows; rows past the last one are neither written nor read.
        constexpr int kPart = Cfg::kRows * (D + 2);  // floats
        float* part = p.partials + (2 * static_cast<int64_t>(blockIdx.x) + (seg_first == 0 ? 1 : 0)) * kPart;
        float2* dst = reinterpret_cast<float2*>(part + r0 * D + 2 * t4);
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
          if (r0 < p.rows) __stcg(dst + (kg * kMine + i) * 4, make_float2(part_o[i].x, part_o[i].y));
          if (r1 < p.rows) __stcg(dst + 4 * D + (kg * kMine + i) * 4, make_float2(part_o[i].z, part_o[i].w));
        }
        if (kg == 0 && t4 == 0) {
          float* st = part + Cfg::kRows * D;
          __stcg(st + r0, t0);
          __stcg(st + r1, t1);
          __stcg(st + Cfg::kRows + r0, ls0);
          __stcg(st + Cfg::kRows + r1, ls1);
        }
        // CTAs whose shares touch this unit: the owners of its first and its last tile.
        const int64_t g64 = gridDim.x;
        const int64_t first_tile = static_cast<int64_t>(u) * p.tiles_per_unit;
        const int c_first = static_cast<int>(((first_tile + 1) * g64 + n_tiles - 1) / n_tiles - 1);
        const int c_last = static_cast<int>(((first_tile + p.tiles_per_unit) * g64 + n_tiles - 1) / n_tiles - 1);
        auto part_index = [&](int c) { return 2 * c + (c == c_first ? 1 : 0); };
        consumers_sync();
        if (warp == 0) {
          // One flag per part, set to the launch's number once the part is in memory: a flag left over from another
          // launch, or from other use of the memory, is not set. Whoever sees all of a unit's flags set merges. The
          // last to set one does (store, fence, load); two may, and then both write the same bits. A counter
          // in place of the flags would need clearing, or a compare-and-swap that 19 CTAs queue up for (0.5 us each).
          volatile unsigned long long* flags = p.flags;
          // All warps' stores come before the barrier; this thread's fence behind it makes them the flag's predecessors.
          if (lane == 0) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            flags[part_index(blockIdx.x)] = p.launch_tag;
          }
          __syncwarp();
          asm volatile("fence.sc.gpu;" ::: "memory");
          bool all = true;
          for (int c = c_first + lane; c <= c_last; c += 32) all = all && flags[part_index(c)] == p.launch_tag;
          all = __all_sync(0xffffffffu, all);
          asm volatile("fence.acq_rel.gpu;" ::: "memory");
          if (all) {
            // A replayed graph launches with the same number: it has to find the flags clear.
            for (int c = c_first + lane; c <= c_last; c += 32) flags[part_index(c)] = 0;
          }
          if (lane == 0) *s_last = all ? 1 : 0;
        }
        consumers_sync();
        if (*s_last) {
          // All consumers add the parts up: the rows' maxima and sums go to shared memory, and a thread takes four columns of
          // a row at a time, with the loads of a batch of parts issued together: each batch is an L2 round trip.
          // Part c of the unit: every second slot, but the first one, which began in its share, has the slot behind.
          const float* part0 = p.partials + 2 * static_cast<int64_t>(c_first) * kPart;
          auto part_of = [&](int c) { return part0 + c * (2 * kPart) + (c == 0 ? kPart : 0); };
          const int n_parts = c_last - c_first + 1;
          float* sm = reinterpret_cast<float*>(scratch);
          float* sl = sm + n_parts * Cfg::kRows;
          constexpr int kBatch = Cfg::kMergeAhead ? 12 : 8;
          float4 w[kBatch];
          auto fetch = [&](int i, int c0) {
#pragma unroll
            for (int e = 0; e < kBatch; ++e)
              if (c0 + e < n_parts) w[e] = __ldcg(reinterpret_cast<const float4*>(part_of(c0 + e)) + i);
          };
          if (Cfg::kMergeAhead && tid < p.rows * (D / 4)) fetch(tid, 0);
          for (int i = tid; i < n_parts * Cfg::kRows; i += kConsumers * 32) {
            const int r = i % Cfg::kRows;
            if (r < p.rows) {
              const float* st = part_of(i / Cfg::kRows) + Cfg::kRows * D + r;
              sm[i] = __ldcg(st);
              sl[i] = __ldcg(st + Cfg::kRows);
            }
          }
          consumers_sync();
          for (int i = tid; i < p.rows * (D / 4); i += kConsumers * 32) {
            const int r = i / (D / 4), col = i % (D / 4) * 4;
            float m = -INFINITY, l = 0.f;
            for (int c = 0; c < n_parts; ++c) m = fmaxf(m, sm[c * Cfg::kRows + r]);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c = 0; c < n_parts; c += kBatch) {
              if (!Cfg::kMergeAhead || i != tid || c > 0) fetch(i, c);
#pragma unroll
              for (int e = 0; e < kBatch; ++e)
                if (c + e < n_parts) {
                  const float f = part_scale(sm[(c + e) * Cfg::kRows + r], m);
                  l += f * sl[(c + e) * Cfg::kRows + r];
                  acc.x += f * w[e].x;
                  acc.y += f * w[e].y;
                  acc.z += f * w[e].z;
                  acc.w += f * w[e].w;
                }
            }
            if (col < p.head_dim) {
              const float inv = l > 0.f ? 1.f / l : 0.f;
              const int q = r / p.group, h = hk * p.group + (r - q * p.group);
              *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.o_ptr) + b * p.o_batch_stride + q * p.o_row_stride +
                                        h * p.o_head_stride + col) =
                  make_uint2(pack2<BF16>(acc.x * inv, acc.y * inv), pack2<BF16>(acc.z * inv, acc.w * inv));
              if (col == 0) store_lse(r, m, l);
            }
          }
        }
      }
      // The V slot goes back to the loader; as the scratch space it was written by the generic proxy.
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[slot]);
      next_slot();
      if (j == p.tiles_per_unit) {
        j = 0;
        ++u;
      }
    }
  }
  __syncwarp();
  if (*abort_flag) {
    // A wait ran out: copies may still be in flight, give them about a millisecond before the memory is given back.
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
  }
  __syncthreads();
  if (tid == 0) report_abort(abort_flag, p.status);
}

template <int A, int MT, bool BF16, bool PARTS>
cudaError_t launch_one(const DecodeParams& p, int grid, bool early, cudaStream_t stream) {
  using Cfg = DecCfg<A, MT>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(fwd_decode_kernel<A, MT, BF16, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return launch_grid(early, fwd_decode_kernel<A, MT, BF16, PARTS>, dim3(grid), kThreads, Cfg::kSmemBytes, stream, p);
}

template <int A, int MT, bool BF16>
cudaError_t pick_parts(const DecodeParams& p, int grid, bool early, cudaStream_t stream) {
  if constexpr (MT < 4) {
    if (p.partials == nullptr) return launch_one<A, MT, BF16, false>(p, grid, early, stream);
  }
  return launch_one<A, MT, BF16, true>(p, grid, early, stream);
}

template <int A, bool BF16>
cudaError_t pick_rows(const DecodeParams& p, int grid, bool early, cudaStream_t stream) {
  if (p.rows <= 16) return pick_parts<A, 1, BF16>(p, grid, early, stream);
  if (p.rows <= 32) return pick_parts<A, 2, BF16>(p, grid, early, stream);
  return pick_parts<A, 4, BF16>(p, grid, early, stream);
}

template <bool BF16>
cudaError_t pick_dim(const DecodeParams& p, int grid, bool early, cudaStream_t stream) {
  if (p.head_dim <= 64) return pick_rows<1, BF16>(p, grid, early, stream);
  if (p.head_dim <= 128) return pick_rows<2, BF16>(p, grid, early, stream);
  if (p.head_dim <= 192) return pick_rows<3, BF16>(p, grid, early, stream);
  return pick_rows<4, BF16>(p, grid, early, stream);
}

}  // namespace

cudaError_t launch_fwd_decode(const DecodeParams& p, int grid, bool bf16, bool early, cudaStream_t stream) {
  if (p.rows <= 0 || p.rows > kDecodeMaxRows || p.head_dim <= 0 || p.head_dim > 256 || grid <= 0) return cudaErrorInvalidValue;
  return bf16 ? pick_dim<true>(p, grid, early, stream) : pick_dim<false>(p, grid, early, stream);
}

}  // namespace fa2
