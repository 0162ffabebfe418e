// How a dense call is divided over the GPU: pure functions of the arguments and the number of SMs.
#pragma once
#include "../../include/fa2_b200.h"
#include "fa2_params.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>

namespace fa2 {

struct Windows {
  int left, right, causal_alibi;
};
// Window normalisation of the reference (forward/mod.rs:310-328, backward.rs:134-149): clamp
// sides that cover every key to "open", causal means right = 0.
inline Windows normalise_windows(int64_t wl, int64_t wr, bool causal, int64_t seqlen_k, bool causal_first) {
  if (causal_first && causal) wr = 0;
  if (wl >= seqlen_k) wl = -1;
  if (wr >= seqlen_k) wr = -1;
  if (causal) wr = 0;
  Windows w;
  w.causal_alibi = (wl < 0 && wr == 0) ? 1 : 0;
  w.left = wl < 0 ? -1 : static_cast<int>(wl);
  w.right = wr < 0 ? -1 : static_cast<int>(wr);
  return w;
}

// Scratch memory of a forward call that may be split along the keys.
struct Scratch {
  void* ptr;
  int64_t bytes;
  bool holds(int64_t need) const { return ptr != nullptr && bytes >= need && reinterpret_cast<uintptr_t>(ptr) % 256 == 0; }
};

// ---- dense forward with few query rows per kv head (fwd_decode_sm100.cu)
struct DecodePlan {
  int rows = 0;            // query rows per kv head; 0: the path does not take this call
  int tile_lo = 0, tiles = 0;
  int grid = 0, whole_grid = 0;  // CTAs with a workspace, and without one
  bool split = false;            // some unit is shared by CTAs (needs the workspace)
  int64_t flag_bytes = 0, workspace_bytes = 0;
};

// Is the few-row kernel the faster one for a call that it can take? Its consumers do mma.sync on 16, 32 or 64 rows, so a
// key tile costs it more the more rows there are, and a unit's end (parts of eight warps become one) costs it more than
// the general kernel's; it wins where the general kernels read K and V once per query head of a group, or leave SMs idle.
// Both times are estimated in us: a launch, then per CTA its units and its key tiles, or K and V at the memory's rate, then
// the merge of parts. Constants fitted to 5200 measured calls (1 to 64 rows, groups of 1 to 64, 1 to 1000 units, 64 to 16384
// keys, D 64 to 256, both ways each): median error 3-9 %, hence the margin. With the rule 27 of these calls are more than 5 %
// slower than the other way (up to 1.3 times, single heads' worth of work that the shared tiles finish sooner), without it
// 1354 (up to 2.6 times): B64 H8 Sq 64 Sk 64 D128 35 us against 17, B5 H8 Sq 64 Sk 384 D256 25 against 13.
inline bool few_rows_win(const fa2_fwd_args* a, const DecodePlan& d, int64_t keys, int64_t sms) {
  struct Cost { double launch, unit, tile, merge; };
  static constexpr Cost kFew[4][3] = {{{4.5, 1.85, 0.62, 2.9}, {3.9, 2.4, 0.87, 4.7}, {3.4, 3.4, 1.42, 6.3}},
                                      {{3.65, 2.7, 0.94, 3.9}, {3.2, 4.0, 1.52, 5.9}, {3.0, 6.0, 2.1, 9.4}},
                                      {{3.1, 3.85, 1.33, 4.2}, {2.5, 5.7, 2.27, 7.45}, {2.4, 8.95, 3.0, 12.4}},
                                      {{3.25, 4.5, 1.69, 3.6}, {2.7, 6.8, 2.73, 8.4}, {1.2, 11.3, 4.27, 16.2}}};
  static constexpr Cost kGeneral[4] = {{6.4, 1.2, 1.16, 6.1}, {6.75, 1.17, 1.28, 8.55}, {3.0, 3.75, 1.76, 0}, {2.6, 4.3, 1.8, 0}};
  const int atoms = (a->head_dim - 1) / 64, row_tiles = decode_row_tiles(d.rows);
  const Cost& f = kFew[atoms][row_tiles == 4 ? 2 : row_tiles - 1];
  const Cost& g = kGeneral[atoms];
  const double units = static_cast<double>(a->batch) * a->heads_k, heads = static_cast<double>(a->batch) * a->heads;
  const double memory = units * keys * a->head_dim * 4 / 5.9e6;
  // the longest share: its tiles, and the units that it ends in
  double tiles, ends;
  if (d.split) {
    tiles = std::ceil(units * d.tiles / d.grid);
    ends = units <= sms ? 1 : units / d.grid + 1;
  } else {
    ends = std::ceil(units / d.grid);
    tiles = ends * d.tiles;
  }
  const double few = f.launch + std::max(ends * f.unit + tiles * f.tile, memory) + (d.split ? f.merge : 0);
  // One work tile per head; head dims up to 128 may share it between CTAs (plan_stream).
  const double blocks = a->head_dim <= 128 ? d.tiles : (keys + 63) / 64 / 2.0;
  double general = std::ceil(heads / sms) * (g.unit + blocks * g.tile);
  const double shares = std::min<double>(sms, std::floor(heads * d.tiles / 3));
  if (a->head_dim <= 128 && heads <= sms && shares >= 2)
    general = std::min(general, heads * d.tiles / shares * g.tile + (heads / shares + 1) * g.unit + g.merge);
  return few < 0.95 * (g.launch + std::max(general, memory));
}

inline DecodePlan decode_plan(const fa2_fwd_args* a, int sm_count) {
  DecodePlan d;
  const int64_t rows = static_cast<int64_t>(a->seqlen_q) * (a->heads / a->heads_k);
  if (rows <= 0 || rows > kDecodeMaxRows || a->seqlen_k <= 0 || a->head_dim <= 0 || a->head_dim > 256) return d;
  const Windows w = normalise_windows(a->window_left, a->window_right, a->causal != 0, a->seqlen_k, false);
  const int64_t off = static_cast<int64_t>(a->seqlen_k) - a->seqlen_q;
  int64_t lo = 0, hi = a->seqlen_k;
  if (w.left >= 0) lo = std::max<int64_t>(0, off - w.left);
  if (w.right >= 0) hi = std::min<int64_t>(hi, a->seqlen_q - 1 + off + w.right + 1);
  if (hi <= lo) return d;  // no row sees a key
  d.rows = static_cast<int>(rows);
  d.tile_lo = static_cast<int>(lo / 128);
  d.tiles = static_cast<int>((hi + 127) / 128) - d.tile_lo;
  const int64_t units = static_cast<int64_t>(a->batch) * a->heads_k, n = units * d.tiles, sms = sm_count;
  // Whole units per CTA, as evenly as that goes: what happens without a workspace.
  const int64_t per_cta = (units + sms - 1) / sms;
  d.whole_grid = d.grid = static_cast<int>((units + per_cta - 1) / per_cta);
  // Splitting units over CTAs costs about 5 us at the end (parts to memory, flags, merge), as much as a CTA takes for
  // four tiles of its own. Few units: each is cut into as many equal parts as the SMs allow and leave three tiles; at
  // most 24, because one CTA merges them. More units than SMs: equal shares of the whole list when the last,
  // incomplete round of whole units would take more than five tiles longer.
  if (units <= sms) {
    const int64_t parts = std::min<int64_t>({sms / units, 24, d.tiles / 3});
    if (parts > 1) d.grid = static_cast<int>(units * parts);
  } else if (per_cta * d.tiles - n / sms > 5) {
    d.grid = sm_count;
  }
  d.split = d.grid != d.whole_grid || (units > sms && d.grid == sm_count && units % sms != 0);
  if (!few_rows_win(a, d, hi - lo, sms)) return DecodePlan{};
  if (d.split) {
    const int64_t dim = (a->head_dim + 63) / 64 * 64;
    d.flag_bytes = (2 * static_cast<int64_t>(d.grid) * 8 + 255) / 256 * 256;
    d.workspace_bytes = d.flag_bytes + 2 * static_cast<int64_t>(d.grid) * 16 * decode_row_tiles(d.rows) * (dim + 2) * 4;
  }
  return d;
}

// Does the few-row kernel start beside the end of the kernel before it? That saves 2-3 us a call. But the CTAs of the next call
// settle on the SMs that the present one leaves idle, the rest on whichever end first: they no longer lie evenly over the chip,
// which costs calls that read at the memory's rate on a part of the SMs more than it saves. Without it, with it, us a call, D128:
// 80 CTAs of 63 key tiles (4 MB of K and V each) 53.3, 66.0; 96 CTAs of 128 tiles 118, 132; 128 of 128 tiles 154, 168. On the
// other side of the line: 80 CTAs of 8 tiles 12.3, 10.2; 128 of 16 tiles (1 MB) 27.3, 25.2; 136 of 128 tiles 178, 172.
inline bool decode_starts_early(const fa2_fwd_args* a, int tiles_per_unit, int grid, int sm_count) {
  const int64_t tiles = static_cast<int64_t>(a->batch) * a->heads_k * tiles_per_unit;
  return 10 * grid >= 9 * sm_count || tiles * 128 * a->head_dim * 4 / grid <= 1 << 20;
}

// ---- dense forward with few work tiles (fwd_sm100.cu, SHARED): a work tile is 256 query rows of a head, one CTA at a
// time works on it, and with fewer tiles than SMs some have nothing to do. Calls with more tiles are not shared, also
// where a last, nearly empty round would gain (H32 Sq 1500 Sk 16384, 192 tiles: 454 -> 392 us): sharing makes the bits of a
// head depend on how many tiles the call has. A caller that needs them independent for any size leaves the scratch memory
// out (fa2_fwd).
struct StreamPlan {
  int grid = 0;  // 0: one tile per CTA at a time
  int64_t workspace_bytes = 0;
  uint16_t start[kMaxStreamBlocks + 1];
};
inline void plan_stream(const fa2_fwd_args* a, int sm_count, StreamPlan* out) {
  const int64_t mblk = (static_cast<int64_t>(a->seqlen_q) + 255) / 256;
  if (a->head_dim > 128 || mblk <= 0 || mblk > kMaxStreamBlocks || a->seqlen_k <= 0) return;
  const int64_t heads = static_cast<int64_t>(a->batch) * a->heads, tiles = heads * mblk;
  if (tiles > sm_count) return;
  const Windows w = normalise_windows(a->window_left, a->window_right, a->causal != 0, a->seqlen_k, false);
  const int64_t off = static_cast<int64_t>(a->seqlen_k) - a->seqlen_q;
  int64_t total = 0, longest = 0;
  for (int64_t m = 0; m < mblk; ++m) {
    // Key blocks of the tile: the union over its two 128-row stages, as the kernel walks it.
    int64_t jlo = INT64_MAX, jhi = 0;
    for (int s = 0; s < 2; ++s) {
      const int64_t r_lo = m * 256 + s * 128;
      if (r_lo >= a->seqlen_q) break;
      const int64_t r_hi = std::min<int64_t>(r_lo + 127, a->seqlen_q - 1);
      int64_t hi = a->seqlen_k, lo = 0;
      if (w.right >= 0) hi = std::min(hi, r_hi + off + w.right + 1);
      if (w.left >= 0) lo = std::max<int64_t>(0, r_lo + off - w.left);
      if (hi > lo) {
        jlo = std::min(jlo, lo / 128);
        jhi = std::max(jhi, (hi + 127) / 128);
      }
    }
    if (jhi <= jlo) return;  // a tile without keys is in no share
    if (total + jhi - jlo > UINT16_MAX) return;
    out->start[m] = static_cast<uint16_t>(total);
    total += jhi - jlo;
    longest = std::max(longest, jhi - jlo);
  }
  out->start[mblk] = static_cast<uint16_t>(total);
  const int64_t units = total * heads;
  if (units > INT32_MAX / 2) return;
  // Costs in cycles: a key block, a tile's start and end, a part's way to memory, and the merge (a launch, and the parts
  // written and read back, which at D128 hits memory and not the L2); at least three key blocks per CTA. Checked on 1384
  // calls timed with and without sharing (2 to 148 tiles, Sq 65 to 4000, Sk 384 to 9000, masks): of the 231 that D64
  // shares none is slower for it, of the 180 that D128 shares two are by more than 2 % (3 %); the best are 5 times as
  // fast. H4 Sq 128 Sk 9000 D64 94 -> 23 us, H20 Sq 512 Sk 4096 D128 66 -> 46. With the constants of D64 26 more calls of D128
  // were shared, among them H12 Sq 2000 Sk 2048 causal (39 -> 45) and H50 Sq 512 Sk 4096 causal (70 -> 79).
  const bool d128 = a->head_dim > 64;
  const double t_blk = d128 && a->seqlen_q <= 128 ? 2150 : 3300, t_tile = 6000, t_part = 4000, t_merge = 7000;
  const double part_rate = d128 ? 1400 : 3000;  // bytes a cycle
  const int64_t grid = std::min<int64_t>(sm_count, units / 3);
  if (grid < 2) return;
  const double whole = longest * t_blk + t_tile;
  const int64_t bytes = 2 * grid * stream_slot_floats(d128 ? 128 : 64) * 4;
  const double shared = static_cast<double>(units) / grid * t_blk + (static_cast<double>(tiles) / grid + 1) * t_tile + t_part +
                        t_merge + static_cast<double>(std::min<int64_t>(grid, tiles) + grid) / (2.0 * grid) * bytes / part_rate;
  if (shared > 0.92 * whole) return;
  out->grid = static_cast<int>(grid);
  out->workspace_bytes = (bytes + 255) / 256 * 256;
}

// ---- order of the backward's CTAs. One CTA walks a key block of a (batch, kv head); CTAs start in grid order, so a call
// ends with whatever starts last. Under a causal mask the first key block of a head sees every query row and the last one
// only its own: listed head by head, the last head's long walks start late and most SMs wait for them. So a group of
// heads lists all first key blocks, then all second ones ...: the call ends with short walks. What the group's CTAs read
// and add into should stay in the L2 (126 MB), so calls of many CTAs, whose end weighs little, take groups of about
// 96 MB (of Q, dO, the accumulator, K and V); with up to four CTAs per SM the end weighs more than the traffic. Whole heads are
// dealt out evenly, rounded up, so that a group of two or three large heads can be nearly twice as large: the longer list is
// worth more than the bound (B2 H64/8 S8192 in pairs of 136 MB 7763 us, one by one 8037). Forward and
// backward, causal bf16, head by head -> grouped: B4 H16/4 S2048 softcap 448 -> 347 us, B2 H32/8 S4096 1183 -> 1001,
// B4 H16 S1000 128 -> 119, B4 H16/8 S2048 D256 885 -> 834, B1 H32 S16384 7444 -> 7358 (in groups of 250 MB 7602).
// Walks of the same length have no such end, but side by side those of one head add into the same rows at the same time;
// small groups mix them: B32 H12 S509 D64 232 -> 228 us, B16 H16 S2048 without a mask 2191 -> 2170 (all heads: 2757). Sliding
// windows are taken for such walks; head by head, in small groups, in groups as for the causal mask: B2 H16 S4096 D64 window 1023
// 213, 215, 207 us, B16 H16 S2048 D128 window 1023 1152, 1136, 1164, B1 H16/4 S8192 D128 window 4095 824, 815, 866.
inline int bwd_head_group(const fa2_bwd_args* a, const Windows& w, int sm_count) {
  if (a->cu_seqlens_q != nullptr) return 1;
  const int64_t heads = std::max<int64_t>(static_cast<int64_t>(a->batch) * a->heads_k, 1);
  const int64_t ctas = heads * ((a->seqlen_k + 127) / 128) * (a->head_dim > 128 ? 2 : 1);
  const int64_t bytes = (static_cast<int64_t>(a->heads) * a->seqlen_q * 8 + static_cast<int64_t>(a->heads_k) * a->seqlen_k * 4) *
                        a->head_dim * a->batch;
  const bool falling = w.right >= 0 && w.left < 0;
  const int64_t limit = !falling ? 16 << 20 : ctas > 4 * sm_count ? 96 << 20 : 320 << 20;
  const int64_t groups = std::min(heads, bytes / limit + 1);
  return static_cast<int>((heads + groups - 1) / groups);
}

// The same for the kernel that computes dQ alone, one CTA per 128 query rows of a head: K and V of a group, which its CTAs
// share, take about 64 MB.
inline int bwd_dq_head_group(const fa2_bwd_args* a, const Windows& w) {
  const int64_t heads = std::max<int64_t>(static_cast<int64_t>(a->batch) * a->heads, 1);
  if (w.right < 0 || w.left >= 0) return 1;
  const int64_t bytes = static_cast<int64_t>(a->seqlen_k) * a->head_dim * 4 * a->heads_k * a->batch;
  const int64_t groups = std::min(heads, bytes / (64 << 20) + 1);
  return static_cast<int>((heads + groups - 1) / groups);
}

// ---- pairs of CTAs (bwd_pair_sm100.cu). Does a backward call that is not split run on them? They add half as much into the dQ
// accumulator, which is what large calls pay for, in time and in power; but both CTAs of a pair walk the query blocks that either of
// them sees, and an iteration alone is no faster. Forward and backward in a steady loop (1000 W), one CTA per key block -> pairs:
// B1 H32 S16384 causal 7709 -> 7461 us, B4 H16/4 S4096 2025 -> 1955, B16 H16 S2048 2265 -> 2220, B2 H32/8 S2048 557 -> 542,
// B4 H16 S4096 causal 1144 -> 1133; with walks of less than 16 blocks B16 H16 S2048 causal 1364 -> 1385, B2 H16 S8192 window 1023
// 684 -> 711; with few CTAs B1 H8/2 S8192 causal 545 -> 551; a soft cap, whose tanh makes the arithmetic the longer part, B4 H16/4 S4096
// causal 1267 -> 1352; B2 H16 S8192 D96 3549 -> 3541. With an odd number of key blocks one CTA of a head has no keys and walks for nothing, which
// a few key blocks do not make up for: B8 H16 Sq 2048 Sk 98 179 -> 207, 354 299 -> 330, 610 425 -> 452, 1122 657 -> 680, 1634 917 -> 929; on this side 1890
// 1029 -> 1036 (B4 Sq 4096 1003 -> 982), 2658 1423 -> 1410, B8 H16/4 S2146 1165 -> 1135, causal, where that walk is short, B4 H16 S3170 718 -> 714.
inline bool bwd_takes_pairs(const fa2_bwd_args* a, const Windows& w, int sm_count) {
  if (a->cu_seqlens_q != nullptr || (a->which & 3) != 3 || a->head_dim <= 96 || a->head_dim > 128 || a->softcap > 0.f ||
      a->alibi_slopes != nullptr)
    return false;
  const int64_t pairs = (static_cast<int64_t>(a->seqlen_k) + 255) / 256, off = static_cast<int64_t>(a->seqlen_k) - a->seqlen_q;
  if (2 * pairs * a->batch * a->heads_k < sm_count * 3 / 2) return false;
  // Query blocks of a head that the first and the last pair walk. Their mean is that of all without a mask and, with no more keys than queries,
  // under a causal one; with more keys or a window on both sides that is larger, and the line lies further up: B2 H16 S8192 causal window
  // 2047 1032, 1031 (a mean of 18 blocks, refused), 3071 1343, 1322 (26, refused), 4095 1593, 1560; Sq 2048 Sk 8192 causal 922, 902 (refused), Sq 4096
  // 1520, 1474.
  auto blocks = [&](int64_t n0) {
    const int64_t n_last = std::min<int64_t>(n0 + 255, a->seqlen_k - 1);
    const int64_t lo = w.right >= 0 ? std::max<int64_t>(0, n0 - off - w.right) : 0;
    const int64_t hi = w.left >= 0 ? std::min<int64_t>(a->seqlen_q, n_last - off + w.left + 1) : a->seqlen_q;
    return hi > lo ? (hi + 127) / 128 - lo / 128 : 0;
  };
  const int64_t first = blocks(0), last = blocks((pairs - 1) * 256);
  if ((a->seqlen_k + 127) / 128 % 2 == 1 && 16 * last > pairs * (first + last)) return false;
  return first + last >= 2 * 16;
}

// Head dims 192 and 256 (bwd_wide_pair_sm100.cu, which has more figures). Its query blocks have 128 rows, those of the other kernel 64,
// and at head dim 192 a quarter of what it does for dK, dV and dQ is padding: calls that pad their rows by a fifth more than in blocks
// of 64 stay there. Without the line, before and after, us: D192 B16 H8 S300 142, 145, B16 H16/4 S300 causal 176, 183, B16 H8 S320 causal
// 125, 129; on this side B16 H8 S450 233, 214, B32 H8 S128 89, 82, B12 H16 S430 causal 259, 262. At head dim 256 such calls stay there if a third of
// their keys is padding too (the second CTA of a pair then has few of them): D256 B128 H16 S32 334, 408, B64 H16 S60 208, 238, B32 H16 S130
// 271, 286, B30 H32 S155 causal 488, 506; on this side B30 H16 S190 311, 300, causal 282, 284, B16 H16 S260 288, 275, causal 241, 242, B64 H16
// S100 293, 282, B4 H16 Sq 64 Sk 2000 199, 194, B16 H32/4 S320 causal 385, 390.
inline bool bwd_wide_takes_pairs(const fa2_bwd_args* a) {
  if (a->cu_seqlens_q != nullptr || (a->which & 3) != 3) return false;
  auto padded = [](int64_t rows, int64_t block) { return (rows + block - 1) / block * block; };
  const bool few_padded_rows = 5 * padded(a->seqlen_q, 128) < 6 * padded(a->seqlen_q, 64);
  const bool few_padded_keys = 3 * static_cast<int64_t>(a->seqlen_k) >= 2 * padded(a->seqlen_k, 128);
  return (a->head_dim == 192 && few_padded_rows) || (a->head_dim == 256 && (few_padded_rows || few_padded_keys));
}

// ---- key blocks shared by several CTAs (bwd_sm100.cu: part_start). A CTA owns 128 keys of one kv head and walks the
// query blocks of all the group's heads; with few (batch, kv head, key block) triples most SMs would have nothing
// to do, or wait for the CTA with the longest walk.
struct BwdSplit {
  int items_per_head = 0;      // 0: not split
  int64_t part_elems = 0;      // elements of one slot (= elements of dK)
  int max_parts = 1;
  uint16_t start[kMaxSplitBlocks + 1];
  int64_t bytes() const { return items_per_head > 0 ? 2 * max_parts * ((part_elems * 4 + 255) / 256 * 256) : 0; }
  // Can the parts lie `before` bytes (a multiple of 256) behind the start of this workspace? They are written 32 bytes at a
  // time; the rest of the workspace needs 16-byte alignment only, so a workspace may be too odd for parts.
  bool fits(const void* workspace, int64_t workspace_bytes, int64_t before) const {
    return items_per_head > 0 && workspace != nullptr && workspace_bytes >= before + bytes() &&
           reinterpret_cast<uintptr_t>(workspace) % 256 == 0;
  }
};
inline void plan_bwd_split(const fa2_bwd_args* a, bool share, int sm_count, BwdSplit* out) {
  const int nblk = (a->seqlen_k + 127) / 128;
  const int64_t units = static_cast<int64_t>(a->batch) * a->heads_k;
  if (!share || a->cu_seqlens_q != nullptr || a->head_dim > 128 || (a->which & 2) == 0 || a->seqlen_q <= 0 || a->seqlen_k <= 0 ||
      nblk > kMaxSplitBlocks || units * nblk > 2 * sm_count)
    return;
  const Windows w = normalise_windows(a->window_left, a->window_right, a->causal != 0, a->seqlen_k, false);
  const int64_t off = static_cast<int64_t>(a->seqlen_k) - a->seqlen_q, group = a->heads / a->heads_k;
  int64_t n[kMaxSplitBlocks], most = 0, total = 0, least = INT64_MAX;
  for (int i = 0; i < nblk; ++i) {
    const int64_t n0 = i * 128LL, n_last = std::min<int64_t>(n0 + 127, a->seqlen_k - 1);
    int64_t lo = 0, hi = a->seqlen_q;
    if (w.right >= 0) lo = std::max<int64_t>(0, n0 - off - w.right);
    if (w.left >= 0) hi = std::min<int64_t>(hi, n_last - off + w.left + 1);
    n[i] = hi > lo ? ((hi + 127) / 128 - lo / 128) * group : 0;
    most = std::max(most, n[i]);
    least = std::min(least, n[i]);
    total += n[i];
  }
  // Costs in cycles, from clock stamps: an iteration of the walk, a CTA's start and end, and per byte of the parts
  // (written and read once each at the memory's rate). The same split for calls with and without dQ: dK and dV are the
  // same bits in both.
  const double t_it = a->head_dim > 64 ? 4300 : 3000, t_cta = 8500;
  const int64_t dkv = static_cast<int64_t>(a->batch) * a->seqlen_k * a->heads_k * a->head_dim;
  const double base_cost = 4000, part_cost = dkv * 16.0 / 3400;
  auto cost = [&](double items, double longest, double all, bool even) {
    if (items <= sm_count) return longest;
    if (even) return std::ceil(items / sm_count) * longest;
    // Walks of all heads in one list, heaviest first, leave little idle at the end; with a head after the other the last
    // head's long walks start late.
    return std::max(longest, all / sm_count + (bwd_head_group(a, w, sm_count) >= units ? t_cta : longest / 2));
  };
  double best = cost(static_cast<double>(units * nblk), most * t_it + t_cta, units * (total * t_it + nblk * t_cta), least == most);
  int best_parts = 1;
  for (int parts = 2; parts <= 8 && parts <= most; ++parts) {
    const int64_t len = (most + parts - 1) / parts;
    int64_t items = 0;
    for (int i = 0; i < nblk; ++i) items += std::max<int64_t>(1, (n[i] + len - 1) / len);
    const double c = cost(static_cast<double>(units * items), len * t_it + t_cta, units * (total * t_it + items * t_cta), true) +
                     base_cost + part_cost * parts;
    if (c < 0.95 * best) {
      best = c;
      best_parts = parts;
    }
  }
  if (best_parts == 1) return;
  const int64_t len = (most + best_parts - 1) / best_parts;
  out->start[0] = 0;
  for (int i = 0; i < nblk; ++i) {
    const int64_t parts = std::max<int64_t>(1, (n[i] + len - 1) / len);
    out->max_parts = std::max<int>(out->max_parts, static_cast<int>(parts));
    out->start[i + 1] = static_cast<uint16_t>(out->start[i] + parts);
  }
  out->items_per_head = out->start[nblk];
  out->part_elems = dkv;
}

}  // namespace fa2
