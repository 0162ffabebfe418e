// Thin inline-PTX wrappers for the sm_100a features the attention kernels use:
// mbarrier, TMA (cp.async.bulk.tensor, no multicast anywhere), tcgen05 MMA with TMEM
// accumulators, tcgen05.ld/st, and the shared-memory / instruction descriptors.
//
// Every wait in here is bounded: a wait that runs out records an error code and makes
// all later waits of the CTA return immediately, so a pipeline bug ends the kernel
// instead of hanging the GPU.
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <stdint.h>
#include <type_traits>

namespace fa2 {

// ---------------------------------------------------------------- addresses
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One try_wait: the hardware may park the thread until the phase completes (it is woken then) or a
// system-dependent time limit expires, so a polling warp does not take issue slots from the warps that share
// its scheduler.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Abort state of one CTA, a word of shared memory: 0, or the site code of the first wait that ran out (a wait stores its code a few
// instructions after it has found the word clear; of two that run out within those, the later one's stays). report_abort hands it on
// when the kernel ends.
struct WaitCtl {
  volatile int* abort_flag;
};

// Upper bound of one wait in SM clock cycles (about a second at B200 clocks).
#ifndef FA2_WAIT_LIMIT_CYCLES
#define FA2_WAIT_LIMIT_CYCLES (1ll << 31)
#endif
static_assert(FA2_WAIT_LIMIT_CYCLES > 0 && FA2_WAIT_LIMIT_CYCLES < (1ll << 32), "waits compare 32 bits of the clock");

__device__ __forceinline__ uint32_t clock32() {
  uint32_t c;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
  return c;
}

// Returns false when the wait ran out (or the CTA already aborted). A kernel has 20 to 40 of these in line and its roles share the
// SM's instruction cache, so there is no more in it than it needs.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint32_t t0 = clock32();
  do {
    if (mbar_try_wait(bar, parity)) return true;
    if (*ctl.abort_flag) return false;
  } while (clock32() - t0 < static_cast<uint32_t>(FA2_WAIT_LIMIT_CYCLES));
  *ctl.abort_flag = code;
  return false;
}
// The longer form, which reads the clock at every eighth try: for a kernel that names this type (the plain forward at head dim 128).
struct SeldomWaitCtl : WaitCtl {};
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const SeldomWaitCtl& ctl, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*ctl.abort_flag) return false;
    if ((it & 7u) == 0u && clock64() - t0 > FA2_WAIT_LIMIT_CYCLES) break;
  }
  if (!*ctl.abort_flag) *ctl.abort_flag = code;
  return false;
}

// The same wait for short hand-offs between the warps of one role: it probes the phase without letting the
// hardware park the thread (a parked thread was seen to come back thousands of cycles after the phase
// completed), at the price of issue slots while it spins.
__device__ __forceinline__ bool mbar_wait_spin(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code) {
  const uint32_t t0 = clock32();
  do {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*ctl.abort_flag) return false;
  } while (clock32() - t0 < static_cast<uint32_t>(FA2_WAIT_LIMIT_CYCLES));
  *ctl.abort_flag = code;
  return false;
}

// After the CTA's last barrier, by one thread: the site code goes to the status word (global memory, may be null), which keeps the
// first CTA's.
__device__ __forceinline__ void report_abort(const volatile int* abort_flag, int* status) {
  const int code = *abort_flag;
  if (code != 0 && status != nullptr) atomicCAS(status, 0, code);
}

// Wait of a whole warp. The vote brings the 32 lanes back together (they leave the polling loop in
// different iterations) and makes the outcome warp-uniform, so that the .sync.aligned tcgen05
// instructions that follow are executed by the converged warp.
template <class Ctl>
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, const Ctl& ctl, int code) {
  const bool ok = mbar_wait(bar, parity, ctl, code);
  return __all_sync(0xffffffffu, ok);
}

// ---------------------------------------------------------------- fences
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// ---------------------------------------------------------------- next CTA of the grid
// A running CTA takes over one that has not started. The request's answer (16 bytes) arrives in shared memory on an mbarrier
// that expects them; no request may follow one that was turned down.
__device__ __forceinline__ void ask_next_cta(uint32_t answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer),
               "r"(smem_u32(bar))
               : "memory");
}
// Its x index, or -1 if there is none left. The fence orders the read before the answer is overwritten.
__device__ __forceinline__ int next_cta(uint32_t answer) {
  int x;
  asm volatile(
      "{\n\t.reg .b128 a;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 a, [%1];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
      "mov.b32 %0, -1;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, a;\n\t"
      "fence.proxy.async.shared::cta;\n\t}"
      : "=r"(x)
      : "r"(answer)
      : "memory");
  return x;
}

// ---------------------------------------------------------------- dependent launch
// The kernels are launched so that a grid may start while the one before it in the stream ends (launch_grid). A grid
// touches global memory only behind early_wait, which returns once everything before it in the stream has completed
// and is visible; what precedes it (barriers, TMEM, descriptors) runs beside the end of that. Every CTA waits, so that a
// grid never ends before its predecessor. early_trigger, behind the wait, lets the next grid start as soon as all CTAs
// of this one have started. Every grid waits, whatever its arguments: memory that a call frees on its return is given to the
// next call in the stream, and only a grid that has waited is promised to see what was written before it. B1 H32/8 Sk 8192
// decoding 16.4 -> 13.0 us a call, B4 H16/4 S2048 softcap forward and backward 373 -> 366, B32 H12 S509 D64 229.4 -> 222.9.
// Packed batches and long few-row calls that leave SMs idle (decode_starts_early) start when the grid before them has ended.
// The memory-bound kernels of the backward are launched the usual way: their blocks otherwise settle on the SMs that the grid
// before them leaves first, and large calls got slower (forward and backward of B16 H16 S2048 D128 causal 1330 -> 1399 us).
__device__ __forceinline__ void early_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void early_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 4-D tiled load global -> shared, completion on an mbarrier. c0 is the innermost
// coordinate and must make c0 * element_size a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2,
                                             int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
// fp32 add-reduce of a shared-memory tile into global memory (used for dQ accumulation).
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2,
                                                  int c3) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::
                   "l"(reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- TMEM
// One warp allocates; the base address lands in shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------- descriptors
// 64-bit shared-memory matrix descriptor, 128-byte swizzle, sm_100 version field.
//   bits [0,14)  start address >> 4        bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) version = 1
//   bits [61,64) layout type (2 = SWIZZLE_128B)
// K-major operand (rows of 128 bytes along K): SBO = 1024 (8 rows), LBO unused (=1).
// MN-major operand (rows of 128 bytes along M/N, one row per k): SBO = bytes between
// groups of 8 k, LBO = bytes between 64-element chunks along M/N.
__host__ __device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// The same with 64-byte swizzle: rows of 64 bytes, 512 bytes for 8 of them.
__host__ __device__ __forceinline__ uint64_t make_smem_desc_64(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return make_smem_desc(saddr, lbo_bytes, sbo_bytes) ^ (6ull << 61);
}

// ---------------------------------------------------------------- MMA
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Variants that add compile-time offsets (in 16-byte units) to the descriptors inside the asm
// block: an unrolled k-step loop then costs two adds per MMA and no registers for precomputed
// descriptors (the compiler cannot hoist what it cannot see).
template <uint32_t AOFF16, uint32_t BOFF16>
__device__ __forceinline__ void mma_ss_o(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 ra, rb;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "add.s64 ra, %1, %5;\n\tadd.s64 rb, %2, %6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], ra, rb, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(AOFF16), "n"(BOFF16)
      : "memory");
}
template <uint32_t ACOL, uint32_t BOFF16>
__device__ __forceinline__ void mma_ts_o(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 rb;\n\t.reg .b32 ta;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "add.s64 rb, %2, %6;\n\tadd.u32 ta, %1, %5;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], rb, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(ACOL), "n"(BOFF16)
      : "memory");
}
// True in exactly one lane of a converged warp. A single-thread role entered through this predicate, rather than
// through a comparison of the lane index, lets the compiler keep the role's descriptors, addresses and loop
// counters in uniform registers: the issuer loop of the backward kernel shrank from 14.5 KB to 6.7 KB of code.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}

// Calls f(std::integral_constant<int, 0>{}) ... f(integral_constant<int, N-1>{}).
template <int N, int I = 0, class F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<N, I + 1>(f);
  }
}

// Arrive once on `bar` when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ---------------------------------------------------------------- CTA pairs
// Two CTAs of a cluster whose tensor cores work on one MMA of M = 128 or 256 rows, half of the rows in each CTA's TMEM. One thread of
// the CTA of rank 0 issues it; a descriptor names the same shared-memory offset in both: A has the CTA's own rows, B its half of the N
// rows (or columns). Measured: 128x128x16 takes 32 cycles, 256x128x16 64, with either operand A in shared memory or TMEM.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address of a shared-memory word of this CTA in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t peer_smem(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Arrival at a barrier of either CTA. What is handed over with it is tensor memory, ordered by the tcgen05 fences, or shared memory of
// this CTA, on which the writers' proxy fence has completed before. (With .release.cluster, which also waits for everything that the
// thread has sent to the other CTA, an arrival takes up to 1300 cycles in place of 50: B1 H32 S16384 8377 us in place of 7356.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Copy from this CTA's shared memory to the other one's; the bytes are counted at a barrier of the receiver.
__device__ __forceinline__ void bulk_copy_cluster(uint32_t cluster_dst, uint32_t src, uint32_t bytes, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(cluster_dst), "r"(src),
               "r"(bytes), "r"(cluster_bar)
               : "memory");
}
// tma_load_4d into this CTA, whose bytes are counted at a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* m, uint32_t cluster_bar, int c0, int c1, int c2,
                                                 int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(void* smem_dst, const CUtensorMap* m, uint32_t cluster_bar, int c0, int c1, int c2, int c3,
                                                 int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6, %7}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <uint32_t AOFF16, uint32_t BOFF16>
__device__ __forceinline__ void mma_pair_ss_o(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 ra, rb;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "add.s64 ra, %1, %5;\n\tadd.s64 rb, %2, %6;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], ra, rb, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(AOFF16), "n"(BOFF16)
      : "memory");
}
template <uint32_t ACOL, uint32_t BOFF16>
__device__ __forceinline__ void mma_pair_ts_o(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 rb;\n\t.reg .b32 ta;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "add.s64 rb, %2, %6;\n\tadd.u32 ta, %1, %5;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [ta], rb, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(ACOL), "n"(BOFF16)
      : "memory");
}
// Arrives at the barrier of both CTAs when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

// ---------------------------------------------------------------- TMEM <-> registers
// 32x32b: thread i of the warp owns TMEM lane (lane_base + i); register j is column (col + j).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- register budget
template <int N>
__device__ __forceinline__ void reg_alloc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_dealloc() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Bits [lo, hi) of a 32-bit word; either end may lie outside [0, 32). PTX shifts by 32 or more give zero.
__device__ __forceinline__ uint32_t bit_range(int lo, int hi) {
  uint32_t from_lo, from_hi;
  asm("shl.b32 %0, %1, %2;" : "=r"(from_lo) : "r"(0xffffffffu), "r"(max(lo, 0)));
  asm("shl.b32 %0, %1, %2;" : "=r"(from_hi) : "r"(0xffffffffu), "r"(max(hi, 0)));
  return from_lo & ~from_hi;
}
// v[i] = fill for every i outside [lo, hi). The tests go through words of 32 bits: one constant bit per element in
// place of two comparisons.
template <int N, typename T>
__device__ __forceinline__ void fill_outside(T* v, int lo, int hi, T fill) {
  static_assert(N % 32 == 0, "whole words");
#pragma unroll
  for (int c = 0; c < N; c += 32) {
    const uint32_t keep = bit_range(lo - c, hi - c);
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (!(keep & (1u << i))) v[c + i] = fill;
  }
}

// ---------------------------------------------------------------- math
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The hardware's tanh, good to 2^-11.
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// ---- packed fp32x2 arithmetic (two fp32 lanes in one 64-bit register; one issue slot for both)
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Pack two fp32 into one 32-bit word of two 16-bit floats: `lo` in bits [0,16).
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t r;
  if constexpr (BF16) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  } else {
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  }
  return r;
}

}  // namespace fa2
