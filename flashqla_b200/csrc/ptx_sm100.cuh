// Thin inline-PTX wrappers for the Blackwell (sm_100a) primitives the kernels use:
// mbarriers with BOUNDED waits, TMA tiled copies (cp.async.bulk.tensor), tensor memory
// (tcgen05.alloc / ld / st) and the 5th-generation tensor-core MMA (tcgen05.mma) with its shared
// memory / instruction descriptors.  Every copy has one destination CTA (no clusters are launched).
#pragma once

#include <cuda.h>
#include <stdint.h>

#include "common.cuh"

namespace qla {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: gives up after `kSpinLimit` polls or `kWaitLimitNs` of wall time, whichever comes
// first (each try_wait itself blocks for a hardware-defined interval, so the poll count alone does not
// bound the time), records the failure in *status and returns false so that the caller can leave its
// loop.  A healthy kernel never gets near the limit.  The recorded word is
//   code | parity << 16 | warp << 20      (callers put the barrier's index into bits 8..15 of `code`).
// The first poll is inlined (the barrier has usually completed already); the polling loop is a single
// non-inlined copy: there are dozens of call sites and the per-chunk code of the chunk kernels has to
// fit the instruction cache.
constexpr uint32_t kSpinLimit = 1u << 20;
constexpr unsigned long long kWaitLimitNs = 2000000000ull;
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void record_wait_failure(int* status, int code, uint32_t parity) {
  if (status != nullptr) atomicCAS(status, 0, code | static_cast<int>(parity << 16) | static_cast<int>((threadIdx.x >> 5) << 20));
}
// The polling loop itself; `limit_ns` is kWaitLimitNs everywhere except in the self-test of this very path.
__device__ __forceinline__ bool mbar_wait_polling(uint64_t* bar, uint32_t parity, int* status, int code,
                                                  unsigned long long limit_ns) {
  const unsigned long long t0 = global_timer_ns();
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u) {
      if (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0)
        return false;  // another role already failed: do not keep the SM busy
      if (global_timer_ns() - t0 > limit_ns) break;
    }
  }
  record_wait_failure(status, code, parity);
  return false;
}

// One look at a barrier: mbarrier.test_wait never suspends the thread.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait executed by a CONVERGED warp, verdict warp-uniform (mbar_wait_addr).  The first poll is inline and not voted on:
// the lanes of a converged warp execute the try_wait as one instruction on one barrier word and see the
// same answer, so either all of them return here or all of them enter the (non-inlined) polling loop,
// whose vote makes the verdict uniform even at the edge of the time limit.
//
// It is made for kernels that live from their instruction cache.  All code that a CTA executes per chunk shares
// the SM's 32 KB instruction cache (beyond it a line costs some 40 cycles, measured with straight-line code; beyond
// 128 KB twice that), and a wait appears some thirty times in a scan kernel: here a call site is one try_wait on a
// 32-bit shared address and a two-argument call that is hardly ever taken.  What the slow path reports with
// (status word, first barrier, number of the first barrier in the status code) is left in shared memory by
// mbar_wait_setup, which must run before a barrier of the CTA that precedes every wait.
struct WaitContext {
  int* status;
  uint32_t first_bar;
  int code_base;
};
__device__ __forceinline__ WaitContext* mbar_wait_context() {
  __shared__ WaitContext ctx;
  return &ctx;
}
__device__ __forceinline__ void mbar_wait_setup(int* status, uint64_t* bars, int code_base) {
  WaitContext* c = mbar_wait_context();
  c->status = status;
  c->first_bar = smem_u32(bars);
  c->code_base = code_base;
}
__device__ __forceinline__ bool mbar_try_wait_addr(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.b32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(ok)
      : "r"(addr), "r"(parity)
      : "memory");
  return ok != 0;
}
static __device__ __noinline__ bool mbar_wait_addr_slow(uint32_t addr, uint32_t parity) {
  WaitContext* c = mbar_wait_context();
  const unsigned long long t0 = global_timer_ns();
  bool done = false;
  uint32_t i = 0;
  for (; i < kSpinLimit; ++i) {
    done = mbar_try_wait_addr(addr, parity);
    if (done) break;
    if ((i & 63u) == 63u) {
      if (c->status != nullptr && *reinterpret_cast<volatile int*>(c->status) != 0) return __all_sync(__activemask(), false);
      if (global_timer_ns() - t0 > kWaitLimitNs) break;
    }
  }
  if (!done)
    record_wait_failure(c->status, kStatusBarrierTimeout | ((c->code_base + static_cast<int>((addr - c->first_bar) >> 3)) << 8), parity);
  return __all_sync(__activemask(), done) != 0;
}
__device__ __forceinline__ bool mbar_wait_addr(uint32_t addr, uint32_t parity) {
  if (mbar_try_wait_addr(addr, parity)) return true;
  return mbar_wait_addr_slow(addr, parity);
}

// The wait of a warp that issues MMAs: no call.  Uniform registers do not survive a call, so that with one anywhere in the
// issuing loop every descriptor lives in ordinary registers and is moved over for each instruction.  Bounded like the others,
// but it reports nothing itself: the issuing warp does so behind its loop (report_issuer), where it costs the loop nothing.
// `alive` false: one poll.
__device__ __forceinline__ bool mbar_wait_nocall(uint32_t addr, uint32_t parity, bool alive,
                                                 unsigned long long limit_ns = kWaitLimitNs) {
  if (mbar_try_wait_addr(addr, parity)) return alive;
  const unsigned long long until = global_timer_ns() + (alive ? limit_ns : 0ull);
  while (!mbar_try_wait_addr(addr, parity))
    if (global_timer_ns() > until) return false;
  return alive;
}
// Several barriers at once: one look at all of them, whose latencies overlap (a wait that is over already takes some 70 cycles, and an
// issuer has ten of them per chunk), then one after the other.
__device__ __forceinline__ bool mbar_wait_nocall2(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred P, Q;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 Q, [%3], %4;\n"
      "and.pred P, P, Q;\nselp.b32 %0, 1, 0, P;\n}\n"
      : "=r"(ok) : "r"(a), "r"(pa), "r"(b), "r"(pb) : "memory");
  if (ok != 0) return true;
  return mbar_wait_nocall(a, pa, true) && mbar_wait_nocall(b, pb, true);
}
__device__ __forceinline__ bool mbar_wait_nocall3(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb, uint32_t c, uint32_t pc) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred P, Q, R;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 Q, [%3], %4;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 R, [%5], %6;\n"
      "and.pred P, P, Q;\nand.pred P, P, R;\nselp.b32 %0, 1, 0, P;\n}\n"
      : "=r"(ok) : "r"(a), "r"(pa), "r"(b), "r"(pb), "r"(c), "r"(pc) : "memory");
  if (ok != 0) return true;
  return mbar_wait_nocall(a, pa, true) && mbar_wait_nocall(b, pb, true) && mbar_wait_nocall(c, pc, true);
}
// `num_bars` (one past the kernel's last barrier) stands for "one of the issuer's waits".
__device__ __forceinline__ void report_issuer(int* status, bool alive, int num_bars) {
  if (!alive) record_wait_failure(status, kStatusBarrierTimeout | (num_bars << 8), 0);
}

__device__ __forceinline__ float ex2(float x) {  // 2^x, approximate (the MUFU behind __expf)
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rcp(float x) {  // 1 / x, approximate
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2(float x) {  // log2, approximate
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ------------------------------------------------------------------------------ fences
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ------------------------------------------------------------------------------ TMA
// Tiled 3-D load: coordinates are (x = innermost element, y, z); x * elem_size must be a multiple
// of 16 bytes.  Completion is signalled on `bar` with the byte count of the box.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// A 4-D box: both 64-column halves of a 128-wide tile in one copy (see make_tmap_halves).
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_l2_4d(const CUtensorMap* m, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// Bring a box into L2 only (no shared-memory destination, no completion tracking).
__device__ __forceinline__ void tma_prefetch_l2_3d(const CUtensorMap* m, int x, int y, int z) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory"); }
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* src, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// Untiled copy: both addresses on 16 bytes, a multiple of 16 bytes.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Wait until the bulk stores of all committed groups have finished READING shared memory.
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read_but1() {  // all but the newest group
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ------------------------------------------------------------------------------ tensor memory
// Allocate `ncols` (power of two >= 32) TMEM columns; executed by ONE full warp.  The base address
// is written to *dst_smem.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 32 bit: thread i of the warp reads lane (base lane + i); register j = column + j.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
        "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 16 lanes x 256 bit fragments: the warp reads lanes L .. L + 15 (L = lane field of the address: the first or
// the second half of the warp's 32-lane partition, i.e. the rows of an M = 64 accumulator placed at lane offset
// 0 or 16) and thread t = 4 g + c receives, per group j of eight columns, the four values
//   r[4j + 0..1] = (lane L + g,     columns 8j + 2c, 8j + 2c + 1)
//   r[4j + 2..3] = (lane L + g + 8, the same columns)
// - the accumulator layout of mma.sync m16n8 tiles.
__device__ __forceinline__ void tmem_ld_frag8(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
        "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_frag4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_frag2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// The inverse of tmem_ld_frag4: the warp writes the fragments (tmem_wait_st before they are announced).
__device__ __forceinline__ void tmem_st_frag4(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 16 lanes x 128 bit fragments of a tile of packed 16-bit values: thread 4 g + c receives, per group j of four 32-bit
// columns (eight values), r[2j] = (lane L + g, 32-bit column 4j + c), r[2j + 1] = (lane L + g + 8, the same column) -
// the registers of 8 x 8 matrices of 16-bit values.
__device__ __forceinline__ void tmem_ld_pack8(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x128b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_pack4(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x128b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// Store four 8 x 8 matrices of 16-bit values transposed: register x holds, in thread 4 g + c, the elements
// (row g, columns 2c, 2c + 1) of matrix x; lane i gives the address of memory row i % 8 (= column i % 8) of matrix i / 8.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t saddr, const uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
// Not transposed: register x holds, in thread 4 g + c, elements (row g, columns 2c, 2c + 1) of matrix x; lane i gives the
// address of row i % 8 of matrix i / 8.
__device__ __forceinline__ void stmatrix_x4(uint32_t saddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------------------ descriptors
// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets
// (all >> 4), descriptor version 1 at bit 46, swizzle mode at bits 61-63 (2 = 128-byte swizzle).
// For 128B-swizzled tiles the tile base must be 1024-byte aligned; stepping the start address by
// 32 bytes moves 16 bf16 along the contiguous direction inside the swizzle atom.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

enum : uint32_t { kMajorK = 0, kMajorMN = 1 };
enum : uint32_t { kFmtF16 = 0, kFmtBF16 = 1 };

// Instruction descriptor of tcgen05.mma.kind::f16 with fp32 accumulation.
__host__ __device__ constexpr uint32_t mma_idesc(uint32_t m, uint32_t n, uint32_t fmt, uint32_t a_major,
                                                  uint32_t b_major) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (a_major << 15) | (b_major << 16) | ((n >> 3) << 17) |
         ((m >> 4) << 24);
}

// ---- whole products issued by a CONVERGED warp.
// A tcgen05.mma is issued by one thread, but when that thread sits in a divergent branch every operand
// lives in per-thread registers and has to be moved to uniform registers one by one: measured ~55-68
// cycles of issue per instruction, more than the tensor pipe needs for N <= 128.  Issued from a
// converged warp with the leader picked by elect.sync INSIDE the asm block, the operand arithmetic stays
// on the uniform datapath and the cost drops to 22 cycles, below the pipe's own (34 at N = 64, 68 at N = 128).  (As a loop with an
// election per instruction it was 50: the issuer of a scan, with 40 products and a dozen waits per chunk, was what a chunk took.)
// Descriptor steps are 32-bit adds on the low word (the 14-bit address field never carries).
// All steps are in units of 16 bytes.  `JUMP` replaces `STEP` between k-steps 3 and 4 (the second
// 64-element half of a 128-wide operand).  Every block ends with up to two tcgen05.commit on the
// barriers whose shared-memory addresses are passed in (0 = none), so that a product and its completion
// signal cost one leader election.
#define QLA_UMMA_COMMITS(B1, B2)                                                                      \
  "setp.ne.b32 c1, " B1 ", 0;\nsetp.ne.b32 c2, " B2 ", 0;\nand.pred c1, c1, e;\nand.pred c2, c2, e;\n"   \
  "@c1 tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [" B1 "];\n"              \
  "@c2 tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [" B2 "];\n"
#define QLA_UMMA_SS_STEP(SA, SB)                                                                     \
  "add.u32 alo, alo, " SA "; add.u32 blo, blo, " SB "; mov.b64 da, {alo, ahi}; mov.b64 db, {blo, bhi};\n" \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, t;\n"
#define QLA_UMMA_SS_HEAD                                                                              \
  "{\n.reg .pred p, t, e, c1, c2;\n.reg .b32 alo, ahi, blo, bhi;\n.reg .b64 da, db;\n"                         \
  "elect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\n"                         \
  "mov.b64 {alo, ahi}, %1;\nmov.b64 {blo, bhi}, %2;\n"                                                 \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
// D[tmem] (+)= A[smem] B[smem], K = 64 (four instructions).
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ss_k64(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            bool accumulate, uint32_t commit1 = 0, uint32_t commit2 = 0) {
  asm volatile(QLA_UMMA_SS_HEAD QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6")
               QLA_UMMA_COMMITS("%7", "%8") "}\n"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)),
                 "n"(A_STEP), "n"(B_STEP), "r"(commit1), "r"(commit2)
               : "memory");
}
// The same, M = 128, writing only the accumulator's lanes 0..63 whose bit of `mask_low` is clear and 64..127 of `mask_high`
// (either mask serves two quadrants of 32 lanes).
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ss_k64_lanes(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                  uint32_t mask_low, uint32_t mask_high, bool accumulate, uint32_t commit = 0) {
#define QLA_UMMA_LANES_STEP                                                                                               \
  "add.u32 alo, alo, %4; add.u32 blo, blo, %5; mov.b64 da, {alo, ahi}; mov.b64 db, {blo, bhi};\n"                          \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%6, %6, %7, %7}, t;\n"
  asm volatile(
      "{\n.reg .pred p, t, e, c1;\n.reg .b32 alo, ahi, blo, bhi;\n.reg .b64 da, db;\n"
      "elect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %9, 0;\nsetp.eq.b32 t, 0, 0;\nsetp.ne.b32 c1, %8, 0;\nand.pred c1, c1, e;\n"
      "mov.b64 {alo, ahi}, %1;\nmov.b64 {blo, bhi}, %2;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%6, %6, %7, %7}, p;\n"
      QLA_UMMA_LANES_STEP QLA_UMMA_LANES_STEP QLA_UMMA_LANES_STEP
      "@c1 tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%8];\n}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(A_STEP), "n"(B_STEP), "r"(mask_low), "r"(mask_high), "r"(commit),
        "r"(static_cast<uint32_t>(accumulate))
      : "memory");
#undef QLA_UMMA_LANES_STEP
}
// The same with everything known at run time only: low words of both descriptors and their steps; `hi` is the high word.
__device__ __forceinline__ void umma_ss_k64_steps(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc,
                                                  bool accumulate, uint32_t a_step, uint32_t b_step) {
  asm volatile(
      "{\n.reg .pred p, t, e;\n.reg .b32 alo, blo;\n.reg .b64 da, db;\n"
      "elect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %5, 0;\nsetp.eq.b32 t, 0, 0;\n"
      "mov.b32 alo, %1;\nmov.b32 blo, %2;\nmov.b64 da, {alo, %3};\nmov.b64 db, {blo, %3};\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n"
      "add.u32 alo, alo, %6; add.u32 blo, blo, %7; mov.b64 da, {alo, %3}; mov.b64 db, {blo, %3};\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n"
      "add.u32 alo, alo, %6; add.u32 blo, blo, %7; mov.b64 da, {alo, %3}; mov.b64 db, {blo, %3};\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n"
      "add.u32 alo, alo, %6; add.u32 blo, blo, %7; mov.b64 da, {alo, %3}; mov.b64 db, {blo, %3};\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, t;\n}\n"
      ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "r"(a_step), "r"(b_step)
      : "memory");
}
// D[tmem] (+)= A[smem] B[smem], K = 128 (eight instructions).
template <int A_STEP, int A_JUMP, int B_STEP, int B_JUMP>
__device__ __forceinline__ void umma_ss_k128(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             bool accumulate, uint32_t commit1 = 0, uint32_t commit2 = 0) {
  asm volatile(QLA_UMMA_SS_HEAD QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6")
               QLA_UMMA_SS_STEP("%7", "%8") QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6") QLA_UMMA_SS_STEP("%5", "%6")
               QLA_UMMA_COMMITS("%9", "%10") "}\n"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)),
                 "n"(A_STEP), "n"(B_STEP), "n"(A_JUMP), "n"(B_JUMP), "r"(commit1), "r"(commit2)
               : "memory");
}
#undef QLA_UMMA_SS_STEP
#undef QLA_UMMA_SS_HEAD
#define QLA_UMMA_TS_STEP(SB)                                                                         \
  "add.u32 aa, aa, 8; add.u32 blo, blo, " SB "; mov.b64 db, {blo, bhi};\n"                             \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], db, %3, t;\n"
#define QLA_UMMA_TS_HEAD                                                                              \
  "{\n.reg .pred p, t, e, c1, c2;\n.reg .b32 aa, blo, bhi;\n.reg .b64 db;\n"                                   \
  "elect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\nsetp.eq.b32 t, 0, 0;\n"                         \
  "mov.b32 aa, %1;\nmov.b64 {blo, bhi}, %2;\n"                                                         \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
// D[tmem] (+)= A[tmem] B[smem], K = 64: A advances 8 TMEM columns (16 values of 16 bits) per instruction.
template <int B_STEP>
__device__ __forceinline__ void umma_ts_k64(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                            bool accumulate, uint32_t commit1 = 0, uint32_t commit2 = 0) {
  asm volatile(QLA_UMMA_TS_HEAD QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5")
               QLA_UMMA_COMMITS("%6", "%7") "}\n"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "n"(B_STEP),
                 "r"(commit1), "r"(commit2)
               : "memory");
}
// The same with the second half of A (values 32..63) 32 columns behind the first.
#define QLA_UMMA_TS_STEP_A(SA, SB)                                                                   \
  "add.u32 aa, aa, " SA "; add.u32 blo, blo, " SB "; mov.b64 db, {blo, bhi};\n"                        \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], db, %3, t;\n"
template <int B_STEP>
__device__ __forceinline__ void umma_ts_k64_halves(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                   bool accumulate, uint32_t commit1 = 0, uint32_t commit2 = 0) {
  asm volatile(QLA_UMMA_TS_HEAD QLA_UMMA_TS_STEP_A("8", "%5") QLA_UMMA_TS_STEP_A("24", "%5") QLA_UMMA_TS_STEP_A("8", "%5")
               QLA_UMMA_COMMITS("%6", "%7") "}\n"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "n"(B_STEP),
                 "r"(commit1), "r"(commit2)
               : "memory");
}
#undef QLA_UMMA_TS_STEP_A
// D[tmem] (+)= A[tmem] B[smem], K = 128.
template <int B_STEP, int B_JUMP>
__device__ __forceinline__ void umma_ts_k128(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             bool accumulate, uint32_t commit1 = 0, uint32_t commit2 = 0) {
  asm volatile(QLA_UMMA_TS_HEAD QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%6")
               QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5") QLA_UMMA_TS_STEP("%5")
               QLA_UMMA_COMMITS("%7", "%8") "}\n"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(static_cast<uint32_t>(accumulate)), "n"(B_STEP),
                 "n"(B_JUMP), "r"(commit1), "r"(commit2)
               : "memory");
}
#undef QLA_UMMA_TS_STEP
#undef QLA_UMMA_TS_HEAD
#undef QLA_UMMA_COMMITS
// tcgen05.commit from a converged warp (same elected lane as the umma_* helpers).
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar))
      : "memory");
}

// Byte offset of element (row, 16-byte chunk `c16`) inside a 128B-swizzled tile whose rows are
// 128 bytes (64 bf16) wide: chunk index is XORed with (row mod 8).
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t c16) {
  return row * 128u + ((c16 ^ (row & 7u)) << 4);
}

}  // namespace ptx

// ------------------------------------------------------------------------------ host: tensor maps
// cuTensorMapEncodeTiled fetched through the runtime (no link-time dependency on libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();

// Map over a [rows(tokens), heads, width] tensor of 16-bit elements; box = [box_rows, 1, box_width].
int make_tmap_3d(CUtensorMap* out, const void* base, uint64_t tokens, uint64_t heads, uint64_t width,
                 uint32_t box_rows, uint32_t box_width, bool swizzle128, bool is_bf16);
// Map over a [tokens, heads, 128] tensor of 16-bit elements as (64 columns, heads, tokens, 2 halves): one box
// [2][box_rows][64] is a 128-wide tile in the two 128B-swizzled halves that the MMA descriptors read.
int make_tmap_halves(CUtensorMap* out, const void* base, uint64_t tokens, uint64_t heads, uint32_t box_rows, bool is_bf16);

}  // namespace qla
