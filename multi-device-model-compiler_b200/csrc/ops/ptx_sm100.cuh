// Thin inline-PTX wrappers for the Blackwell (sm_100a) features the tensor-core kernels
// use: mbarrier, TMA tile copies (never with cluster multicast), tcgen05 MMA with TMEM
// accumulators.  Every wait is bounded: it gives up after kWaitTimeoutNs, and the caller
// turns that into an error code in global memory instead of hanging the GPU.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace mdc {
namespace ptx {

constexpr unsigned long long kWaitTimeoutNs = 2000000000ull;  // 2 s

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// The warp's number, as a value that the compiler knows to be the same in all lanes: what a branch on it
// encloses is then code of a converged warp, with addresses and descriptors in uniform registers.  (Without
// it an MMA loop with a wait per k-block took 353 cycles a k-block, 289 with it, where the MMAs of
// 128 x 64 x 64 take 193.)
__device__ __forceinline__ int warp_index() {
  return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
}

// The MMA and TMA loops are run by a whole converged warp, and the instructions that one thread
// has to issue carry their own election (`elect.sync` picks the same lane every time).  A loop
// entered by lane 0 alone is divergent code to the compiler: its addresses and descriptors then
// go through vector registers and every tcgen05 / TMA instruction waits for the moves.  Measured
// in a one-tile Gemm: about 590 cycles per 64-wide k-block (four MMAs, one commit) in the
// one-lane form, 400 in this one; the MMAs of a 256 x 256 pair tile themselves need 512.

// Where one thread runs a role from end to end (attention: few MMAs between long waits), it is the elected one: to the
// compiler a branch on `elect.sync` holds one thread of a converged warp, a branch on the lane's number does not.  128 x
// 256 tokens, 8 heads of 128, causal 70.7 -> 64.8 us; 48 x 512, 16 heads of 64, padded 87.4 -> 85.2.  No `elect.sync`
// inside such a branch: the other lanes never come.

// ---------------- mbarrier ----------------
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity.  Returns false if `*abort_flag` (shared
// memory, set by any role that gave up) becomes non-zero or the time limit passes; the
// caller then records an error and leaves its loop.
// SLEEP_NS > 0 puts the thread to sleep between polls: for kernels in which many warps wait
// at once, whose polling would otherwise take the issue slots of the warps doing the work.
template <int SLEEP_NS = 0>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          volatile uint32_t *abort_flag) {
  // The global timer is slow to read, so the clock of the time limit only starts at the
  // 64th failed poll: an ordinary wait never touches it.
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if constexpr (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
    if ((++spins & 0x3f) == 0) {
      if (*abort_flag) return false;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > kWaitTimeoutNs) {
        *abort_flag = 1;
        return false;
      }
    }
  }
}

// The wait of a role that one elected thread runs from end to end (`if (elect_one()) { ... }`).
__device__ __forceinline__ bool mbar_wait_elected(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag) {
  return mbar_wait(bar, parity, abort_flag);
}

// The same wait for a whole (converged) warp: lane 0 polls, the others are released by the
// shuffle.  Keeps 31 of 32 threads off the barrier word and off the global timer, which is
// slow to read when hundreds of threads do so at once.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity,
                                               volatile uint32_t *abort_flag) {
  uint32_t ok = 1;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, abort_flag) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  return ok != 0;
}

// The wait of a loop that a whole converged warp runs.  Every lane polls for itself and sees the
// barrier with its own acquire; the vote gives all of them one verdict.  (A lane's own verdict mixes
// the barrier, the abort flag and the timer, so when a wait gives up the lanes need not agree, and a
// loop that some of them leave strands the others at its next warp-wide instruction.)
__device__ __forceinline__ bool mbar_wait_all(uint64_t *bar, uint32_t parity,
                                              volatile uint32_t *abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// A ring's next barrier, looked at without waiting ahead of this turn's MMAs or loads, and the wait itself one
// turn later.  The round trip to the barrier then passes behind that work: a k-block of 128 x 128 x 64 took
// 304 cycles with the wait alone, 268 with the look ahead of it (257 of MMAs).
__device__ __forceinline__ uint32_t mbar_look(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ bool mbar_wait_looked(uint32_t looked, uint64_t *bar, uint32_t parity,
                                                 volatile uint32_t *abort_flag) {
  return __all_sync(0xffffffffu, looked != 0) || mbar_wait_all(bar, parity, abort_flag);
}

// ---------------- TMA (cp.async.bulk.tensor), plain tile copies only ----------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
// x = innermost coordinate (elements); x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void *smem_dst, const CUtensorMap *map, uint64_t *bar,
                                            int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x),
      "r"(y)
      : "memory");
}
// Three-dimensional tile: (x, y, z) = (innermost, middle, outermost) coordinates.
__device__ __forceinline__ void tma_load_3d(void *smem_dst, const CUtensorMap *map, uint64_t *bar,
                                            int32_t x, int32_t y, int32_t z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x),
      "r"(y), "r"(z)
      : "memory");
}
// 128-pixel x 64-channel patch tile of an NHWC tensor through an im2col map: (c, w, h, n) is the
// window origin of the first pixel (inside the map's pixel box), (off_w, off_h) the filter tap; the
// hardware walks the following pixels of the box, image after image, and fills what lies outside the
// image (the padding) with zeros.
__device__ __forceinline__ void tma_load_im2col_4d(void *smem_dst, const CUtensorMap *map, uint64_t *bar, int32_t c,
                                                   int32_t w, int32_t h, int32_t n, uint16_t off_w, uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h),
      "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, const void *smem_src,
                                             int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *smem_src,
                                             int32_t x, int32_t y, int32_t z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
// generic-proxy writes to shared memory -> visible to the async proxy (TMA store, MMA)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------- tcgen05 / TMEM ----------------
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; issued by ONE thread.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Two operand descriptors of 64-wide k-blocks: their low words move, the high ones are constant.
struct KblockDesc {
  uint32_t a_lo, a_hi, b_lo, b_hi;
};
__device__ __forceinline__ KblockDesc kblock_desc(uint64_t a, uint64_t b) {
  return {static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b), static_cast<uint32_t>(b >> 32)};
}
// NKB (one or four) k-blocks of 64, four MMAs each, called by a whole warp and issued by its elected lane;
// only the first MMA may start a new accumulation.  Along a k-block the operands advance by two units of
// 16 bytes (32 bytes of a swizzled row; B by B_STEP where it is laid out otherwise), from one k-block to the
// next by a_kb / b_kb units.
// A tile of few columns is bound by this warp's instructions, not by the tensor pipe: 32-bit address
// arithmetic and four k-blocks per election instead of 64-bit adds and an election each.
#define MDC_KBLOCK(CGS, A, B, P)                                             \
  "add.u32 x1, " A ", 2;\n"                                                  \
  "add.u32 y1, " B ", %9;\n"                                                 \
  "add.u32 x2, " A ", 4;\n"                                                  \
  "add.u32 y2, " B ", %10;\n"                                                \
  "add.u32 x3, " A ", 6;\n"                                                  \
  "add.u32 y3, " B ", %11;\n"                                                \
  "mov.b64 da, {" A ", %2};\n"                                               \
  "mov.b64 db, {" B ", %4};\n"                                               \
  "@e tcgen05.mma.cta_group::" CGS ".kind::f16 [%0], da, db, %5, " P ";\n"   \
  "mov.b64 da, {x1, %2};\n"                                                  \
  "mov.b64 db, {y1, %4};\n"                                                  \
  "@e tcgen05.mma.cta_group::" CGS ".kind::f16 [%0], da, db, %5, 1;\n"       \
  "mov.b64 da, {x2, %2};\n"                                                  \
  "mov.b64 db, {y2, %4};\n"                                                  \
  "@e tcgen05.mma.cta_group::" CGS ".kind::f16 [%0], da, db, %5, 1;\n"       \
  "mov.b64 da, {x3, %2};\n"                                                  \
  "mov.b64 db, {y3, %4};\n"                                                  \
  "@e tcgen05.mma.cta_group::" CGS ".kind::f16 [%0], da, db, %5, 1;\n"
#define MDC_KBLOCKS_1(CGS)                                                   \
  "{\n"                                                                      \
  ".reg .pred p, e;\n"                                                       \
  ".reg .b32 x1, x2, x3, y1, y2, y3;\n"                                      \
  ".reg .b64 da, db;\n"                                                      \
  "elect.sync _|e, 0xffffffff;\n"                                            \
  "setp.ne.b32 p, %6, 0;\n" MDC_KBLOCK(CGS, "%1", "%3", "p") "}\n"
#define MDC_KBLOCKS_4(CGS)                                                   \
  "{\n"                                                                      \
  ".reg .pred p, e;\n"                                                       \
  ".reg .b32 x1, x2, x3, y1, y2, y3, ka1, ka2, ka3, kb1, kb2, kb3;\n"        \
  ".reg .b64 da, db;\n"                                                      \
  "elect.sync _|e, 0xffffffff;\n"                                            \
  "setp.ne.b32 p, %6, 0;\n"                                                  \
  "add.u32 ka1, %1, %7;\n"                                                   \
  "add.u32 kb1, %3, %8;\n"                                                   \
  "add.u32 ka2, ka1, %7;\n"                                                  \
  "add.u32 kb2, kb1, %8;\n"                                                  \
  "add.u32 ka3, ka2, %7;\n"                                                  \
  "add.u32 kb3, kb2, %8;\n" MDC_KBLOCK(CGS, "%1", "%3", "p")                 \
  MDC_KBLOCK(CGS, "ka1", "kb1", "1") MDC_KBLOCK(CGS, "ka2", "kb2", "1") MDC_KBLOCK(CGS, "ka3", "kb3", "1") "}\n"
template <int CG, int NKB, int B_STEP = 2>
__device__ __forceinline__ void umma_f16_ss_kblocks(uint32_t d_tmem, const KblockDesc &d, uint32_t idesc, uint32_t accumulate,
                                                    uint32_t a_kb = 0, uint32_t b_kb = 0) {
  static_assert((CG == 1 || CG == 2) && (NKB == 1 || NKB == 4), "");
#define MDC_KBLOCK_ARGS \
  "r"(d_tmem), "r"(d.a_lo), "r"(d.a_hi), "r"(d.b_lo), "r"(d.b_hi), "r"(idesc), "r"(accumulate), "r"(a_kb), "r"(b_kb), \
      "n"(B_STEP), "n"(2 * B_STEP), "n"(3 * B_STEP) : "memory"
  if constexpr (CG == 1 && NKB == 1) asm volatile(MDC_KBLOCKS_1("1")::MDC_KBLOCK_ARGS);
  else if constexpr (CG == 1) asm volatile(MDC_KBLOCKS_4("1")::MDC_KBLOCK_ARGS);
  else if constexpr (NKB == 1) asm volatile(MDC_KBLOCKS_1("2")::MDC_KBLOCK_ARGS);
  else asm volatile(MDC_KBLOCKS_4("2")::MDC_KBLOCK_ARGS);
#undef MDC_KBLOCK_ARGS
}
#undef MDC_KBLOCK
#undef MDC_KBLOCKS_1
#undef MDC_KBLOCKS_4
// One K = 16 step, called by a whole warp and issued by its elected lane.
__device__ __forceinline__ void umma_f16_ss_warp(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]; A was written to TMEM by tcgen05.st.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrives once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void umma_commit_warp(uint64_t *bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(smem_u32(bar))
      : "memory");
}
// Same wait, but naming the destination registers of the load it completes: the compiler
// must then keep every use of them after this point (the load fills them asynchronously).
__device__ __forceinline__ void tmem_ld_wait_regs(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                 "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                 "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait_regs(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                 "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i gets lane (base+i), columns c..c+31.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}

// ---------------- CTA pairs (cluster of 2, tcgen05 cta_group::2) ----------------
// The two CTAs of a pair cooperate on one MMA of M = 256: each stages its own 128 rows of
// A and its half of the B rows; the leader (cluster rank 0) issues the MMA for both.  All
// transfers stay plain per-CTA TMA loads (nothing is multicast); only mbarrier signals
// cross between the two CTAs, through shared::cluster addresses obtained with mapa.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  // the non-.aligned forms: threads of a warp may reach this point separately
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// shared::cta address of this CTA -> shared::cluster address of the same offset in CTA `rank`
__device__ __forceinline__ uint32_t mapa_u32(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
// TMA tile load whose completion is signalled on a barrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_cg2(void *smem_dst, const CUtensorMap *map,
                                                uint32_t bar_cluster_addr, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x),
      "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_cg2(void *smem_dst, const CUtensorMap *map,
                                                uint32_t bar_cluster_addr, int32_t x, int32_t y, int32_t z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x),
      "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_cg2(uint32_t *smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_cg2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_cg2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// arrives on the barrier at this shared-memory offset in every CTA of `cta_mask` once the pair's
// MMAs issued so far have completed; called by a whole warp
__device__ __forceinline__ void umma_commit_cg2_warp(uint64_t *bar, uint16_t cta_mask) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
      "}\n" ::"r"(smem_u32(bar)), "h"(cta_mask)
      : "memory");
}

// ---------------- descriptors ----------------
// Shared-memory matrix descriptor for a 128-byte-swizzled operand tile whose rows are
// 128 bytes (64 16-bit elements) and whose 8-row groups are 1024 bytes apart.
//   bits  0-13 start address >> 4        bits 16-29 leading byte offset >> 4
//   bits 32-45 stride byte offset >> 4   bits 46-47 descriptor version (1 on sm_100)
//   bits 61-63 swizzle mode (2 = 128 B)
// K-major operand ([rows][64 k-elements]): SBO = 1024 (next 8 rows), LBO unused (1).
// MN-major operand ([k][64 mn-elements]):  SBO = 1024 (next 8 k), LBO = byte distance
// between 64-element column blocks along MN.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes,
                                                         uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3ffff) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// Instruction descriptor for tcgen05.mma kind::f16 with fp32 accumulation.
//   bits 4-5 D format (1 = f32); 7-9 A format, 10-12 B format (0 = f16, 1 = bf16);
//   bit 15 A is MN-major; bit 16 B is MN-major; bits 17-22 N>>3; bits 24-28 M>>4.
__host__ __device__ constexpr uint32_t make_idesc_f16(uint32_t m, uint32_t n, bool bf16,
                                                      bool a_mn_major, bool b_mn_major) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) |
         ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) | ((n >> 3) << 17) |
         ((m >> 4) << 24);
}

// Two fp32 lanes per instruction (fma.rn.f32x2 and friends, sm_100): kernels whose
// arithmetic is bound by instruction issue halve their FMA / MUL / ADD count with these.
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_get(F2 x, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}


}  // namespace ptx
}  // namespace mdc
