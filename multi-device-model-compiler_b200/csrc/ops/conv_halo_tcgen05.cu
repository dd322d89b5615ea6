// Convolution as an implicit Gemm whose patches never exist: out[n, oc, oh, ow] = sum over taps and channels,
// fp16 operands, fp32 accumulation in tensor memory, fp32 NCHW in and out.
//
// A tile is 128 output pixels.  The input pixels that its windows cover (16 rows of 8 outputs under a 3 x 3 window: 18
// rows of 10) come into shared memory once per 64 channels, and the patch of a tap is that region with another start
// address in the operand's descriptor: no copy per tap, and between the taps nothing to wait for.  (The im2col kernel
// fetches each input element once per tap out of L2 and hands over a stage per tap.)
//   kCopy   conv_prepare_kernel has rewritten the input as NHWC fp16, with zeros between images; a region is one or a few
//           tiled TMA boxes, 128 bytes a pixel, swizzled by the address, which a shifted start keeps consistent.
//   else    up to 32 channels: twelve warps read the NCHW input and write regions by channel groups of eight,
//           [group][pixel][16 bytes], unswizzled: eight neighbouring pixels are a core matrix.  A unit is 32 pixels, dealt
//           in turn; the next sixteen channels' loads are in flight while these are converted.  With a stride of two, rows
//           and columns are kept in classes.
//           Up to eight channels make one group, and an MMA takes two taps of a filter row: the second half of its sixteen
//           k lies as far from the first as the next tap's pixel.  The last tap of an odd row is paired with zeros, not with
//           the pixel beyond the window: zero weights would turn an infinity there into NaN.  Below sixteen channels a sum
//           is made in parts (halo_chain).
//           The filter is packed by a launch ahead, which lets this one start after its own wait: input, bias and residual,
//           older than that launch, are read before the filter is complete.
//   warps 0-7   epilogue: accumulator -> bias, residual, ReLU -> NCHW, alternate tiles on up to four accumulators
//   warp 8      filter blocks of 64 k by TMA, kept for the CTA's life where they fit
//   warp 9      MMA issuer; where a tap's pixels start is read from the constant bank
//   warps 10-   input
//
// Bound: a copy's regions leave the MMAs (42 to 58 cycles each below 128 channels) or the stores, a warp's 32 pixels
// being four rows of a channel; straight from the input, the load / store unit: four lines to a load and to a store.
// conv_plan.h has the times and the line to the other kernels.  Offsets computed per tap, and elections per MMA, cost 300
// cycles a k-block: 16x32x113x91->32 7x7 134 us that way, 71 with a loop over rows and columns, 66 from the constant bank.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "conv_epilogue.cuh"
#include "conv_plan.h"
#include "fast_div.h"
#include "gemm_common.cuh"
#include "ops_common.h"
#include "ptx_sm100.cuh"

namespace mdc {

namespace convh {
constexpr int BM = 128, BK = 64;
constexpr int MAX_STAGES = kHaloFilterStages;
constexpr int EPI_WARPS = 8, IN_WARPS = kHaloInputWarps;
constexpr int threads(bool copy) { return (EPI_WARPS + 2 + (copy ? 1 : IN_WARPS)) * 32; }

struct Params : HaloTile {
  const float *x, *bias, *add;
  float *out;
  int N, IC, H, W, OC, KH, KW, OH, OW, PHL, PWL, SH, SW, DH, DW;
  Divisor by_ntiles, by_tiles_w, by_iw, by_hv, by_hvo;
  int alternate;              // epilogue: the two warps of a lane quarter take alternate tiles instead of alternate channels
  int taps;                   // entries of `tap`
  int n_tiles, num_tiles, relu;
  uint32_t tmem_cols;
  int accs;                   // accumulators in tensor memory, of `splits` sums each
  // A's descriptor in units of 16 bytes: leading offset, high word, from sixteen channels to the next
  uint32_t lead, a_hi, a_step;
  uint32_t *err;
  // What is added to the low word of A's descriptor for a tap (a pair of taps): where its pixels start, and with a tap
  // that has no partner the way to the zeros.  In the constant bank, so that the loop over taps has no arithmetic.
  uint32_t tap[kHaloMaxTaps];
  uint16_t sum[kHaloMaxTaps];  // few channels: columns to the MMA's sum, and in the top bit whether it adds to it
};
}  // namespace convh

// STEPS MMAs of sixteen channels each: A moves on by two planes (a_step units of 16 bytes), B by 32 bytes.
template <int STEPS>
__device__ __forceinline__ void umma_planes(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t a_step, uint32_t b_lo, uint32_t b_hi,
                                            uint32_t idesc, uint32_t accumulate) {
#define MDC_HEAD                                                             \
  "{\n"                                                                      \
  ".reg .pred p, e;\n"                                                       \
  ".reg .b32 x, y;\n"                                                        \
  ".reg .b64 da, db;\n"                                                      \
  "elect.sync _|e, 0xffffffff;\n"                                            \
  "setp.ne.b32 p, %7, 0;\n"                                                  \
  "mov.b64 da, {%1, %2};\n"                                                  \
  "mov.b64 db, {%4, %5};\n"                                                  \
  "add.u32 x, %1, %3;\n"                                                     \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %6, p;\n"
#define MDC_STEP(I)                                                          \
  "add.u32 y, %4, " I ";\n"                                                  \
  "mov.b64 da, {x, %2};\n"                                                   \
  "mov.b64 db, {y, %5};\n"                                                   \
  "add.u32 x, x, %3;\n"                                                      \
  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %6, 1;\n"
#define MDC_ARGS "r"(d), "r"(a_lo), "r"(a_hi), "r"(a_step), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory"
  if constexpr (STEPS == 1) asm volatile(MDC_HEAD "}\n" ::MDC_ARGS);
  else if constexpr (STEPS == 2) asm volatile(MDC_HEAD MDC_STEP("2") "}\n" ::MDC_ARGS);
  else if constexpr (STEPS == 3) asm volatile(MDC_HEAD MDC_STEP("2") MDC_STEP("4") "}\n" ::MDC_ARGS);
  else asm volatile(MDC_HEAD MDC_STEP("2") MDC_STEP("4") MDC_STEP("6") "}\n" ::MDC_ARGS);
#undef MDC_HEAD
#undef MDC_STEP
#undef MDC_ARGS
}

template <bool kCopy, bool kAdd>
__global__ void __launch_bounds__(convh::threads(kCopy), 1)
conv_halo_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const convh::Params p) {
  using namespace convh;
  using namespace ptx;
  constexpr int THREADS = threads(kCopy);
  extern __shared__ uint8_t smem_dyn[];
  __shared__ uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full_bar[4], acc_empty_bar[4], filter_bar;
  __shared__ uint64_t filter_full_bar[MAX_STAGES], filter_empty_bar[MAX_STAGES];
  __shared__ uint32_t tmem_slot, abort_flag_s;
  volatile uint32_t *abort_flag = &abort_flag_s;
  // the filter's blocks, and the regions of a copy, are 128-byte swizzled: 1024-byte aligned
  uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t *regions = base, *filter_s = base + p.regions_bytes;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int b_bytes = p.bn * BK * 2;
  float *bias_s = reinterpret_cast<float *>(filter_s + (p.resident ? p.num_kb : p.filter_stages * p.filter_kbs) * b_bytes);

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    if (kCopy) tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full_bar[i], kCopy ? 1u : static_cast<uint32_t>(p.qb));
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < p.filter_stages; ++i) {
      mbar_init(&filter_full_bar[i], 1);
      mbar_init(&filter_empty_bar[i], 1);
    }
    for (int a = 0; a < p.accs; ++a) {
      mbar_init(&acc_full_bar[a], 1);
      mbar_init(&acc_empty_bar[a], p.alternate ? EPI_WARPS / 2 : EPI_WARPS);
    }
    mbar_init(&filter_bar, 1);
    mbar_init_fence();
  }
  if (warp == EPI_WARPS + 1) {
    tmem_alloc(&tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  if (!kCopy && p.pairs) {
    // a region's second plane: zeros
    for (int s = 0; s < p.stages; ++s)
      for (int i = threadIdx.x; i < p.h.plane_px; i += THREADS)
        *reinterpret_cast<uint4 *>(regions + s * p.region_bytes + 16 * (p.h.plane_px + i)) = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_launch_dependents();  // after this CTA holds its tensor memory (see the Gemm kernel)
  if (kCopy) pdl_wait();

  if (warp < EPI_WARPS) {
    // ---- epilogue: thread = pixel, registers = channels; the two warps of a lane quarter take alternate groups of ----
    // ---- sixteen channels                                                                                        ----
    for (int i = threadIdx.x; i < (p.OC + 31) / 32 * 32; i += EPI_WARPS * 32)
      bias_s[i] = p.bias && i < p.OC ? __ldg(p.bias + i) : 0.f;
    asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
    constexpr int G = kCopy ? 32 : 16;
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const int r = quarter * 32 + lane;
    const int P = p.OH * p.OW;
    const int c_first = p.alternate ? 0 : half * G, c_step = p.alternate ? G : 2 * G;
    int acc = p.alternate ? half : 0;
    const int acc_step = p.alternate ? 2 : 1;
    const uint32_t acc_cols = p.tmem_cols / static_cast<uint32_t>(p.accs);
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x + (p.alternate ? half * gridDim.x : 0); tile < p.num_tiles; tile += (p.alternate ? 2 : 1) * gridDim.x) {
      const int mt = p.by_ntiles.div(tile), n0 = p.by_ntiles.mod(tile, mt) * p.bn;
      // the pixel's row, margins between images counted, and its column; pixels of a margin belong to no output
      int vr, ow;
      if (p.h.flat) {
        vr = p.by_iw.div(mt * BM + r), ow = p.by_iw.mod(mt * BM + r, vr);
      } else {
        const int tr = p.by_tiles_w.div(mt);
        vr = tr * 16 + (r >> 3), ow = p.by_tiles_w.mod(mt, tr) * 8 + (r & 7);
      }
      const int img = p.by_hvo.div(vr), oh = p.by_hvo.mod(vr, img);
      const bool live = img < p.N && oh < p.OH && ow < p.OW;
      const int64_t out_base = live ? (static_cast<int64_t>(img) * p.OC + n0) * P + oh * p.OW + ow : 0;
      const int nc = min(p.bn, p.OC - n0);  // live channels of the tile
      float extra[kAdd ? G : 1];
      auto fetch = [&](int c0) __attribute__((always_inline)) {
        if constexpr (kAdd) {
          if (live) conv_fetch(extra, p.add + out_base + static_cast<int64_t>(c0) * P, P, nc - c0);
        }
      };
      if constexpr (kAdd) {
#pragma unroll
        for (int j = 0; j < G; ++j) extra[j] = 0.f;
      }
      if (c_first < nc) fetch(c_first);  // in flight while the accumulator is waited for
      if (!mbar_wait_warp(&acc_full_bar[acc], acc_phase, abort_flag)) {
        atomicCAS(p.err, 0u, 0x62000000u);
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int c0 = c_first; c0 < nc; c0 += c_step) {
        uint32_t a[G];
        const uint32_t addr = tmem_base + acc * acc_cols + lane_base + static_cast<uint32_t>(c0);
        if constexpr (G == 32) tmem_ld_32x32(addr, a);
        else tmem_ld_32x16(addr, a);
        tmem_ld_wait_regs(a);
        if constexpr (!kCopy) {
          for (int i = 1; i < p.splits; ++i) {
            uint32_t more[16];
            tmem_ld_32x16(addr + static_cast<uint32_t>(i * p.bn), more);
            tmem_ld_wait_regs(more);
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = __float_as_uint(__uint_as_float(a[j]) + __uint_as_float(more[j]));
          }
        }
        conv_finish<G, kAdd>(a, bias_s + n0 + c0, extra, p.relu != 0);
        if (c0 + c_step < nc) fetch(c0 + c_step);
        if (live) conv_store(p.out + out_base + static_cast<int64_t>(c0) * P, a, P, nc - c0);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty_bar[acc]);
      if ((acc += acc_step) >= p.accs) acc -= p.accs, acc_phase ^= 1;
    }
  } else if (warp == EPI_WARPS) {
    // ---------------- filter ----------------
    if (!kCopy) pdl_wait();  // the launch that packs it; all that is older was complete when this kernel started
    if (p.resident) {
      if (elect_one()) {
        mbar_arrive_expect_tx(&filter_bar, static_cast<uint32_t>(p.num_kb * b_bytes));
        for (int kb = 0; kb < p.num_kb; ++kb) tma_load_2d(filter_s + kb * b_bytes, &tmap_w, &filter_bar, kb * BK, 0);
      }
      __syncwarp();
    } else {
      int stage = 0;
      uint32_t phase = 0, looked = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
        const int n0 = p.by_ntiles.mod(tile, p.by_ntiles.div(tile)) * p.bn;
        for (int kb = 0; kb < p.num_kb; kb += p.filter_kbs) {
          if (!mbar_wait_looked(looked, &filter_empty_bar[stage], phase ^ 1, abort_flag)) {
            atomicCAS(p.err, 0u, 0x67000000u | static_cast<uint32_t>(stage));
            ok = false;
            break;
          }
          const int next = stage + 1 == p.filter_stages ? 0 : stage + 1;
          looked = mbar_look(&filter_empty_bar[next], next ? phase ^ 1 : phase);
          if (elect_one()) {
            const int n = min(p.filter_kbs, p.num_kb - kb);
            mbar_arrive_expect_tx(&filter_full_bar[stage], static_cast<uint32_t>(n * b_bytes));
            for (int i = 0; i < n; ++i)
              tma_load_2d(filter_s + (stage * p.filter_kbs + i) * b_bytes, &tmap_w, &filter_full_bar[stage], (kb + i) * BK, n0);
          }
          if (++stage == p.filter_stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    // ---------------- MMA issuer (whole warp, elected lane issues) ----------------
    const uint32_t idesc = make_idesc_f16(BM, static_cast<uint32_t>(p.bn), false, false, false);
    const uint64_t f0 = make_smem_desc_sw128(smem_u32(filter_s), 16, 1024);
    const uint32_t f_lo = static_cast<uint32_t>(f0), f_hi = static_cast<uint32_t>(f0 >> 32);
    const uint32_t b_step = static_cast<uint32_t>(b_bytes / 16);
    const uint32_t a_lo0 = (smem_u32(regions) >> 4) | p.lead << 16, region_units = p.region_bytes / 16;
    const uint32_t acc_cols = p.tmem_cols / static_cast<uint32_t>(p.accs);
    int stage = 0, acc = 0, f_stage = 0;
    uint32_t phase = 0, acc_phase = 0, looked = 0, f_phase = 0, f_looked = 0;
    bool ok = true;
    if (p.resident && !mbar_wait_all(&filter_bar, 0, abort_flag)) {
      atomicCAS(p.err, 0u, 0x65000000u);
      ok = false;
    }
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
      if (!mbar_wait_all(&acc_empty_bar[acc], acc_phase ^ 1, abort_flag)) {
        atomicCAS(p.err, 0u, 0x64000000u);
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem_base + acc * acc_cols;
      uint32_t accumulate = 0, b_lo = f_lo;
      int left = 0, kbs_left = p.num_kb;  // k-blocks left in the filter's stage, and to come after it
      auto filter_ready = [&]() __attribute__((always_inline)) -> bool {  // ahead of a k-block
        if (left != 0) return true;
        if (!mbar_wait_looked(f_looked, &filter_full_bar[f_stage], f_phase, abort_flag)) {
          atomicCAS(p.err, 0u, 0x66000000u | static_cast<uint32_t>(f_stage));
          return false;
        }
        tc_fence_after();
        const int next = f_stage + 1 == p.filter_stages ? 0 : f_stage + 1;
        f_looked = mbar_look(&filter_full_bar[next], next ? f_phase : f_phase ^ 1);
        b_lo = f_lo + static_cast<uint32_t>(f_stage * p.filter_kbs) * b_step;
        left = min(p.filter_kbs, kbs_left);
        kbs_left -= left;
        return true;
      };
      auto filter_done = [&]() __attribute__((always_inline)) {  // after a k-block
        if (--left == 0) {
          umma_commit_warp(&filter_empty_bar[f_stage]);
          if (++f_stage == p.filter_stages) { f_stage = 0; f_phase ^= 1; }
        }
      };
      // The MMAs of one region.  STEPS: sixteens of channels of a tap; few channels: 0 pairs of taps, 5 single ones.
      auto taps = [&](auto steps, auto resident, uint32_t region) __attribute__((always_inline)) -> bool {
        constexpr int STEPS = decltype(steps)::value;
        constexpr bool RES = decltype(resident)::value;
        if constexpr (STEPS == 0) {
          // a k-block holds four pairs, rows of the filter one after the other
          auto one = [&](int t, uint32_t b) __attribute__((always_inline)) {
            umma_planes<1>(d + (p.sum[t] & 0x7fffu), region + p.tap[t], p.a_hi, 0, b, f_hi, idesc, static_cast<uint32_t>(p.sum[t] >> 15));
          };
          for (int t = 0; t < p.taps; t += 4) {
            if (!RES && !filter_ready()) return false;
            one(t, b_lo);
            if (t + 1 < p.taps) one(t + 1, b_lo + 2);
            if (t + 2 < p.taps) one(t + 2, b_lo + 4);
            if (t + 3 < p.taps) one(t + 3, b_lo + 6);
            b_lo += b_step;
            if (!RES) filter_done();
          }
        } else if constexpr (STEPS == 5) {
          for (int t = 0; t < p.taps; ++t) {
            if (!RES && !filter_ready()) return false;
            umma_planes<1>(d + (p.sum[t] & 0x7fffu), region + p.tap[t], p.a_hi, 0, b_lo, f_hi, idesc, static_cast<uint32_t>(p.sum[t] >> 15));
            b_lo += b_step;
            if (!RES) filter_done();
          }
        } else {
          for (int t = 0; t < p.taps; ++t) {
            if (!RES && !filter_ready()) return false;
            umma_planes<STEPS>(d, region + p.tap[t], p.a_hi, p.a_step, b_lo, f_hi, idesc, accumulate);
            accumulate = 1;
            b_lo += b_step;
            if (!RES) filter_done();
          }
        }
        return true;
      };
      auto of_steps = [&](auto resident, int steps, uint32_t region) __attribute__((always_inline)) -> bool {
        if (steps == 1) return taps(std::integral_constant<int, 1>{}, resident, region);
        if constexpr (kCopy) {
          if (steps == 2) return taps(std::integral_constant<int, 2>{}, resident, region);
          if (steps == 3) return taps(std::integral_constant<int, 3>{}, resident, region);
          return taps(std::integral_constant<int, 4>{}, resident, region);
        } else {
          if (steps == 0) return taps(std::integral_constant<int, 0>{}, resident, region);
          if (steps == 5) return taps(std::integral_constant<int, 5>{}, resident, region);
          return taps(std::integral_constant<int, 2>{}, resident, region);
        }
      };
      for (int cb = 0; cb < (kCopy ? p.ncb : 1); ++cb) {
        if (!mbar_wait_looked(looked, &full_bar[stage], phase, abort_flag)) {
          atomicCAS(p.err, 0u, 0x63000000u | static_cast<uint32_t>(stage));
          ok = false;
          break;
        }
        tc_fence_after();
        const int next = stage + 1 == p.stages ? 0 : stage + 1;
        looked = mbar_look(&full_bar[next], next ? phase : phase ^ 1);
        const uint32_t region = a_lo0 + static_cast<uint32_t>(stage) * region_units;
        const int steps = !kCopy && p.chain ? (p.pairs ? 0 : 5) : kCopy && cb + 1 < p.ncb ? 4 : p.last_steps;
        ok = p.resident ? of_steps(std::true_type{}, steps, region) : of_steps(std::false_type{}, steps, region);
        if (!ok) break;
        umma_commit_warp(&empty_bar[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      umma_commit_warp(&acc_full_bar[acc]);
      if (++acc == p.accs) acc = 0, acc_phase ^= 1;
    }
  } else if constexpr (kCopy) {
    // ---------------- input: regions of the copy ----------------
    int stage = 0;
    uint32_t phase = 0, looked = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
      const int mt = p.by_ntiles.div(tile);
      int x, y = 0;
      if (p.h.flat) {
        x = mt * BM - p.PHL * p.h.Wv - p.PWL;
      } else {
        const int tr = p.by_tiles_w.div(mt);
        x = p.by_tiles_w.mod(mt, tr) * 8 - p.PWL, y = tr * 16 - p.PHL;
      }
      for (int cb = 0; cb < p.ncb; ++cb) {
        if (!mbar_wait_looked(looked, &empty_bar[stage], phase ^ 1, abort_flag)) {
          atomicCAS(p.err, 0u, 0x61000000u | static_cast<uint32_t>(stage));
          ok = false;
          break;
        }
        const int next = stage + 1 == p.stages ? 0 : stage + 1;
        looked = mbar_look(&empty_bar[next], next ? phase ^ 1 : phase);
        if (elect_one()) {
          mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>(p.boxes * p.box_px * 128));
          for (int b = 0; b < p.boxes; ++b)
            tma_load_3d(regions + stage * p.region_bytes + b * p.box_px * 128, &tmap_x, &full_bar[stage], cb * BK, x + b * p.box_px, y);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else {
    // ---------------- input: NCHW fp32 -> regions ----------------
    const int HW = p.H * p.W;
    const uint64_t plane = static_cast<uint32_t>(HW);
    const int log_sh = p.SH - 1, log_sw = p.SW - 1;
    constexpr int kOutside = 1 << 30;  // mark of a pixel outside the image
    // Where this warp is: tile, piece of the region, sixteen of its channels; the region's place in the ring.
    struct Cursor {
      int tile, piece, step, stage;
      uint32_t phase;
    };
    auto settle = [&](Cursor &c) __attribute__((always_inline)) {  // pieces past the end are those of the next regions
      while (c.piece >= p.qb) {
        c.piece -= p.qb;
        c.tile += gridDim.x;
        if (++c.stage == p.stages) c.stage = 0, c.phase ^= 1;
      }
    };
    const char *src = nullptr;  // of the loads to come: this lane's pixel in the first of its channels
    int at = 0;                 // that pixel in a plane of the region, kOutside added for padding; negative for none
    auto map = [&](const Cursor &c) __attribute__((always_inline)) {
      const int q = c.piece * 32 + lane, mt = p.by_ntiles.div(c.tile);
      int row, col;
      bool in = q < p.h.px;
      at = in ? q : -1;
      if (p.h.flat) {
        const int px = mt * BM - p.PHL * p.h.Wv - p.PWL + q;
        in = in && px >= 0;
        row = in ? p.by_iw.div(px) : 0, col = in ? p.by_iw.mod(px, row) : 0;
      } else {
        const int tr = p.by_tiles_w.div(mt), tc = p.by_tiles_w.mod(mt, tr);
        const int rh = p.by_iw.div(q), rw = p.by_iw.mod(q, rh);
        row = tr * 16 * p.SH - p.PHL + rh, col = tc * 8 * p.SW - p.PWL + rw;
        if (in) at = ((rh & log_sh) * p.SW + (rw & log_sw)) * p.h.class_px + (rh >> log_sh) * p.h.pitch + (rw >> log_sw);
        in = in && row >= 0;
      }
      const int img = in ? p.by_hv.div(row) : 0, h = in ? p.by_hv.mod(row, img) : 0;
      in = in && img < p.N && h < p.H && static_cast<unsigned>(col) < static_cast<unsigned>(p.W);
      if (at >= 0 && !in) at |= kOutside;
      // pixels outside read an element that is there and drop it: no branch per load
      src = reinterpret_cast<const char *>(p.x + static_cast<int64_t>(in ? img : 0) * p.IC * HW + (in ? h * p.W + col : 0));
    };
    auto load = [&](const Cursor &c, float (&dst)[16]) __attribute__((always_inline)) {
      const int n = p.IC - c.step * 16;
      if (n >= 16) {
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[j] = __ldg(reinterpret_cast<const float *>(src + plane * (4u * j)));
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[j] = j < n ? __ldg(reinterpret_cast<const float *>(src + plane * (4u * j))) : 0.f;
      }
    };
    Cursor cur{static_cast<int>(blockIdx.x), warp - EPI_WARPS - 2, 0, 0, 0};
    settle(cur);
    float va[16], vb[16];
    int at_a = -1, at_b = -1;
    if (cur.tile < p.num_tiles) {
      map(cur);
      load(cur, va);
      at_a = at;
    }
    // One sixteen of channels of a piece: the next one's loads go out ahead of this one's use.  False at the end.  (Two
    // calls with their buffers exchanged: a copy between buffers would wait for the loads.)
    auto turn = [&](const float (&v)[16], int at_v, float (&ahead)[16], int &at_ahead) __attribute__((always_inline)) -> bool {
      if (cur.tile >= p.num_tiles) return false;
      Cursor nx = cur;
      const bool last = ++nx.step == p.last_steps;
      if (last) {
        nx.step = 0, nx.piece += IN_WARPS;
        settle(nx);
        if (nx.tile < p.num_tiles) map(nx);
      } else {
        src += plane * 64;
      }
      if (nx.tile < p.num_tiles) load(nx, ahead);
      at_ahead = at;
      if (cur.step == 0 && !mbar_wait_warp(&empty_bar[cur.stage], cur.phase ^ 1, abort_flag)) {
        if (lane == 0) atomicCAS(p.err, 0u, 0x60000000u | static_cast<uint32_t>(cur.stage));
        return false;
      }
      if (at_v >= 0) {
        const bool in = at_v < kOutside;
        uint8_t *dst = regions + static_cast<uint32_t>(cur.stage) * p.region_bytes +
                       (static_cast<uint32_t>(2 * cur.step * p.h.plane_px + (at_v & (kOutside - 1))) << 4);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i == 1 && p.pairs) break;  // one group of channels
          uint4 o = make_uint4(pack_pair<__half>(v[8 * i], v[8 * i + 1]), pack_pair<__half>(v[8 * i + 2], v[8 * i + 3]),
                               pack_pair<__half>(v[8 * i + 4], v[8 * i + 5]), pack_pair<__half>(v[8 * i + 6], v[8 * i + 7]));
          if (!in) o = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4 *>(dst + static_cast<uint32_t>(i * p.h.plane_px) * 16) = o;
        }
      }
      if (last) {
        fence_proxy_async_smem();  // the tensor core reads the region through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[cur.stage]);
      }
      cur = nx;
      return true;
    };
    while (turn(va, at_a, vb, at_b) && turn(vb, at_b, va, at_a)) {
    }
  }

  __syncwarp();
  if (*abort_flag) {
    // a wait gave up: give copies still in flight time to land before the CTA retires
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == EPI_WARPS + 1) tmem_dealloc(tmem_base, p.tmem_cols);
}

// The filter, OIHW fp32, as rows of fp16 in the order the MMAs take it, zeros where there is no weight:
//   [OC][tap][64], or with pairs of taps [OC][filter row][pair][2][8], rows padded to 64.
// A block of threads per output channel.
struct FilterPackParams {
  const float *w;
  __half *out;
  int IC, KH, KW, taps, pairs, row;  // row: elements per output channel
};
__global__ void __launch_bounds__(256) conv_filter_kernel(const FilterPackParams p) {
  pdl_wait();
  pdl_launch_dependents();  // after the wait: what is older is complete for the kernel that follows
  const int64_t oc = blockIdx.x;
  if (p.pairs) {
    const int per_row = (p.KW + 1) / 2;
    for (int i = threadIdx.x; i < p.row; i += 256) {
      const int ic = i & 7, pair = i >> 4, kh = pair / per_row, kw = (pair - kh * per_row) * 2 + (i >> 3 & 1);
      const bool in = kh < p.KH && kw < p.KW && ic < p.IC;
      p.out[oc * p.row + i] = __float2half_rn(in ? __ldg(p.w + ((oc * p.IC + ic) * p.KH + kh) * p.KW + kw) : 0.f);
    }
    return;
  }
  // the block's 64 x taps weights are contiguous in w: strided reads, served by L1 after the first touch
  const float *w = p.w + oc * p.IC * p.taps;
  __half *out = p.out + oc * p.row;
  for (int i = threadIdx.x; i < p.taps * 64; i += 256) {
    const int ic = i & 63, tap = i >> 6;
    out[i] = __float2half_rn(ic < p.IC ? __ldg(w + ic * p.taps + tap) : 0.f);
  }
}

namespace {
template <bool kCopy, bool kAdd>
void launch_halo(const CUtensorMap &tx, const CUtensorMap &tw, const convh::Params &p, int sms, cudaStream_t s) {
  auto kern = conv_halo_kernel<kCopy, kAdd>;
  static bool set_on[64] = {false};  // the attribute is per device
  const int dev = device_info().device;
  bool &set = set_on[(dev >= 0 && dev < 64) ? dev : 0];
  if (!set) {
    if (!check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kHaloMaxSmem)),
                    "cudaFuncSetAttribute(conv)"))
      return;
    set = true;
  }
  // the fewest CTAs that finish in the same number of rounds
  const int rounds = (p.num_tiles + sms - 1) / sms, grid = (p.num_tiles + rounds - 1) / rounds;
  {
    ProfileScope prof(kCatGemm, s);
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>(grid)), dim3(convh::threads(kCopy)), p.smem, s, 1, tx, tw, p),
               "launch conv_halo_kernel");
  }
  launched("conv_halo_kernel");
}

// What follows from a call's shape, kept for the next call of that shape (a plan, not a result; working it out takes
// longer than a launch).
struct HaloChoice {
  int64_t shape[17];
  int sms = 0;
  ConvForm form;  // kOther: for the other kernels
  bool sampled;
  ConvShape c;  // after conv_sampled; its pointers are the call's that made the entry and are not used
  convh::Params p;
};
const HaloChoice &halo_choice(const ConvShape &call, int sms) {
  static thread_local HaloChoice cache[64];
  const int64_t shape[17] = {call.N,  call.IC, call.H,   call.W,   call.OC, call.KH, call.KW, call.OH,          call.OW,
                             call.SH, call.SW, call.PHL, call.PWL, call.DH, call.DW, call.relu, call.add != nullptr};
  uint64_t key = 0;
  for (int64_t v : shape) key = (key ^ static_cast<uint64_t>(v)) * 0x9E3779B97F4A7C15ull;
  HaloChoice &e = cache[key >> 58];
  if (e.sms == sms && std::equal(shape, shape + 17, e.shape)) return e;
  std::copy(shape, shape + 17, e.shape);
  e.sms = sms, e.c = call, e.sampled = conv_sampled(e.c);
  e.form = conv_form(e.c, sms, conv_persistent_takes(call), &e.p);
  if (e.form == ConvForm::kOther) return e;
  const ConvShape &c = e.c;
  convh::Params &p = e.p;
  const bool copy = form_copies(e.form);
  p.N = int(c.N), p.IC = int(c.IC), p.H = int(c.H), p.W = int(c.W), p.OC = int(c.OC), p.KH = int(c.KH), p.KW = int(c.KW);
  p.OH = int(c.OH), p.OW = int(c.OW), p.PHL = int(c.PHL), p.PWL = int(c.PWL), p.SH = int(c.SH), p.SW = int(c.SW);
  p.DH = int(c.DH), p.DW = int(c.DW), p.relu = c.relu ? 1 : 0;
  p.n_tiles = int((c.OC + p.bn - 1) / p.bn), p.num_tiles = int(p.h.m_tiles * p.n_tiles);
  p.by_ntiles = Divisor(p.n_tiles), p.by_tiles_w = Divisor(p.h.tiles_w), p.by_iw = Divisor(p.h.IW);
  p.by_hv = Divisor(p.h.Hv), p.by_hvo = Divisor(p.h.HvO);
  p.alternate = p.num_tiles > sms ? 1 : 0;
  p.accs = p.splits * p.bn <= 128 ? 4 : 2;
  p.tmem_cols = 32;
  while (p.tmem_cols < static_cast<uint32_t>(p.accs * p.splits * p.bn)) p.tmem_cols *= 2;
  auto pixel = [&](int64_t rh, int64_t rw) {  // of the region, that a tap starts at
    return static_cast<uint32_t>(((rh % c.SH) * c.SW + rw % c.SW) * p.h.class_px + rh / c.SH * p.h.pitch + rw / c.SW);
  };
  const uint32_t group = p.h.flat ? 8u : static_cast<uint32_t>(p.h.pitch);  // pixels from eight of a tile to the next eight
  if (copy) {
    // 128-byte swizzled: a pixel is eight units, sixteen channels two
    p.lead = 1, p.a_hi = group * 8 | 1u << 14 | 2u << 29, p.a_step = 2;
  } else {
    p.lead = p.pairs ? pixel(0, c.DW) : static_cast<uint32_t>(p.h.plane_px);
    p.a_hi = group | 1u << 14, p.a_step = 2 * static_cast<uint32_t>(p.h.plane_px);
  }
  p.taps = 0;
  for (int64_t kh = 0; kh < c.KH; ++kh)
    for (int64_t kw = 0; kw < c.KW; kw += p.pairs ? 2 : 1)
      p.tap[p.taps++] = pixel(kh * c.DH, kw * c.DW) * (copy ? 8 : 1) +
                        (p.pairs && kw + 1 == c.KW ? (static_cast<uint32_t>(p.h.plane_px) - p.lead) << 16 : 0u);
  for (int t = 0; p.chain && t < p.taps; ++t)
    p.sum[t] = static_cast<uint16_t>(t / p.chain * p.bn | (t % p.chain ? 1 << 15 : 0));
  return e;
}
}  // namespace

bool conv_halo(const ConvShape &call, cudaStream_t s) {
  using namespace convh;
  const DeviceInfo &di = device_info();
  const HaloChoice &e = halo_choice(call, di.sms);
  if (e.form == ConvForm::kOther) return false;
  const bool copy = form_copies(e.form);
  // An output that overlaps the input: a launch that copies the input has read it before the first store.
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(call.x), o0 = reinterpret_cast<uintptr_t>(call.out);
  if (!copy && call.IC >= 16 && o0 < x0 + static_cast<uintptr_t>(call.N * call.IC * call.H * call.W) * 4 &&
      x0 < o0 + static_cast<uintptr_t>(call.N * call.OC * call.OH * call.OW) * 4)
    return false;
  const ConvShape &c = e.c;
  Params p = e.p;
  p.x = call.x, p.bias = call.bias, p.add = call.add, p.out = call.out;
  p.err = device_error_slot();
  if (!p.err) return true;

  const int64_t Kp = static_cast<int64_t>(p.num_kb) * BK;
  const int64_t copy_h = p.h.Hv, copy_w = p.h.flat ? p.h.Wv : c.W, Cp = (c.IC + 7) / 8 * 8;
  const uint64_t w_bytes = (static_cast<uint64_t>(c.OC) * Kp * 2 + 255) / 256 * 256;
  const uint64_t x_bytes = copy ? static_cast<uint64_t>(c.N) * copy_h * copy_w * Cp * 2 : 0;
  const int before = mgpuGetLastError();
  char *ws = static_cast<char *>(mgpuMemAllocAsync(w_bytes + x_bytes, s));
  if (!ws) {
    if (!x_bytes) return true;
    if (before == 0) mgpuClearLastError();  // an earlier failure's status stays; the caller's other kernels take over
    return false;
  }
  CUtensorMap tx = {}, tw;
  bool ok = encode_tmap_2d(&tw, ws, MGPU_DTYPE_F16, static_cast<uint64_t>(Kp), static_cast<uint64_t>(c.OC), static_cast<uint64_t>(Kp) * 2, BK,
                           static_cast<uint32_t>(p.bn), false);
  if (ok && copy) {
    const uint64_t px = static_cast<uint64_t>(Cp) * 2, rows = static_cast<uint64_t>(c.N * copy_h), width = static_cast<uint64_t>(copy_w);
    const uint64_t gdim[3] = {static_cast<uint64_t>(Cp), p.h.flat ? rows * width : width, p.h.flat ? 1 : rows};
    const uint64_t gstr[2] = {px, px * width};
    const uint32_t box[3] = {BK, static_cast<uint32_t>(p.h.flat ? p.box_px : p.h.IW), static_cast<uint32_t>(p.h.flat ? 1 : p.h.px / p.h.IW)};
    ok = encode_tmap(&tx, MGPU_DTYPE_F16, 3, ws + w_bytes, gdim, gstr, box, CU_TENSOR_MAP_SWIZZLE_128B, false) &&
         conv_prepare(c, call, e.sampled, copy_h, copy_w, ws + w_bytes, ws, s);
  } else if (ok) {
    const FilterPackParams f{call.w, reinterpret_cast<__half *>(ws), int(c.IC), int(c.KH), int(c.KW), int(c.KH * c.KW), p.pairs, int(Kp)};
    {
      ProfileScope prof(kCatElementwise, s);
      check_cuda(launch_chain(conv_filter_kernel, dim3(static_cast<unsigned>(c.OC)), dim3(256), 0, s, 1, f), "launch conv_filter_kernel");
    }
    launched("conv_filter_kernel");
  }
  if (ok) {
    auto launch = copy ? (p.add ? launch_halo<true, true> : launch_halo<true, false>)
                       : (p.add ? launch_halo<false, true> : launch_halo<false, false>);
    launch(tx, tw, p, di.sms, s);
  }
  mgpuMemFreeAsync(ws, s);
  return ok;
}

}  // namespace mdc
