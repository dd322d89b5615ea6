// Convolution as an implicit Gemm on persistent CTAs: out[n, oc, oh, ow] = sum_k patch[pixel, k] *
// filter[oc, k], fp16 operands, fp32 accumulation in tensor memory, fp32 NCHW at the boundary.
//
// One CTA per SM walks tiles of 128 output pixels x bn channels.  Loading patches, the MMAs and the
// epilogue belong to different warps and TMEM holds two accumulators, so the three run side by side,
// also across tiles; a CTA that does one tile and retires (conv_tcgen05.cu) has them one after the
// other and spends most of its life in memory round trips.
//
// Two sources of patches:
//   * kIm2col (16 or more input channels).  conv_prepare_kernel first rewrites the input as
//     NHWC fp16 (padded to 8 channels) and the filter as [OC][channel block][tap][64].  A k-block is one
//     tap of 64 channels, fetched by a single im2col TMA instruction: no thread touches a patch
//     element, and the padding comes from the hardware's zero fill.  The rewrite reads and writes
//     each input element once, the patch loads then read two bytes instead of four, from L2.
//   * kGather, kGatherFar (fewer channels, where an NHWC pixel is shorter than the 16 bytes TMA can
//     address).  Three groups of four warps build alternate k-blocks from the NCHW input, one
//     thread per pixel; where k lies in the window comes from the constant bank.
// The filter stays in shared memory for the CTA's life when it fits there.
//
// Bound: of short patches and many channels the stores, else instruction issue of the gather; of im2col k-blocks the hand-over of a stage and the issue of its MMAs, about
// 400 cycles a k-block where the MMAs of 64 columns take 193 (conv_plan.h says which calls conv_halo_kernel takes instead).
// Measured, whole call, one after another from the host, before (gather kernel of conv_tcgen05.cu, one tile per CTA) and after.
// Inputs changing from call to call:
//   16 x 3 x 256 x 256 -> 64, 3 x 3                      217 ->  56 us (43 of HBM time; 55 in a graph)
//   32 x 128 x 28 x 28 -> 128, 3 x 3                            19 us
// L2 flushed between calls:
//   18 x 128 x 43 x 51 -> 76, 5 x 5, stride 2            116 ->  34 us
// With warp roles by an index that the compiler knows to be uniform and the next barrier looked at ahead (ptx_sm100.cuh)
// the first shape went from 73 to 64 us, 32 x 256 x 14 x 14 -> 256 from 22.9 to 16.9, 32 x 512 x 7 x 7 -> 512 from 32 to 25.
// The gather was bound by instruction issue: run-time divisions and per-channel tests in the
// epilogue, 2.7 us a tile of 128 x 64; with multiplicative division, whole-group stores and the
// two epilogue halves on alternate tiles 1.3 us (150 -> 77 us for the first shape).  With the taps in the constant bank,
// one test a value at the edges, no work on other groups' tiles and a ring that is never shorter than the groups 64 -> 56,
// 32 x 3 x 224 x 224 -> 64 stride 2 48.5 -> 34.9, 43 x 6 x 255 x 256 -> 8 dilation 2 271 -> 134; in a graph 200 shapes of 1 to 15 channels,
// those that regions take among them, 0.79 of the time, none above 1.03.
#include <cuda_fp16.h>

#include "conv_epilogue.cuh"
#include "conv_plan.h"
#include "fast_div.h"
#include "gemm_common.cuh"
#include "ops_common.h"
#include "ptx_sm100.cuh"

namespace mdc {

namespace convp {
constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int MAX_STAGES = kRingMaxStages;
constexpr int EPI_WARPS = 8;
constexpr int GATHER_GROUPS = kGatherGroups, GATHER_WARPS = GATHER_GROUPS * 4;
constexpr size_t kMaxSmem = 224 * 1024;
// warps: 0-7 epilogue, 8 TMA, 9 MMA, then the gather warps
constexpr int threads(bool gather) { return (EPI_WARPS + 2 + (gather ? GATHER_WARPS : 0)) * 32; }

struct Params {
  const float *x, *bias, *add;
  float *out;
  int IC, H, W, OC, KW, OH, OW, PHL, PWL, SH, SW, DH, DW, taps;
  int M, P, K;          // output pixels, pixels per image, patch length (gather)
  Divisor by_p, by_ow, by_ntiles;
  int num_kb, last_k;   // k-blocks; live values of a gather tile's last block / of a partial channel block
  int ncb;              // 64-channel blocks (im2col)
  int bn, n_tiles, num_tiles, stages, resident, relu;
  uint32_t tmem_cols;
  uint32_t *err;
};
// Where the patches come from.  Where a gathered k lies is read from the constant bank: kGather for patches of up to
// kNearTaps values, windows of up to 16 x 15 taps and inputs that 32 bits address (conv_taps_near), kGatherFar for the others.
enum Source { kIm2col, kGather, kGatherFar };
template <int kSource>
struct Taps {};
template <>
struct Taps<kGather> : NearTaps {};
template <>
struct Taps<kGatherFar> : FarTaps {};
}  // namespace convp

// The value where `in`, else zero; never a branch.
__device__ __forceinline__ float ldg_if(bool in, const float *src) {
  float v;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "mov.f32 %0, 0f00000000;\n"
      "@p ld.global.nc.f32 %0, [%2];\n"
      "}\n"
      : "=f"(v)
      : "r"(static_cast<uint32_t>(in)), "l"(src));
  return v;
}

template <int kSource, bool kAdd>
__global__ void __launch_bounds__(convp::threads(kSource != convp::kIm2col), 1)
conv_persistent_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                       const convp::Params p, const __grid_constant__ convp::Taps<kSource> taps) {
  using namespace convp;
  constexpr bool gather = kSource != kIm2col;
  using namespace ptx;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full_bar[2], acc_empty_bar[2], filter_bar;
  __shared__ uint32_t tmem_slot, abort_flag_s;
  volatile uint32_t *abort_flag = &abort_flag_s;
  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int b_bytes = p.bn * BK * 2;
  const int stage_bytes = A_BYTES + (p.resident ? 0 : b_bytes);
  uint8_t *filter_s = tiles + p.stages * stage_bytes;
  float *bias_s = reinterpret_cast<float *>(filter_s + (p.resident ? p.num_kb * b_bytes : 0));

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    if (!gather) tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
    const uint32_t loaders = gather ? (p.resident ? 4u : 5u) : 1u;
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full_bar[i], loaders);
      mbar_init(&empty_bar[i], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full_bar[a], 1);
      mbar_init(&acc_empty_bar[a], gather ? EPI_WARPS / 2 : EPI_WARPS);
    }
    mbar_init(&filter_bar, 1);
    mbar_init_fence();
  }
  if (warp == EPI_WARPS + 1) {
    tmem_alloc(&tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_launch_dependents();  // after this CTA holds its tensor memory (see the Gemm kernel)
  pdl_wait();

  if (warp < EPI_WARPS) {
    // ---- epilogue: thread = pixel, registers = channels; a warp's 32 pixels are neighbours, so the ----
    // ---- store of a channel is one line.  The two warps of a lane quarter take alternate groups of ----
    // ---- channels, or alternate tiles where tiles are many and short (gather).                     ----
    for (int i = threadIdx.x; i < (p.OC + 31) / 32 * 32; i += EPI_WARPS * 32)
      bias_s[i] = p.bias && i < p.OC ? __ldg(p.bias + i) : 0.f;
    asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
    constexpr int G = gather ? 16 : 32;  // channels per group: as many as the registers allow
    const int quarter = warp & 3, half = warp >> 2;
    const int c_first = gather ? 0 : half * G, c_step = gather ? G : 2 * G;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    int acc = gather ? half : 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x + (gather ? half * gridDim.x : 0); tile < p.num_tiles; tile += (gather ? 2 : 1) * gridDim.x) {
      const int mt = p.by_ntiles.div(tile), n0 = p.by_ntiles.mod(tile, mt) * p.bn;
      const int m = mt * BM + quarter * 32 + lane;
      const bool live = m < p.M;
      const int img = live ? p.by_p.div(m) : 0, pix = live ? p.by_p.mod(m, img) : 0;
      const int64_t out_base = (static_cast<int64_t>(img) * p.OC + n0) * p.P + pix;
      const int nc = min(p.bn, p.OC - n0);  // live channels of the tile
      float extra[kAdd ? G : 1];
      auto fetch = [&](int c0) __attribute__((always_inline)) {
        if constexpr (kAdd) {
          if (live) conv_fetch(extra, p.add + out_base + static_cast<int64_t>(c0) * p.P, p.P, nc - c0);
        }
      };
      if constexpr (kAdd) {
#pragma unroll
        for (int j = 0; j < G; ++j) extra[j] = 0.f;
      }
      fetch(c_first);  // in flight while the accumulator is waited for
      if (!mbar_wait_warp(&acc_full_bar[acc], acc_phase, abort_flag)) {
        atomicCAS(p.err, 0u, 0x52000000u);
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int c0 = c_first; c0 < nc; c0 += c_step) {
        uint32_t a[G];
        const uint32_t addr = tmem_base + acc * (p.tmem_cols / 2) + lane_base + static_cast<uint32_t>(c0);
        if constexpr (G == 32) tmem_ld_32x32(addr, a);
        else tmem_ld_32x16(addr, a);
        tmem_ld_wait_regs(a);
        conv_finish<G, kAdd>(a, bias_s + n0 + c0, extra, p.relu != 0);
        if (c0 + c_step < nc) fetch(c0 + c_step);
        if (live) conv_store(p.out + out_base + static_cast<int64_t>(c0) * p.P, a, p.P, nc - c0);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty_bar[acc]);
      if (gather || (acc ^= 1) == 0) acc_phase ^= 1;
    }
  } else if (warp == EPI_WARPS) {
    // ---------------- TMA: filter blocks, and the patches when they are not gathered ----------------
    if (p.resident) {
      if (elect_one()) {
        mbar_arrive_expect_tx(&filter_bar, static_cast<uint32_t>(p.num_kb * b_bytes));
        for (int kb = 0; kb < p.num_kb; ++kb) tma_load_2d(filter_s + kb * b_bytes, &tmap_w, &filter_bar, kb * BK, 0);
      }
      __syncwarp();
    }
    if (!gather || !p.resident) {
      int stage = 0;
      uint32_t phase = 0, looked = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
        const int mt = tile / p.n_tiles, n0 = (tile - mt * p.n_tiles) * p.bn;
        const int m0 = mt * BM, img = m0 / p.P, pix = m0 - img * p.P, oh = pix / p.OW;
        const int h0 = oh * p.SH - p.PHL, w0 = (pix - oh * p.OW) * p.SW - p.PWL;
        int c0 = 0, kh = 0, kw = 0;  // k-blocks run over the taps of 64 channels, then the next 64
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!mbar_wait_looked(looked, &empty_bar[stage], phase ^ 1, abort_flag)) {
            atomicCAS(p.err, 0u, 0x51000000u | static_cast<uint32_t>(stage));
            ok = false;
            break;
          }
          const int next = stage + 1 == p.stages ? 0 : stage + 1;
          looked = mbar_look(&empty_bar[next], next ? phase ^ 1 : phase);
          if (elect_one()) {
            uint8_t *sa = tiles + stage * stage_bytes;
            mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>((gather ? 0 : A_BYTES) + (p.resident ? 0 : b_bytes)));
            if (!gather)
              tma_load_im2col_4d(sa, &tmap_x, &full_bar[stage], c0, w0, h0, img, static_cast<uint16_t>(kw * p.DW),
                                 static_cast<uint16_t>(kh * p.DH));
            if (!p.resident) tma_load_2d(sa + A_BYTES, &tmap_w, &full_bar[stage], kb * BK, n0);
          }
          if (++kw == p.KW) {
            kw = 0;
            if (++kh * p.KW == p.taps) kh = 0, c0 += BK;
          }
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    // ---------------- MMA issuer (whole warp, elected lane issues) ----------------
    const uint32_t idesc = make_idesc_f16(BM, static_cast<uint32_t>(p.bn), false, false, false);
    const uint64_t a0 = make_smem_desc_sw128(smem_u32(tiles), 16, 1024);
    const uint64_t f0 = make_smem_desc_sw128(smem_u32(filter_s), 16, 1024);
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0, looked = 0;
    bool ok = true;
    if (p.resident && !mbar_wait_all(&filter_bar, 0, abort_flag)) {
      atomicCAS(p.err, 0u, 0x55000000u);
      ok = false;
    }
    // the blocks that may be partial: the last one of a gathered patch, all taps of the last 64 channels
    const int partial_from = p.last_k == BK ? p.num_kb : p.num_kb - (gather ? 1 : p.taps);
    const int partial_steps = (p.last_k + 15) / 16;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
      if (!mbar_wait_all(&acc_empty_bar[acc], acc_phase ^ 1, abort_flag)) {
        atomicCAS(p.err, 0u, 0x54000000u);
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem_base + acc * (p.tmem_cols / 2);
      for (int kb = 0; kb < p.num_kb; ++kb) {
        if (!mbar_wait_looked(looked, &full_bar[stage], phase, abort_flag)) {
          atomicCAS(p.err, 0u, 0x53000000u | static_cast<uint32_t>(stage));
          ok = false;
          break;
        }
        tc_fence_after();
        const int next = stage + 1 == p.stages ? 0 : stage + 1;
        looked = mbar_look(&full_bar[next], next ? phase : phase ^ 1);
        const uint64_t ad = a0 + static_cast<uint64_t>(stage * (stage_bytes / 16));
        const uint64_t bd = p.resident ? f0 + static_cast<uint64_t>(kb * (b_bytes / 16)) : ad + A_BYTES / 16;
        if (kb < partial_from) {
          umma_f16_ss_kblocks<1, 1>(d, kblock_desc(ad, bd), idesc, kb != 0 ? 1u : 0u);
        } else {
          for (int k = 0; k < partial_steps; ++k)
            umma_f16_ss_warp(d, ad + static_cast<uint64_t>(2 * k), bd + static_cast<uint64_t>(2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
        }
        umma_commit_warp(&empty_bar[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      umma_commit_warp(&acc_full_bar[acc]);
      if ((acc ^= 1) == 0) acc_phase ^= 1;
    }
  } else if constexpr (gather) {
    // ---------------- gather: one thread per pixel, groups of four warps take alternate k-blocks ----------------
    // Where k lies is the same for all lanes: out of the constant bank a value costs its load and an addition of the uniform
    // datapath.  Out of a table in shared memory it took a load of that, a 64-bit addition and a test more (64 us at
    // 16x3x256x256->64 3x3, now 56); and every group worked out every tile's pixels, where a third of the tiles are its own.
    const int group = (warp - EPI_WARPS - 2) >> 2;
    const int row = ((warp - EPI_WARPS - 2) & 3) * 32 + lane;
    const uint32_t row_off = static_cast<uint32_t>(row) * 128u, swz = static_cast<uint32_t>(row & 7);
    const int KH = p.taps / p.KW, max_dh = (KH - 1) * p.DH, max_dw = (p.KW - 1) * p.DW;
    int block = group, tile_block = 0;  // this group's next k-block, and the tile's first, counted over all tiles of the CTA
    int stage = group;  // (no fewer stages than groups: conv_ring_stages)
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, tile_block += p.num_kb) {
      if (block >= tile_block + p.num_kb) continue;  // short patches: not every tile has one for every group
      const int m = p.by_ntiles.div(tile) * BM + row;
      const bool live = m < p.M;
      int h0 = 0, w0 = 0, img = 0;
      if (live) {
        img = p.by_p.div(m);
        const int pix = p.by_p.mod(m, img), oh = p.by_ow.div(pix);
        h0 = oh * p.SH - p.PHL;
        w0 = p.by_ow.mod(pix, oh) * p.SW - p.PWL;
      }
      // windows of the whole warp inside the image: no bounds tests
      const bool interior = __all_sync(0xffffffffu, live && h0 >= 0 && w0 >= 0 && h0 + max_dh < p.H && w0 + max_dw < p.W);
      // The window's origin, which may lie outside the image (then only live taps are read): bytes from the front of the
      // input, or its address.  And which rows and columns of the window lie outside.
      [[maybe_unused]] const char *front = nullptr;
      [[maybe_unused]] uint32_t at = 0, outside = 0x80000000u;
      [[maybe_unused]] const float *origin = p.x;
      if constexpr (kSource == kGather) {
        front = reinterpret_cast<const char *>(p.x) - taps.lead;
        at = taps.lead + static_cast<uint32_t>((img * p.IC * p.H + h0) * p.W + w0) * 4u;
        if (!interior) {
          for (int kh = 0; kh < KH; ++kh)
            if (!live || static_cast<unsigned>(h0 + kh * p.DH) >= static_cast<unsigned>(p.H)) outside |= 1u << kh;
          for (int kw = 0; kw < p.KW; ++kw)
            if (static_cast<unsigned>(w0 + kw * p.DW) >= static_cast<unsigned>(p.W)) outside |= 0x10000u << kw;
        }
      } else {
        origin += (static_cast<int64_t>(img) * p.IC * p.H + h0) * p.W + w0;
      }
      for (; block < tile_block + p.num_kb; block += GATHER_GROUPS) {
        const int kb = block - tile_block;
        const int pieces = kb == p.num_kb - 1 ? (p.last_k + 31) / 32 : 2;  // of 32 values
        uint8_t *sa = tiles + stage * stage_bytes + row_off;
        for (int h = 0; h < pieces; ++h) {
          float v[32];
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            const int k = kb * BK + h * 32 + c;
            if (interior && k + 8 <= p.K) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if constexpr (kSource == kGather) v[c + j] = __ldg(reinterpret_cast<const float *>(front + taps.off[k + j] + at));
                else v[c + j] = __ldg(origin + taps.off[k + j]);
              }
            } else if (k < p.K) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if constexpr (kSource == kGather) {
                  v[c + j] = ldg_if((outside & taps.need[k + j]) == 0, reinterpret_cast<const float *>(front + taps.off[k + j] + at));
                } else {
                  const uint32_t pos = taps.pos[k + j];
                  v[c + j] = ldg_if(live && k + j < p.K && static_cast<unsigned>(h0 + static_cast<int>(pos >> 16)) < static_cast<unsigned>(p.H) &&
                                        static_cast<unsigned>(w0 + static_cast<int>(pos & 0xffff)) < static_cast<unsigned>(p.W),
                                    origin + taps.off[k + j]);
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) v[c + j] = 0.f;
            }
          }
          // the loads are in flight; only now does the stage have to be free
          if (h == 0 && !mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
            atomicCAS(p.err, 0u, 0x50000000u | static_cast<uint32_t>(stage));
            ok = false;
            break;
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 q;
            q.x = pack_pair<__half>(v[c * 8 + 0], v[c * 8 + 1]);
            q.y = pack_pair<__half>(v[c * 8 + 2], v[c * 8 + 3]);
            q.z = pack_pair<__half>(v[c * 8 + 4], v[c * 8 + 5]);
            q.w = pack_pair<__half>(v[c * 8 + 6], v[c * 8 + 7]);
            // 128-byte swizzle: 16-byte chunk c of row r lives at chunk (c ^ (r & 7))
            *reinterpret_cast<uint4 *>(sa + ((static_cast<uint32_t>(h * 4 + c) ^ swz) << 4)) = q;
          }
        }
        if (!ok) break;
        fence_proxy_async_smem();  // the tensor core reads these rows through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[stage]);
        stage += GATHER_GROUPS;
        if (stage >= p.stages) stage -= p.stages, phase ^= 1;
      }
    }
  }

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

// Operands of the persistent kernels in one launch: blocks below `input_blocks` rewrite the input
// (NCHW fp32 -> NHWC fp16, channels zero-padded to Cp) in tiles of 64 pixels x 64 channels of one
// image, the others one (output channel, block of 64 input channels) of the filter each:
// OIHW fp32 -> [OC][channel block][tap][64] fp16, or for the gather kernel its own order padded to Kp.
// Bound by bytes: 6 per input element.  A lane reads 16 channels of its pixel, all in flight, a line per warp and
// channel, and writes one whole sector: nothing goes through shared memory (a 64 x 64 transposition there had
// twice the instructions).  32 x 64 x 56 x 56 in a whole call 34.1 -> 31.9 us; cold, 9 x 32 x 239 x 207 56.3 -> 46.0.
struct ConvPrepareParams {
  const float *x, *w;
  __half *x16, *w16;
  int IC, HW, Cp, pixel_tiles, channel_tiles, taps, ncb;
  int K, Kp;        // gather order (ncb == 0): patch length and row pitch
  int sampled, H, W, SH, SW, PHL, PWL;  // sampled: pixel (h, w) of the copy is (h*SH - PHL, w*SW - PWL) of the input
  Divisor by_w;
  int64_t input_blocks;
};
__global__ void __launch_bounds__(256) conv_prepare_kernel(const ConvPrepareParams p) {
  pdl_launch_dependents();
  pdl_wait();
  int64_t b = blockIdx.x;
  if (b < p.input_blocks) {
    const int ct = static_cast<int>(b % p.channel_tiles);
    b /= p.channel_tiles;
    const int pt = static_cast<int>(b % p.pixel_tiles);
    // warp: 32 pixels x 16 channels, a lane's channels one 32-byte sector of its pixel's row
    const int q = pt * 64 + (threadIdx.x >> 5 & 1) * 32 + (threadIdx.x & 31), c0 = ct * 64 + (threadIdx.x >> 6) * 16;
    if (q >= p.HW || c0 >= p.Cp) return;
    const int plane = p.sampled ? p.H * p.W : p.HW;
    int at = q;  // where the pixel lies in a plane
    bool in = true;
    if (p.sampled) {
      const int oh = p.by_w.div(q), h = oh * p.SH - p.PHL, w = p.by_w.mod(q, oh) * p.SW - p.PWL;
      in = static_cast<unsigned>(h) < static_cast<unsigned>(p.H) && static_cast<unsigned>(w) < static_cast<unsigned>(p.W);
      at = h * p.W + w;
    }
    const int n = min(16, p.IC - c0);  // live channels; what is left of Cp is zeros
    // pixels outside read an element that is there and drop it: no branch per load
    const char *src = reinterpret_cast<const char *>(p.x + (b / p.pixel_tiles * p.IC + c0) * static_cast<int64_t>(plane) + (in ? at : 0));
    float v[16];
    if (n == 16) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __ldcs(reinterpret_cast<const float *>(src + static_cast<uint64_t>(static_cast<uint32_t>(plane)) * (4u * j)));
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        v[j] = j < n ? __ldcs(reinterpret_cast<const float *>(src + static_cast<uint64_t>(static_cast<uint32_t>(plane)) * (4u * j))) : 0.f;
    }
    uint32_t o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
      o[e] = in ? *reinterpret_cast<const uint32_t *>(&h) : 0u;
    }
    __half *dst = p.x16 + (b / p.pixel_tiles * p.HW + q) * static_cast<int64_t>(p.Cp) + c0;
    if (p.Cp % 16 == 0) {
      st_global_32B(dst, o);
    } else {
      *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
      if (c0 + 8 < p.Cp) *reinterpret_cast<uint4 *>(dst + 8) = make_uint4(o[4], o[5], o[6], o[7]);
    }
    return;
  }
  b -= p.input_blocks;
  if (p.ncb == 0) {
    const float *w = p.w + b * p.K;
    __half *out = p.w16 + b * p.Kp;
    for (int i = threadIdx.x; i < p.Kp; i += 256) out[i] = __float2half_rn(i < p.K ? __ldg(w + i) : 0.f);
    return;
  }
  // the block's 64 x taps weights are contiguous in w: strided reads, served by L1 after the first touch
  const int cb = static_cast<int>(b % p.ncb);
  const int64_t oc = b / p.ncb;
  const float *w = p.w + (oc * p.IC + cb * 64) * static_cast<int64_t>(p.taps);
  __half *out = p.w16 + (oc * p.ncb + cb) * static_cast<int64_t>(p.taps) * 64;
  for (int i = threadIdx.x; i < p.taps * 64; i += 256) {
    const int ic = i & 63, tap = i >> 6;
    out[i] = __float2half_rn(cb * 64 + ic < p.IC ? __ldg(w + ic * p.taps + tap) : 0.f);
  }
}

namespace {
using EncodeIm2col = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const int *, const int *, cuuint32_t, cuuint32_t,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeIm2col encode_im2col() {
  static const EncodeIm2col fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<EncodeIm2col>(f);
  }();
  return fn;
}

template <bool kAdd, int kSource>
void launch_persistent(const CUtensorMap &tx, const CUtensorMap &tw, const convp::Params &p, const convp::Taps<kSource> &taps, size_t smem,
                       int sms, cudaStream_t s) {
  auto kern = conv_persistent_kernel<kSource, kAdd>;
  static bool set_on[64] = {false};  // the attribute is per device
  const int dev = device_info().device;
  bool &set = set_on[(dev >= 0 && dev < 64) ? dev : 0];
  if (!set) {
    if (!check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(convp::kMaxSmem)),
                    "cudaFuncSetAttribute(conv)"))
      return;
    set = true;
  }
  // the fewest CTAs that finish in the same number of rounds
  const int rounds = (p.num_tiles + sms - 1) / sms, grid = (p.num_tiles + rounds - 1) / rounds;
  {
    ProfileScope prof(kCatGemm, s);
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>(grid)), dim3(convp::threads(kSource != convp::kIm2col)), smem, s, 1, tx, tw, p, taps),
               "launch conv_persistent_kernel");
  }
  launched("conv_persistent_kernel");
}
}  // namespace

bool conv_persistent_takes(const ConvShape &call) { return conv_dense_describes(call) && (conv_gathers(call) || encode_im2col() != nullptr); }

bool conv_prepare(const ConvShape &c, const ConvShape &call, bool sampled, int64_t copy_h, int64_t copy_w, void *x16, void *w16,
                  cudaStream_t s) {
  const bool gather = conv_gathers(c);
  const int64_t taps = c.KH * c.KW, ncb = (c.IC + 63) / 64, K = c.IC * taps;
  ConvPrepareParams q;
  q.x = call.x, q.w = call.w, q.w16 = static_cast<__half *>(w16), q.x16 = static_cast<__half *>(x16);
  q.IC = int(c.IC), q.HW = int(copy_h * copy_w), q.Cp = int((c.IC + 7) / 8 * 8), q.taps = int(taps), q.ncb = gather ? 0 : int(ncb);
  q.K = int(K), q.Kp = int((K + 7) / 8 * 8);
  q.sampled = sampled || copy_h != c.H || copy_w != c.W ? 1 : 0;
  q.H = int(call.H), q.W = int(call.W);
  // a copy with margins is one of stride 1: pixel for pixel
  q.SH = sampled ? int(call.SH) : 1, q.SW = sampled ? int(call.SW) : 1;
  q.PHL = sampled ? int(call.PHL) : 0, q.PWL = sampled ? int(call.PWL) : 0;
  q.by_w = Divisor(copy_w);
  q.pixel_tiles = int((copy_h * copy_w + 63) / 64), q.channel_tiles = int(ncb);
  q.input_blocks = gather ? 0 : c.N * q.pixel_tiles * q.channel_tiles;
  const int64_t blocks = q.input_blocks + c.OC * (gather ? 1 : ncb);
  if (blocks > INT32_MAX) return false;
  {
    ProfileScope prof(kCatElementwise, s);
    check_cuda(launch_chain(conv_prepare_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, s, 1, q), "launch conv_prepare_kernel");
  }
  launched("conv_prepare_kernel");
  return true;
}

bool conv_persistent(const ConvShape &call, cudaStream_t s) {
  using namespace convp;
  if (!conv_persistent_takes(call)) return false;
  ConvShape c = call;
  const bool sampled = conv_sampled(c), gather = conv_gathers(c);
  const DeviceInfo &di = device_info();
  const int64_t window = c.KH * c.KW, K = c.IC * window, M = c.N * c.OH * c.OW;
  const int64_t Cp = (c.IC + 7) / 8 * 8, ncb = (c.IC + 63) / 64;
  const int64_t num_kb = gather ? (K + BK - 1) / BK : ncb * window;
  const int64_t Kp = gather ? (K + 7) / 8 * 8 : num_kb * BK;
  const int64_t m_tiles = (M + BM - 1) / BM;
  if (num_kb > (1 << 20)) return false;

  Params p;
  p.x = c.x, p.bias = c.bias, p.add = c.add, p.out = c.out;
  p.IC = int(c.IC), p.H = int(c.H), p.W = int(c.W), p.OC = int(c.OC), p.KW = int(c.KW), p.OH = int(c.OH), p.OW = int(c.OW);
  p.PHL = int(c.PHL), p.PWL = int(c.PWL), p.SH = int(c.SH), p.SW = int(c.SW), p.DH = int(c.DH), p.DW = int(c.DW);
  p.taps = int(window), p.M = int(M), p.P = int(c.OH * c.OW), p.K = int(K), p.num_kb = int(num_kb), p.ncb = int(ncb);
  p.last_k = int(gather ? K - (num_kb - 1) * BK : c.IC - (ncb - 1) * BK);
  p.relu = c.relu ? 1 : 0;
  p.bn = choose_conv_bn(m_tiles, c.OC, p.num_kb, gather, c.add != nullptr, di.sms);
  p.n_tiles = int((c.OC + p.bn - 1) / p.bn);
  if (m_tiles * p.n_tiles > INT32_MAX) return false;
  p.num_tiles = int(m_tiles * p.n_tiles);
  p.by_p = Divisor(p.P), p.by_ow = Divisor(p.OW), p.by_ntiles = Divisor(p.n_tiles);
  p.tmem_cols = 32;
  while (p.tmem_cols < 2u * p.bn) p.tmem_cols *= 2;
  const int64_t filter_bytes = num_kb * p.bn * BK * 2;
  p.resident = conv_filter_stays(num_kb, p.bn, p.n_tiles, p.num_tiles, di.sms);
  const int64_t stage_bytes = A_BYTES + (p.resident ? 0 : p.bn * BK * 2);
  const int64_t fixed = 1024 + (p.resident ? filter_bytes : 0) + (c.OC + 31) / 32 * 128;
  p.stages = conv_ring_stages(static_cast<int64_t>(kMaxSmem) - 4096 - fixed, stage_bytes, gather);
  if (p.stages == 0) return false;
  const size_t smem = static_cast<size_t>(fixed + p.stages * stage_bytes);
  p.err = device_error_slot();
  if (!p.err) return true;

  // one block for both operands; without memory for it the caller's other kernel takes over
  const uint64_t w_bytes = (static_cast<uint64_t>(c.OC) * Kp * 2 + 255) / 256 * 256;
  const uint64_t x_bytes = gather ? 0 : static_cast<uint64_t>(c.N) * c.H * c.W * Cp * 2;
  const int before = mgpuGetLastError();
  char *ws = static_cast<char *>(mgpuMemAllocAsync(w_bytes + x_bytes, s));
  if (!ws) {
    if (!x_bytes) return true;
    if (before == 0) mgpuClearLastError();  // an earlier failure's status stays
    return false;
  }
  CUtensorMap tx = {}, tw;
  bool ok = encode_tmap_2d(&tw, ws, MGPU_DTYPE_F16, static_cast<uint64_t>(Kp), static_cast<uint64_t>(c.OC),
                           static_cast<uint64_t>(Kp) * 2, BK, static_cast<uint32_t>(p.bn), false);
  if (ok && !gather) {
    const cuuint64_t gdim[4] = {cuuint64_t(Cp), cuuint64_t(c.W), cuuint64_t(c.H), cuuint64_t(c.N)};
    const cuuint64_t gstr[3] = {cuuint64_t(Cp) * 2, cuuint64_t(Cp) * 2 * c.W, cuuint64_t(Cp) * 2 * c.W * c.H};
    const int lower[2] = {-int(c.PWL), -int(c.PHL)}, upper[2] = {int(conv_upper_w(c)), int(conv_upper_h(c))};
    const cuuint32_t estr[4] = {1, cuuint32_t(c.SW), cuuint32_t(c.SH), 1};
    ok = encode_im2col()(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, ws + w_bytes, gdim, gstr, lower, upper, BK, BM, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  ok = ok && conv_prepare(c, call, sampled, c.H, c.W, ws + w_bytes, ws, s);
  if (ok) {
    auto launch = [&](const auto &t) { p.add ? launch_persistent<true>(tx, tw, p, t, smem, di.sms, s) : launch_persistent<false>(tx, tw, p, t, smem, di.sms, s); };
    if (!gather) {
      launch(Taps<kIm2col>());
    } else if (conv_taps_near(c)) {
      Taps<kGather> t;
      fill_taps(c, &t);
      launch(t);
    } else {
      Taps<kGatherFar> t;
      fill_taps(c, &t);
      launch(t);
    }
  }
  mgpuMemFreeAsync(ws, s);
  return ok;
}

}  // namespace mdc
