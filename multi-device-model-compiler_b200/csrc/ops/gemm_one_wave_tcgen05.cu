// Tensor-core Gemm for problems that fit the chip in one wave: the same operation as
// gemm_tcgen05.cu (out = act(A . W^T + bias) + residual, 16-bit operands, fp32 accumulation in
// tensor memory), one output tile per CTA (or CTA pair).
//
// What bounds these shapes is latency, not the tensor pipe: a Gemm of a few hundred rows has too
// few 256 x 256 tiles to use the chip, and every CTA works through its whole K range alone, at
// 0.2 us per 64-wide k-block whatever the tile (MMA issue and barrier waits).  So
//   * the tile is chosen small enough that about every SM has one (choose_gemm_tile), down to
//     16 output columns;
//   * K is never cut: an element is one sum over K in order, as in gemm_tcgen05.cu, whatever the
//     tile.  The tile follows from M, so anything else would let a row's bits depend on the batch
//     that it is in (a sequence run alone, in a host chunk or on another GPU gives the same bits);
//   * a ring stage holds `depth` k-blocks, handed over by one barrier (and fetched by one TMA
//     instruction per operand where K is a multiple of 64), and the ring is as deep as shared memory
//     allows: a short K range is in flight as a whole and costs one memory latency;
//   * A's box is as high as M needs; accumulator rows beyond it hold stale operands and are not
//     stored.  Up to 64 rows the MMA has M = 64: 25 cycles for up to 32 columns instead of 40, which a long K is bound by
//     (99 x 768 x 3072 8.9 -> 6.9 us in a chain of launches, 512 x 768 x 3072 10.6 -> 8.4);
//   * the first piece of the bias and the residual is fetched while the mainloop runs;
//   * W's first stages are requested before the dependency on the previous kernel is resolved
//     when the caller knows the weights to be complete;
//   * results go straight from registers to global memory, 32 bytes per access.  Rows that are not
//     aligned to that, and a K that is no multiple of 64, are left to a variant of their own (kWide =
//     false): as run-time branches they took 2 to 3 % of a 12-layer pass over 99 tokens.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "gemm_common.cuh"
#include "gemm_plan.h"
#include "ops_common.h"

namespace mdc {

namespace onewave {
constexpr int BK = 64;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int MAX_STAGES = 16;
}  // namespace onewave

struct OneWaveParams {
  int M, N, num_kb;  // num_kb: 64-wide k-blocks
  const float *bias;
  const void *residual;
  void *out;
  RowAccess rows;
  int n_tiles;  // column tiles
  int bn, box_m, mma_m, depth, stages;
  int tmem_cols;
  int k_in_x;   // operand maps are (k, row) instead of (64 k, row, k-block)
  int w_ready;  // W may be read before the dependency wait
  uint32_t *err;
};

template <typename T16, typename TOut, int ACT, int CG, bool kWide>
__global__ void __launch_bounds__(onewave::THREADS, 1)
gemm_one_wave_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const OneWaveParams p) {
  using namespace onewave;
  using namespace ptx;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t abort_flag_s;
  volatile uint32_t *abort_flag = &abort_flag_s;

  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int half = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;  // which half of a pair's rows
  const bool leader = half == 0;
  const int tile = static_cast<int>(blockIdx.x) / CG;
  const int m_tile = tile / p.n_tiles, n_tile = tile - m_tile * p.n_tiles;
  const int row0 = (m_tile * CG + half) * p.box_m, col0 = n_tile * p.bn;
  const int depth = p.depth, stages = p.stages;
  const int a_kb_bytes = p.box_m * BK * 2, b_rows = p.bn / CG, b_kb_bytes = b_rows * BK * 2;
  const int a_bytes = a_kb_bytes * depth;
  const int stage_bytes = a_bytes + b_kb_bytes * depth;
  const int steps = (p.num_kb + depth - 1) / depth;

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_cg2(&tmem_slot, static_cast<uint32_t>(p.tmem_cols));
      tmem_relinquish_cg2();
    } else {
      tmem_alloc(&tmem_slot, static_cast<uint32_t>(p.tmem_cols));
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync_all();  // the peer's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_launch_dependents();  // after this CTA holds its tensor memory (see gemm_tcgen05.cu)

  // a stage is always filled whole: k-blocks past the last one read as zeros and are not used
  auto fetch = [&](uint8_t *dst, const CUtensorMap *map, int s, int row, int kb, int kb_bytes) __attribute__((always_inline)) {
    auto box = [&](uint8_t *to, int x, int z) __attribute__((always_inline)) {
      if constexpr (CG == 2) tma_load_3d_cg2(to, map, mapa_u32(smem_u32(&full_bar[s]), 0), x, row, z);
      else tma_load_3d(to, map, &full_bar[s], x, row, z);
    };
    if constexpr (!kWide) {
      if (p.k_in_x) {  // see encode_operand
        for (int d = 0; d < depth; ++d) box(dst + d * kb_bytes, (kb + d) * BK, 0);
        return;
      }
    }
    box(dst, 0, kb);
  };
  auto load_w = [&](int s, int kb) __attribute__((always_inline)) {
    fetch(tiles + s * stage_bytes + a_bytes, &tmap_b, s, col0 + half * b_rows, kb, b_kb_bytes);
  };
  auto load_a = [&](int s, int kb) __attribute__((always_inline)) {
    fetch(tiles + s * stage_bytes, &tmap_a, s, row0, kb, a_kb_bytes);
  };
  auto expect = [&](int s) __attribute__((always_inline)) {
    if (leader) mbar_arrive_expect_tx(&full_bar[s], static_cast<uint32_t>(CG * stage_bytes));
  };

  int early = 0;  // stages whose W is already on its way
  if (warp == 0 && p.w_ready) {
    early = min(stages, steps);
    if (elect_one()) {
      for (int i = 0; i < early; ++i) {
        expect(i);
        load_w(i, i * depth);
      }
    }
    __syncwarp();
  }
  pdl_wait();  // everything above overlaps the previous kernel's tail; activations are read below

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    int stage = 0;
    uint32_t phase = 0, looked = 0;
    for (int i = 0; i < steps; ++i) {
      if (i >= early && !mbar_wait_looked(looked, &empty_bar[stage], phase ^ 1, abort_flag)) {
        atomicCAS(p.err, 0u, 0x81000000u | static_cast<uint32_t>(stage));
        break;
      }
      const int next = stage + 1 == stages ? 0 : stage + 1;
      looked = mbar_look(&empty_bar[next], next ? phase ^ 1 : phase);
      if (elect_one()) {
        if (i >= early) {
          expect(stage);
          load_w(stage, i * depth);
        }
        load_a(stage, i * depth);
      }
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader of the pair) ------------------------------
    if (leader) {
      const uint32_t idesc = make_idesc_f16(static_cast<uint32_t>(p.mma_m * CG), static_cast<uint32_t>(p.bn), std::is_same<T16, __nv_bfloat16>::value,
                                            false, false);
      const KblockDesc desc0 = kblock_desc(make_smem_desc_sw128(smem_u32(tiles), 16, 1024),
                                           make_smem_desc_sw128(smem_u32(tiles) + static_cast<uint32_t>(a_bytes), 16, 1024));
      const uint32_t a_kb16 = static_cast<uint32_t>(a_kb_bytes) >> 4, b_kb16 = static_cast<uint32_t>(b_kb_bytes) >> 4;
      int stage = 0;
      uint32_t phase = 0, looked = 0;
      bool ok = true;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait_looked(looked, &full_bar[stage], phase, abort_flag)) {
          atomicCAS(p.err, 0u, 0x82000000u | static_cast<uint32_t>(stage));
          ok = false;
          break;
        }
        tc_fence_after();
        const int next = stage + 1 == stages ? 0 : stage + 1;
        looked = mbar_look(&full_bar[next], next ? phase : phase ^ 1);
        KblockDesc kd = desc0;
        kd.a_lo += static_cast<uint32_t>(stage * stage_bytes) >> 4;
        kd.b_lo += static_cast<uint32_t>(stage * stage_bytes) >> 4;
        const int n = min(depth, p.num_kb - i * depth);
        if (n == 4) {
          umma_f16_ss_kblocks<CG, 4>(tmem_base, kd, idesc, i != 0 ? 1u : 0u, a_kb16, b_kb16);
        } else {
          for (int d = 0; d < n; ++d) {
            umma_f16_ss_kblocks<CG, 1>(tmem_base, kd, idesc, (i | d) != 0 ? 1u : 0u);
            kd.a_lo += a_kb16, kd.b_lo += b_kb16;
          }
        }
        if constexpr (CG == 2) umma_commit_cg2_warp(&empty_bar[stage], 3);
        else umma_commit_warp(&empty_bar[stage]);
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
      if (ok) {
        if constexpr (CG == 2) umma_commit_cg2_warp(&acc_bar, 3);
        else umma_commit_warp(&acc_bar);
      }
    }
  }
  __syncwarp();

  // ------------------------------ epilogue ------------------------------
  const int ew = warp - 2;
  const int quarter = warp & 3;        // tensor-memory lanes this warp may access
  const int half_sel = ew >> 2;        // which half of the columns
  // columns in pieces of 16 (32 bytes of a 16-bit row, so that vector accesses stay aligned): the first
  // half of the warps takes the first half of the pieces, rounded up
  const int c_mid = (p.bn / 16 + 1) / 2 * 16;
  const int c_begin = half_sel ? c_mid : 0, c_end = half_sel ? p.bn : c_mid;
  // an accumulator of 128 rows has 32 in each quarter of the lanes, one of 64 rows 16
  const int q_rows = p.mma_m / 4;
  const int rows_in_tile = quarter * q_rows + lane;
  if (warp >= 2 && quarter * q_rows < p.box_m) {
    constexpr int NC = 16;
    TOut *out = static_cast<TOut *>(p.out);
    const T16 *res = static_cast<const T16 *>(p.residual);
    const int row = row0 + rows_in_tile;
    const bool row_ok = lane < q_rows && rows_in_tile < p.box_m && row < p.M;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float v[NC], rv[NC];  // bias, then the result; residual
    auto fetch = [&](int c) __attribute__((always_inline)) {
      const int gcol = col0 + c, cols = p.N - gcol;
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] = rv[j] = 0.f;
      if (p.bias) {
        if (kWide || p.rows.fast) {
#pragma unroll
          for (int j = 0; j < NC; j += 4) {
            if (j < cols) {
              const float4 q = __ldg(reinterpret_cast<const float4 *>(p.bias + gcol + j));
              v[j] = q.x, v[j + 1] = q.y, v[j + 2] = q.z, v[j + 3] = q.w;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < NC; ++j)
            if (j < cols) v[j] = __ldg(p.bias + gcol + j);
        }
      }
      if (res && row_ok) {
        const size_t off = static_cast<size_t>(row) * p.N + gcol;
        if constexpr (kWide) {
          if (cols > 0) {
            uint32_t rr[NC / 2];
            ld_global_32B(res + off, rr);
#pragma unroll
            for (int j = 0; j < NC; j += 8) unpack_res8<T16>(rr + j / 2, rv + j);
          }
        } else {
          load_row<T16, NC>(res + off, rv, cols, p.rows.vec);
        }
      }
    };
    // the first piece's bias and residual come while the mainloop runs
    if (c_begin < c_end) fetch(c_begin);
    bool ok = true;
    if (!mbar_wait_warp(&acc_bar, 0, abort_flag)) {
      if (lane == 0) atomicCAS(p.err, 0u, 0x83000000u);
      ok = false;
    }
    tc_fence_after();
#pragma unroll 1
    for (int c = c_begin; ok && c < c_end; c += NC) {
      const int gcol = col0 + c;
      if (gcol >= p.N) break;  // uniform across the warp
      uint32_t acc[NC];
      tmem_ld_32x16(t_lane + static_cast<uint32_t>(c), acc);
      if (c != c_begin) fetch(c);
      const size_t off = static_cast<size_t>(row) * p.N + gcol;
      const int cols = p.N - gcol;
      tmem_ld_wait_regs(acc);
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] += __uint_as_float(acc[j]);
      if (kWide || p.rows.fast) {
        act_fast_n<ACT, NC>(v);
      } else {
#pragma unroll
        for (int j = 0; j < NC; ++j) v[j] = act_apply_t<ACT>(v[j]);
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] += rv[j];
      if (row_ok) {
        if constexpr (kWide) store_out16<TOut>(out + off, v, cols > 8);
        else store_row<TOut, NC>(out + off, v, cols, p.rows.vec);
      }
    }
  }
  // ------------------------------ teardown ------------------------------
  if (*abort_flag) {
    // a wait gave up: give copies still in flight time to land before the CTA retires
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync_all();  // neither CTA of a pair frees tensor memory under the other
  tc_fence_after();
  if (warp == 1) {
    if constexpr (CG == 2) tmem_dealloc_cg2(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    else tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

template <typename T16, typename TOut, int ACT, int CG, bool kWide>
static void launch_one_wave_cg(const CUtensorMap &ta, const CUtensorMap &tb, const OneWaveParams &p, int grid, size_t smem,
                            cudaStream_t s) {
  auto kern = gemm_one_wave_kernel<T16, TOut, ACT, CG, kWide>;
  constexpr int kMaxDevices = 64;
  static bool attr_set_on[kMaxDevices] = {false};  // the attribute is per device
  const int dev = device_info().device;
  bool &attr_set = attr_set_on[(dev >= 0 && dev < kMaxDevices) ? dev : 0];
  if (!attr_set) {
    if (!check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneWaveMaxSmem),
                    "cudaFuncSetAttribute(gemm one-wave)"))
      return;
    attr_set = true;
  }
  {
    ProfileScope prof(kCatGemm, s);
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>(grid)), dim3(onewave::THREADS), smem, s, CG, ta, tb, p),
               "launch gemm one-wave");
  }
  launched("gemm_one_wave_kernel");
}

template <typename T16, typename TOut>
static void launch_one_wave_act(const CUtensorMap &ta, const CUtensorMap &tb, const OneWaveParams &p, int cg, int grid,
                                size_t smem, int act, cudaStream_t s) {
  const bool wide = p.rows.wide && !p.k_in_x;
#define MDC_ONE_WAVE(ACT_)                                                                      \
  do {                                                                                          \
    if (cg == 2 && wide) launch_one_wave_cg<T16, TOut, ACT_, 2, true>(ta, tb, p, grid, smem, s); \
    else if (cg == 2) launch_one_wave_cg<T16, TOut, ACT_, 2, false>(ta, tb, p, grid, smem, s);   \
    else if (wide) launch_one_wave_cg<T16, TOut, ACT_, 1, true>(ta, tb, p, grid, smem, s);       \
    else launch_one_wave_cg<T16, TOut, ACT_, 1, false>(ta, tb, p, grid, smem, s);                \
  } while (0)
  switch (act) {
  case MGPU_ACT_NONE: MDC_ONE_WAVE(kActNone); break;
  case MGPU_ACT_RELU: MDC_ONE_WAVE(kActRelu); break;
  case MGPU_ACT_GELU_ERF: MDC_ONE_WAVE(kActGeluErf); break;
  case MGPU_ACT_GELU_TANH: MDC_ONE_WAVE(kActGeluTanh); break;
  default: fail("mgpuMatmulEx16: unknown activation");
  }
#undef MDC_ONE_WAVE
}

// A [rows, Kp] row-major 16-bit matrix.  Kp a multiple of 64: as (64 k, row, k-block), so that one
// box holds several k-blocks.  Otherwise the last k-block would run into the next row, so the map is
// (k, row) and ends at Kp, one k-block per box and `depth` boxes per stage: the hand-over of a stage
// costs 0.2 us however it is filled (69 x 141 x 3720: 20.3 us with one k-block a stage, 11.6 with four).
static bool encode_operand(CUtensorMap *map, const void *base, int32_t dtype, int64_t rows, int64_t Kp, int box_rows,
                           int depth) {
  const bool blocked = Kp % onewave::BK == 0;
  const uint64_t gdim[3] = {static_cast<uint64_t>(blocked ? onewave::BK : Kp), static_cast<uint64_t>(rows),
                            static_cast<uint64_t>(blocked ? Kp / onewave::BK : 1)};
  const uint64_t gstr[2] = {static_cast<uint64_t>(Kp) * 2, onewave::BK * 2};
  const uint32_t box[3] = {onewave::BK, static_cast<uint32_t>(box_rows), static_cast<uint32_t>(blocked ? depth : 1)};
  return encode_tmap(map, dtype, 3, base, gdim, gstr, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

void gemm_one_wave_launch(const GemmTile &t, const void *a, const void *w_nk, const float *bias, const void *residual,
                       void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act,
                       bool w_ready, cudaStream_t s) {
  uint32_t *err = device_error_slot();
  if (!err) return;
  CUtensorMap ta, tb;
  if (!encode_operand(&ta, a, dtype, M, Kp, t.box_m, t.depth) || !encode_operand(&tb, w_nk, dtype, N, Kp, t.bn / t.cg, t.depth))
    return;
  OneWaveParams p;
  p.M = static_cast<int>(M), p.N = static_cast<int>(N);
  p.num_kb = static_cast<int>((Kp + onewave::BK - 1) / onewave::BK);
  p.k_in_x = Kp % onewave::BK != 0;
  p.bias = bias, p.residual = residual, p.out = out;
  p.rows = row_access(N, out, dtype_size(out_dtype), residual, bias);
  p.n_tiles = static_cast<int>((N + t.bn - 1) / t.bn);
  p.bn = t.bn, p.box_m = t.box_m, p.mma_m = t.mma_m, p.stages = t.stages;
  p.depth = t.depth;
  p.tmem_cols = 32;
  while (p.tmem_cols < t.bn) p.tmem_cols *= 2;
  p.w_ready = w_ready ? 1 : 0;
  p.err = err;
  const int64_t m_tiles = (M + static_cast<int64_t>(t.box_m) * t.cg - 1) / (static_cast<int64_t>(t.box_m) * t.cg);
  const int grid = static_cast<int>(m_tiles * p.n_tiles * t.cg);
  const size_t stage = static_cast<size_t>(p.depth) * (t.box_m + t.bn / t.cg) * onewave::BK * 2;
  // an MMA reads mma_m rows of A whatever the box holds: past the last box that must still be this
  // CTA's memory
  const size_t ring = stage * t.stages + (t.mma_m - t.box_m) * onewave::BK * 2;
  // never less than half of an SM's: two CTAs on one SM, of this launch or of the next, take turns at the SM's port while
  // others idle (2337 x 256 x 256 4.1 -> 3.5 us, 1592 x 704 x 256 4.7 -> 4.0, 99 x 768 x 768 3.44 -> 3.30; nothing loses 2 %)
  size_t smem = std::max<size_t>(ring + 1024, 117 * 1024);
  // An SM's shared memory is set up in steps, and what a CTA leaves of its step is for the blocks of the launch behind it: a ring
  // that fills one asks for the next.  With 2 KB left of 196 the conversion ahead of the next Gemm starts on idle SMs only:
  // mgpuMatmul of 608 x 448 x 1152 9.2 -> 8.1 us a call in a graph, 9.8 -> 8.3 direct, 4096 x 512 x 512 12.7 -> 12.0, 512 x 1000 x 2048 12.1 ->
  // 11.6; chains of Gemms alone do not mind.  Not beside a large weight, whose conversion needs the L1: 256 x 4096 x 1024
  // 11.8 -> 12.3, 372 x 3008 x 2752 1.07 of the time.
  if (N * Kp <= 1 << 21)
    for (const size_t step : {132, 164, 196})
      if (smem + 2048 <= step * 1024 && smem + 2048 + 12 * 1024 > step * 1024) smem = step * 1024;
  if (dtype == MGPU_DTYPE_F16) {
    if (out_dtype == MGPU_DTYPE_F16) launch_one_wave_act<__half, __half>(ta, tb, p, t.cg, grid, smem, act, s);
    else if (out_dtype == MGPU_DTYPE_F32) launch_one_wave_act<__half, float>(ta, tb, p, t.cg, grid, smem, act, s);
    else fail("mgpuMatmulEx16: output type must be the operand type or F32");
  } else {
    if (out_dtype == MGPU_DTYPE_BF16) launch_one_wave_act<__nv_bfloat16, __nv_bfloat16>(ta, tb, p, t.cg, grid, smem, act, s);
    else if (out_dtype == MGPU_DTYPE_F32) launch_one_wave_act<__nv_bfloat16, float>(ta, tb, p, t.cg, grid, smem, act, s);
    else fail("mgpuMatmulEx16: output type must be the operand type or F32");
  }
}

}  // namespace mdc
