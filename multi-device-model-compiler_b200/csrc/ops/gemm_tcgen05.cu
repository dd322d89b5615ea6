// Tensor-core Gemm for sm_100a: out[M,N] = act(A[M,K] . W[N,K]^T + bias[N]) + residual[M,N]
// with 16-bit operands (fp16 or bf16), fp32 accumulation in tensor memory and a fused
// epilogue.  Replaces the cuBLASLt calls of lib/Kernels/GPU/Ops.cu:59-120 (mgpuMatmul) and
// :136-234 (mgpuMatmulEx: bias / ReLU / residual epilogues).
//
// Structure (one persistent CTA per SM, 10 warps):
//   warp 0   TMA producer: cp.async.bulk.tensor tiles of A (128 x 64) and W (256 x 64) into
//            a ring of 128-byte-swizzled shared memory, completion on mbarriers.
//   warp 1   MMA issuer: tcgen05.mma (M=128, N=256, K=16) reading the shared-memory tiles
//            through matrix descriptors; tcgen05.commit releases the stage to the producer
//            and, after the last k-block, hands the accumulator over.  Both loops are run by the
//            whole warp with the elected lane issuing (see ptx_sm100.cuh: the one-lane form was
//            bound by instruction issue, 590 cycles per k-block where the MMAs need 512).
//   warps 2-9 epilogue: tcgen05.ld the 128 x 256 fp32 accumulator out of TMEM (each warp
//            its 32-lane quarter, two warps per quarter splitting the columns), add bias,
//            apply the activation, add the residual, convert and store.  Two forms (kWide):
//            Rows that can be moved 32 bytes at a time: a thread owns a row, and two threads store
//            64 bytes of each other's (store_row_pairs), so nothing is staged.  The ring has two
//            more stages, and the residual and the bias are fetched before the accumulator is waited for.
//            A short K is bound by this epilogue: with sectors stored one by one and the residual piece by
//            piece it took 6940 cycles a tile, 10900 with residual, beside 6144 of MMAs at K = 768.  Graph
//            replays, operands in turn, against that form: 32768 x 2304 x 768 117 -> 108 us, 32768 x 768 x 768
//            with residual 59.7 -> 52.7, 12288 x 768 x 768 18.8 -> 16.2; at K up to 168 and rows off 64 bytes
//            the exchange costs up to 4 % (28588 x 80 x 144 7.55 / 7.80, but 40000 x 176 x 64 10.4 / 10.5, 20000 x
//            1000 x 128 36.4 / 35.5: no rule found).  (The bias a tile ahead and the pieces written out without
//            a residual too: 5145 x 536 x 64 6.53 -> 6.66, 20450 x 112 x 168 8.32 -> 8.70, 36322 x 384 x 64 17.2 ->
//            17.9, 32768 x 2304 x 768 108 -> 111.  Stores spread over the mainloop by the
//            clock: no gain.  16 epilogue warps: 8 us slower at 32768 x 3072 x 768 with GELU.)
//            Rows of other multiples of 16 bytes (N = 8 mod 16, or a pointer off its 32-byte
//            boundary): each warp stages 32 rows x 128 bytes in swizzled shared memory and moves
//            it with one TMA store, the residual arrives by a TMA load, and 96 KiB of the ring go
//            to that.  32768 x 1000 x 768: 51 us, with residual 66; with 16-byte accesses from
//            registers, half a sector each, 57 and 84; one element at a time 351 and 516.
//            Ragged rows, and a bias off its boundary, are stored from registers.
// TMEM holds two accumulators (2 x 256 columns) so the epilogue of tile i overlaps the
// mainloop of tile i+1.  Every CTA fetches its own tiles with plain TMA loads and relies on
// L2 for reuse.  All waits are bounded (see ptx_sm100.cuh).
//
// Two variants of the same kernel (template parameter CG):
//   CG = 1  one CTA per 128 x 256 tile (small problems).
//   CG = 2  CTA pairs (cluster of 2, tcgen05 cta_group::2) on 256 x 256 tiles: each CTA
//           stages its 128 rows of A and HALF of the W rows (32 KiB per k-block instead of
//           48), the leader CTA issues one M = 256 MMA for the pair, each CTA keeps its own
//           128 x 256 accumulator and runs its own epilogue.  Tensor-core operand reads and
//           TMA writes compete for shared-memory bandwidth; halving the W bytes per SM is
//           what lifts the mainloop.
// Measured, 12-layer step of 256 x 128 tokens (hidden 768): 7.38 ms with the one-lane loops and the
// staged epilogue on 4 stages; whole-warp loops and direct stores 7.15 (4 stages); bias out of L1
// 6.95 (4 stages), 6.89 (5), 6.88 (6); 7 stages leave L1 too small for the residual: 7.05.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "gemm_common.cuh"
#include "gemm_plan.h"
#include "ops_common.h"

namespace mdc {

namespace gemm {
constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int TMEM_COLS = 512;
constexpr int EPI_BUF_BYTES = 4096;  // staged rows: 32 x 128 bytes, per warp
template <int CG, bool kWide>
struct Cfg {
  static constexpr int B_ROWS = BN / CG;            // W rows this CTA stages per k-block
  static constexpr int B_BYTES = B_ROWS * BK * 2;   // 32 KiB (CG 1) / 16 KiB (CG 2)
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = kWide ? (CG == 2 ? 6 : 4) : (CG == 2 ? 4 : 3);
  // staged rows: output (two buffers for pairs, so that a chunk does not wait for the previous one's
  // TMA store to drain) and residual
  static constexpr int OUT_BUFS = CG == 2 ? 2 : 1;
  static constexpr int EPI_WARP_BYTES = kWide ? 0 : (OUT_BUFS + 1) * EPI_BUF_BYTES;
  static constexpr size_t SMEM_BYTES =
      static_cast<size_t>(STAGES) * STAGE_BYTES + EPI_WARPS * EPI_WARP_BYTES + 1024;  // + alignment slack
};
}  // namespace gemm

struct GemmParams {
  int M, N, K;  // K already padded to a multiple of 8
  const float *bias;
  const void *residual;
  void *out;
  RowAccess rows;
  int num_m_blocks, num_n_blocks;
  int cta_group;  // 1: one CTA per 128 x bn tile; 2: CTA pairs on 256 x bn tiles
  int bn;         // tile width in output columns: 256, 192 or 128 (accumulators stay 256 TMEM columns apart)
  int cw;         // staged rows: columns per chunk, 64 (16-bit output, 128-byte rows) or 32
  uint32_t *err;
};
// tensor maps of the staged rows
template <bool kWide>
struct RowMaps {
  CUtensorMap out, res;
};
template <>
struct RowMaps<true> {};

// Staged rows, or rows moved 32 bytes at a time; the latter without a residual are a kernel of their own.  Its registers (115 to
// 142 a thread; 160 to 168 with a residual) leave an SM room for the blocks of the launch behind it, which are then in place
// when this one ends: mgpuMatmul of 2590 x 1472 x 256, whose next call converts its operands, 13.2 -> 10.9 us in a graph and 14.3 ->
// 12.7 in direct calls, 2272 x 2496 x 320 16.3 -> 14.9, 3200 x 1024 x 384 13.6 -> 12.1; Gemms behind one another the same.
enum RowForm { kStagedRows, kWideRows, kWideResidual };

template <typename T16, typename TOut, int ACT, int CG, int FORM>
__global__ void __launch_bounds__(gemm::THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ RowMaps<FORM != kStagedRows> rows, const GemmParams p) {
  constexpr bool kWide = FORM != kStagedRows;
  using namespace gemm;
  using namespace ptx;
  using C = Cfg<CG, kWide>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full_bar[2], acc_empty_bar[2];
  // bias of the columns each epilogue warp handles: kept out of L1, of which the ring leaves little
  __shared__ __align__(16) float bias_s[kWide ? EPI_WARPS : 1][kWide ? BN / 2 : 4];
  __shared__ uint64_t res_bar[kWide ? 1 : EPI_WARPS];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t abort_flag_s;
  volatile uint32_t *abort_flag = &abort_flag_s;

  // 128-byte-swizzled tiles need 1024-byte aligned bases
  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // CG == 2: the two CTAs of a cluster work on one 256-row tile; rank 0 leads
  const int cta_rank = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const bool leader = cta_rank == 0;
  const int worker = static_cast<int>(blockIdx.x) / CG, num_workers = static_cast<int>(gridDim.x) / CG;
  // tiles are (CG * 128) rows x bn columns, numbered with the column block running fastest:
  // the workers that run side by side then share their rows of A (read from HBM once, found
  // in L2 by the other column blocks) while W, which is small, stays in L2 throughout
  const int num_m_units = (p.num_m_blocks + CG - 1) / CG;
  const int num_tiles = num_m_units * p.num_n_blocks;
  const int num_kb = (p.K + BK - 1) / BK;
  const int bn = p.bn;  // tile width; this CTA stages bn / CG rows of W per k-block
  const uint32_t stage_tx_bytes = static_cast<uint32_t>(A_BYTES + (bn / CG) * BK * 2);

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);   // the leader's arrive.expect_tx (covers both CTAs' bytes)
      mbar_init(&empty_bar[s], 1);  // one tcgen05.commit
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full_bar[a], 1);
      mbar_init(&acc_empty_bar[a], CG * EPI_WARPS * 32);  // epilogue threads of the whole pair
    }
    if constexpr (!kWide)
      for (int w = 0; w < EPI_WARPS; ++w) mbar_init(&res_bar[w], 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_cg2(&tmem_slot, TMEM_COLS);
      tmem_relinquish_cg2();
    } else {
      tmem_alloc(&tmem_slot, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync_all();  // the peer's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  // Only now, with this CTA's tensor memory allocated, may the next kernel of the chain be set
  // up: a dependent CTA that shared the SM and took tensor-memory columns first would wait for
  // this grid while this CTA waited for its columns.
  pdl_launch_dependents();
  pdl_wait();  // everything above overlaps the previous kernel's tail; operands are read below

  if (warp == 0) {
    // ------------------------------ TMA producer (whole warp, elected lane issues) ------------------------------
    int stage = 0;
    uint32_t phase = 0, looked = 0;
    bool ok = true;
    for (int tile = worker; ok && tile < num_tiles; tile += num_workers) {
      const int m_blk = (tile / p.num_n_blocks) * CG + cta_rank, n_blk = tile % p.num_n_blocks;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_looked(looked, &empty_bar[stage], phase ^ 1, abort_flag)) {
          atomicCAS(p.err, 0u, 0x10000000u | static_cast<uint32_t>(stage));
          ok = false;
          break;
        }
        const int next = stage + 1 == STAGES ? 0 : stage + 1;
        looked = mbar_look(&empty_bar[next], next ? phase ^ 1 : phase);
        if (elect_one()) {
          uint8_t *sa = tiles + stage * STAGE_BYTES;
          uint8_t *sb = sa + A_BYTES;
          if constexpr (CG == 2) {
            // both CTAs' copies complete on the LEADER's barrier, which expects the bytes of both
            const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), 0);
            if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * stage_tx_bytes);
            tma_load_2d_cg2(sa, &tmap_a, bar, kb * BK, m_blk * BM);
            tma_load_2d_cg2(sb, &tmap_b, bar, kb * BK, n_blk * bn + cta_rank * (bn / 2));
          } else {
            mbar_arrive_expect_tx(&full_bar[stage], stage_tx_bytes);
            tma_load_2d(sa, &tmap_a, &full_bar[stage], kb * BK, m_blk * BM);
            tma_load_2d(sb, &tmap_b, &full_bar[stage], kb * BK, n_blk * bn);
          }
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only; whole warp, elected lane issues) ----------------
    if (leader) {
      const uint32_t idesc = make_idesc_f16(BM * CG, static_cast<uint32_t>(bn),
                                            std::is_same<T16, __nv_bfloat16>::value, false, false);
      const uint64_t desc0 = make_smem_desc_sw128(smem_u32(tiles), 16, 1024);
      int stage = 0;
      uint32_t phase = 0, looked = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = worker; ok && tile < num_tiles; tile += num_workers) {
        if (!mbar_wait_all(&acc_empty_bar[acc], acc_phase ^ 1, abort_flag)) {
          atomicCAS(p.err, 0u, 0x30000000u | static_cast<uint32_t>(acc));
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_looked(looked, &full_bar[stage], phase, abort_flag)) {
            atomicCAS(p.err, 0u, 0x20000000u | static_cast<uint32_t>(stage));
            ok = false;
            break;
          }
          tc_fence_after();
          const int next = stage + 1 == STAGES ? 0 : stage + 1;
          looked = mbar_look(&full_bar[next], next ? phase : phase ^ 1);
          // (descriptors hold addresses in units of 16 bytes)
          const uint64_t a_desc = desc0 + static_cast<uint64_t>(stage * (STAGE_BYTES / 16));
          const uint64_t b_desc = a_desc + A_BYTES / 16;
          umma_f16_ss_kblocks<CG, 1>(d_tmem, kblock_desc(a_desc, b_desc), idesc, kb != 0 ? 1u : 0u);
          // the stage is reusable (in both CTAs) once these MMAs have read it
          if constexpr (CG == 2) {
            umma_commit_cg2_warp(&empty_bar[stage], 3);
          } else {
            umma_commit_warp(&empty_bar[stage]);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        // accumulator complete: wake the epilogue warps of both CTAs
        if constexpr (CG == 2) {
          umma_commit_cg2_warp(&acc_full_bar[acc], 3);
        } else {
          umma_commit_warp(&acc_full_bar[acc]);
        }
        if ((acc ^= 1) == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int ew = warp - 2;
    const int quarter = warp & 3;   // TMEM lane quarter this warp may access
    const int half_sel = ew >> 2;   // which 128 accumulator columns this warp handles
    TOut *out = static_cast<TOut *>(p.out);
    const T16 *res = FORM == kWideRows ? nullptr : static_cast<const T16 *>(p.residual);
    [[maybe_unused]] uint8_t *my_out_base = tiles + STAGES * STAGE_BYTES + ew * C::EPI_WARP_BYTES;
    [[maybe_unused]] uint8_t *my_res = my_out_base + C::OUT_BUFS * EPI_BUF_BYTES;
    [[maybe_unused]] int out_buf = 0;
    [[maybe_unused]] uint32_t res_phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    // the accumulator is handed back to the leader's MMA thread, in whichever CTA it lives
    const uint32_t acc_empty_addr0 = mapa_u32(smem_u32(&acc_empty_bar[0]), 0);
    const uint32_t acc_empty_addr1 = mapa_u32(smem_u32(&acc_empty_bar[1]), 0);
    const int half_cols = bn / 2;
    [[maybe_unused]] constexpr int MAX_SUBS = BN / 2 / 32;
    // pieces of the residual in flight; the GELUs' code is too long to be written out four times (4096 x 3072 x 768 22.1 -> 23.7 us)
    [[maybe_unused]] constexpr int RES_AHEAD = ACT == kActNone || ACT == kActRelu ? MAX_SUBS : 1;
    for (int tile = worker; tile < num_tiles; tile += num_workers) {
      const int m_blk = (tile / p.num_n_blocks) * CG + cta_rank, n_blk = tile % p.num_n_blocks;
      const int row = m_blk * BM + quarter * 32 + lane;
      const bool row_ok = row < p.M;
      const int gcol_base = n_blk * bn + half_sel * half_cols;
      const uint32_t t_base = tmem_base + static_cast<uint32_t>(acc * BN + half_sel * half_cols) +
                              (static_cast<uint32_t>(quarter * 32) << 16);
      // pieces of 32 columns that hold real columns (uniform across the warp)
      const int n_sub = gcol_base >= p.N ? 0 : min(half_cols / 32, (p.N - gcol_base + 31) / 32);
      // one lane polls, the shuffle releases the others (256 threads would otherwise spin on the
      // barrier word beside the tensor pipe for most of a mainloop)
      auto wait_acc = [&]() __attribute__((always_inline)) -> bool {
        const bool done = mbar_wait_warp(&acc_full_bar[acc], acc_phase, abort_flag);
        if (!done) atomicCAS(p.err, 0u, 0x40000000u | static_cast<uint32_t>(acc));
        tc_fence_after();
        return done;
      };
      if constexpr (kWide) {
        // The warp owns 32 rows x half_cols accumulator columns, read from tensor memory in pieces of 32; the
        // next piece's load is in flight while this one goes through bias / activation / residual.  All of the
        // tile's residual, and its bias, are requested before the accumulator is waited for.
        const size_t row_off = static_cast<size_t>(row) * p.N + gcol_base;
        uint32_t raw[32];
        [[maybe_unused]] uint32_t rr[RES_AHEAD][16];
        auto fetch_res = [&](int sub, uint32_t *r) __attribute__((always_inline)) {
          if (res && row_ok && sub < n_sub) {
            ld_global_32B(res + row_off + sub * 32, r);
            if (gcol_base + sub * 32 + 16 < p.N) ld_global_32B(res + row_off + sub * 32 + 16, r + 8);
          }
        };
#pragma unroll
        for (int sub = 0; sub < RES_AHEAD; ++sub) fetch_res(sub, rr[sub]);
        if (p.bias) {
          const int c = gcol_base + lane * 4;
          float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
          if (c < p.N) b = __ldg(reinterpret_cast<const float4 *>(p.bias + c));
          __syncwarp();  // the previous tile's values have been read
          *reinterpret_cast<float4 *>(&bias_s[ew][lane * 4]) = b;
          __syncwarp();
        }
        if (!wait_acc()) break;
        if (n_sub > 0) tmem_ld_32x32(t_base, raw);
        auto piece = [&](int sub, uint32_t *r) __attribute__((always_inline)) {
          const int gcol = gcol_base + sub * 32;
          tmem_ld_wait_regs(raw);
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
          if (sub + 1 < n_sub) tmem_ld_32x32(t_base + (sub + 1) * 32, raw);  // overlaps the math below
          if (p.bias) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 b = *reinterpret_cast<const float4 *>(&bias_s[ew][sub * 32 + j]);
              v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
            }
          }
          act_fast_n<ACT, 32>(v);
          if (res) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float rv[8];
              unpack_res8<T16>(r + j / 2, rv);
#pragma unroll
              for (int e = 0; e < 8; ++e) v[j + e] += rv[e];
            }
            if constexpr (RES_AHEAD == 1) fetch_res(sub + 1, r);
          }
          store_row_pairs<TOut>(out, v, row, p.M, gcol, p.N);
        };
        // written out for a residual's registers only: a CTA of few tiles waits for its instructions
        if constexpr (FORM == kWideResidual && RES_AHEAD == MAX_SUBS) {
#pragma unroll
          for (int sub = 0; sub < MAX_SUBS; ++sub)
            if (sub < n_sub) piece(sub, rr[sub]);
        } else {
#pragma unroll 1
          for (int sub = 0; sub < n_sub; ++sub) piece(sub, rr[0]);
        }
      } else if (p.rows.fast) {
        // ---- staged rows.  Output leaves in chunks of cw columns: swizzled buffer -> one TMA store ----
        if (!wait_acc()) break;
        const int cw = p.cw;
        const int SUBS = cw / 32;                          // 32-column pieces per chunk
        const int OUT_ROW_BYTES = cw * static_cast<int>(sizeof(TOut));
        const int RES_ROW_BYTES = cw * 2;                  // residual is 16-bit
        const int row0 = m_blk * BM + quarter * 32;
        // 16-byte pieces of a staged row are XOR-swizzled the way TMA expects them:
        // 128-byte rows: piece ^ (row % 8); 64-byte rows: piece ^ ((row / 2) % 4)
        const int swz_out = OUT_ROW_BYTES == 128 ? (lane & 7) : ((lane >> 1) & 3);
        const int swz_res = RES_ROW_BYTES == 128 ? (lane & 7) : ((lane >> 1) & 3);
        uint32_t raw[32];
        if (n_sub > 0) tmem_ld_32x32(t_base, raw);
        bool chunk_ok = true;
        uint8_t *my_out = my_out_base;
#pragma unroll 1
        for (int sub = 0; sub < n_sub; ++sub) {
          const int gcol = gcol_base + sub * 32;
          const int sub_in_chunk = sub % SUBS;
          const int gcol_chunk = gcol - sub_in_chunk * 32;
          if (sub_in_chunk == 0) {
            if (res && lane == 0) {
              mbar_arrive_expect_tx(&res_bar[ew], 32 * RES_ROW_BYTES);
              tma_load_2d(my_res, &rows.res, &res_bar[ew], gcol_chunk, row0);
            }
            // the TMA store that last used this buffer must have finished reading it
            my_out = my_out_base + out_buf * EPI_BUF_BYTES;
            if (lane == 0) tma_store_wait_read<C::OUT_BUFS - 1>();
            __syncwarp();
            if constexpr (C::OUT_BUFS == 2) out_buf ^= 1;
          }
          tmem_ld_wait_regs(raw);
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
          if (sub + 1 < n_sub) tmem_ld_32x32(t_base + (sub + 1) * 32, raw);  // overlaps the math below
          if (p.bias) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              if (gcol + j < p.N) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(p.bias + gcol + j));
                v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
              }
            }
          }
          act_fast_n<ACT, 32>(v);
          if (res) {
            if (sub_in_chunk == 0) {
              if (!mbar_wait_warp(&res_bar[ew], res_phase, abort_flag)) {
                atomicCAS(p.err, 0u, 0x50000000u | static_cast<uint32_t>(ew));
                chunk_ok = false;
                break;
              }
              res_phase ^= 1;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // this piece is 64 bytes of the residual row
              const int phys = (sub_in_chunk * 4 + j) ^ swz_res;
              const uint4 q = *reinterpret_cast<const uint4 *>(my_res + lane * RES_ROW_BYTES + (phys << 4));
              const uint32_t r[4] = {q.x, q.y, q.z, q.w};
              float rv[8];
              unpack_res8<T16>(r, rv);
#pragma unroll
              for (int e = 0; e < 8; ++e) v[8 * j + e] += rv[e];
            }
          }
          if constexpr (sizeof(TOut) == 2) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // 32 columns = four 16-byte pieces of the staged row
              const int phys = (sub_in_chunk * 4 + j) ^ swz_out;
              store_out8<TOut>(reinterpret_cast<TOut *>(my_out + lane * OUT_ROW_BYTES + (phys << 4)), v + 8 * j);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4 *>(my_out + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                  make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
          if (sub_in_chunk == SUBS - 1 || sub + 1 == n_sub) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&rows.out, my_out, gcol_chunk, row0);  // rows / columns past M / N are clipped
              tma_store_commit();
            }
          }
        }
        if (!chunk_ok) break;
      } else {
        // ---- ragged rows, or a bias off its boundary ----
        if (!wait_acc()) break;
#pragma unroll 1
        for (int sub = 0; sub < n_sub; ++sub) {
          const int gcol = gcol_base + sub * 32, cols = p.N - gcol;
          uint32_t raw[32];
          tmem_ld_32x32(t_base + sub * 32, raw);
          const size_t off = static_cast<size_t>(row) * p.N + gcol;
          float v[32], rv[32];
          if (res && row_ok) load_row<T16, 32>(res + off, rv, cols, p.rows.vec);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = p.bias && j < cols ? __ldg(p.bias + gcol + j) : 0.f;
          tmem_ld_wait_regs(raw);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = act_apply_t<ACT>(__uint_as_float(raw[j]) + v[j]);
          if (row_ok) {
            if (res) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += rv[j];
            }
            store_row<TOut, 32>(out + off, v, cols, p.rows.vec);
          }
        }
      }
      tc_fence_before();
      if constexpr (CG == 2) mbar_arrive_cluster(acc ? acc_empty_addr1 : acc_empty_addr0);
      else mbar_arrive(&acc_empty_bar[acc]);
      if ((acc ^= 1) == 0) acc_phase ^= 1;
    }
    if constexpr (!kWide) {
      if (lane == 0) tma_store_wait<0>();  // all staged output has left shared memory
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
  // neither CTA of a pair may retire (or free tensor memory) while the other can still
  // signal its barriers or read its shared memory
  if constexpr (CG == 2) cluster_sync_all();
  tc_fence_after();
  if (warp == 1) {
    if constexpr (CG == 2) tmem_dealloc_cg2(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------
// The status word the tensor-core kernels write a give-up code into lives in the library
// image (static device storage, zero when the module is loaded), one copy per GPU: no device
// memory is allocated for it, so callers that must not allocate can use and read it too.  Host
// code needs the word's device address, looked up once per device ordinal (a process may
// drive several devices, one at a time).
constexpr int kMaxDevices = 64;
static __device__ uint32_t g_status_word;
static uint32_t *g_err_slots[kMaxDevices] = {nullptr};
static int current_device_index() {
  const int d = device_info().device;
  return (d >= 0 && d < kMaxDevices) ? d : 0;
}

uint32_t *device_error_slot() {
  uint32_t *&slot = g_err_slots[current_device_index()];
  if (!slot) {
    void *sym = nullptr;
    if (!check_cuda(cudaGetSymbolAddress(&sym, g_status_word), "cudaGetSymbolAddress(status word)")) return nullptr;
    slot = static_cast<uint32_t *>(sym);
  }
  return slot;
}

// Rows of the output or the residual in boxes of cw columns x 32 rows.
static bool encode_rows(CUtensorMap *map, const void *base, int32_t dtype, int64_t M, int64_t N, uint32_t cw, size_t elem) {
  const uint64_t dim[2] = {static_cast<uint64_t>(N), static_cast<uint64_t>(M)}, stride = static_cast<uint64_t>(N) * elem;
  const uint32_t box[2] = {cw, 32};
  return encode_tmap(map, dtype, 2, base, dim, &stride, box, cw * elem == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

template <typename T16, typename TOut, int ACT, int CG, int FORM>
static void launch_gemm_cg(const CUtensorMap &ta, const CUtensorMap &tb, const RowMaps<FORM != kStagedRows> &rows, const GemmParams &p,
                           int grid, cudaStream_t s) {
  auto kern = gemm_tcgen05_kernel<T16, TOut, ACT, CG, FORM>;
  constexpr size_t smem = gemm::Cfg<CG, FORM != kStagedRows>::SMEM_BYTES;
  static bool attr_set_on[kMaxDevices] = {false};  // the attribute is per device
  bool &attr_set = attr_set_on[current_device_index()];
  if (!attr_set) {
    if (!check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                    "cudaFuncSetAttribute(gemm)"))
      return;
    attr_set = true;
  }
  {
    ProfileScope prof(kCatGemm, s);
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>(grid)), dim3(gemm::THREADS), smem, s, CG, ta, tb, rows, p),
               "launch gemm");
  }
  launched("gemm_tcgen05_kernel");
}

// p.cta_group selects the variant; grid is CTAs (even for pairs)
template <typename T16, typename TOut, int ACT, bool kWide>
static void launch_gemm(const CUtensorMap &ta, const CUtensorMap &tb, const RowMaps<kWide> &rows, const GemmParams &p, int grid,
                        cudaStream_t s) {
  if constexpr (kWide && ACT != kActGeluTanh) {
    if (!p.residual) {
      if (p.cta_group == 2) launch_gemm_cg<T16, TOut, ACT, 2, kWideRows>(ta, tb, rows, p, grid, s);
      else launch_gemm_cg<T16, TOut, ACT, 1, kWideRows>(ta, tb, rows, p, grid, s);
      return;
    }
  }
  constexpr int FORM = kWide ? kWideResidual : kStagedRows;  // (the tanh GELU takes as many registers without a residual)
  if (p.cta_group == 2) launch_gemm_cg<T16, TOut, ACT, 2, FORM>(ta, tb, rows, p, grid, s);
  else launch_gemm_cg<T16, TOut, ACT, 1, FORM>(ta, tb, rows, p, grid, s);
}

template <typename T16, typename TOut, bool kWide>
static void launch_gemm_act(const CUtensorMap &ta, const CUtensorMap &tb, const RowMaps<kWide> &rows, const GemmParams &p,
                            int grid, int act, cudaStream_t s) {
  switch (act) {
  case MGPU_ACT_NONE: launch_gemm<T16, TOut, kActNone>(ta, tb, rows, p, grid, s); break;
  case MGPU_ACT_RELU: launch_gemm<T16, TOut, kActRelu>(ta, tb, rows, p, grid, s); break;
  case MGPU_ACT_GELU_ERF: launch_gemm<T16, TOut, kActGeluErf>(ta, tb, rows, p, grid, s); break;
  case MGPU_ACT_GELU_TANH: launch_gemm<T16, TOut, kActGeluTanh>(ta, tb, rows, p, grid, s); break;
  default: fail("mgpuMatmulEx16: unknown activation");
  }
}

template <typename T16, typename TOut>
static void launch_gemm_rows(const CUtensorMap &ta, const CUtensorMap &tb, GemmParams &p, int32_t dtype, int32_t out_dtype,
                             int grid, int act, cudaStream_t s) {
  if (p.rows.wide) {
    launch_gemm_act<T16, TOut, true>(ta, tb, RowMaps<true>{}, p, grid, act, s);
    return;
  }
  RowMaps<false> rows{ta, ta};  // placeholders for rows that are not staged
  // staged chunks of 64 columns (128-byte rows) for 16-bit output when a tile half is a multiple of
  // that, else of 32
  p.cw = sizeof(TOut) == 2 && (p.bn / 2) % 64 == 0 ? 64 : 32;
  const uint32_t cw = static_cast<uint32_t>(p.cw);
  if (p.rows.fast) {
    if (!encode_rows(&rows.out, p.out, out_dtype, p.M, p.N, cw, sizeof(TOut))) return;
    if (p.residual && !encode_rows(&rows.res, p.residual, dtype, p.M, p.N, cw, 2)) return;
  }
  launch_gemm_act<T16, TOut, false>(ta, tb, rows, p, grid, act, s);
}

// CTA pairs whenever there are at least two 128-row blocks; MDC_GEMM_CTA_GROUP=1|2 overrides
// (for measurements).
static int choose_cta_group(int64_t M) {
  static const int forced = [] {
    const char *e = getenv("MDC_GEMM_CTA_GROUP");
    return e ? atoi(e) : 0;
  }();
  if (forced == 1 || forced == 2) return forced;
  return M > gemm::BM ? 2 : 1;
}

// Tile width.  A Gemm takes ceil(tiles / workers) waves of tiles; the last wave is as long as
// the others however few tiles it holds, so for some shapes a narrower tile (more, cheaper
// tiles) wastes less: e.g. M = 32768, N = 768 on 74 CTA pairs is 6 waves of 256-wide tiles
// (5.2 needed) but 7 waves of 192-wide ones (6.9 needed) at 3/4 of the cost each.
// MDC_GEMM_BN=256|192|128 overrides (for measurements).
static int choose_bn(int64_t M, int64_t N, int cta_group, int sms) {
  static const int forced = [] {
    const char *e = getenv("MDC_GEMM_BN");
    return e ? atoi(e) : 0;
  }();
  if (forced == 256 || forced == 192 || forced == 128) return forced;
  const int64_t workers = sms / cta_group > 0 ? sms / cta_group : 1;
  const int64_t m_units = (M + gemm::BM * cta_group - 1) / (gemm::BM * cta_group);
  int best = 256;
  double best_cost = 1e300;
  for (int bn : {256, 192, 128}) {
    const int64_t tiles = m_units * ((N + bn - 1) / bn);
    const int64_t waves = (tiles + workers - 1) / workers;
    // per-tile cost: measured, a 192-wide tile takes about 0.95 of the time of a 256-wide one
    // (the k-block time is set by operand delivery into shared memory, which shrinks only
    // from 32 to 28 KiB per CTA), a 128-wide one about 0.8
    const double cost = static_cast<double>(waves) * (bn == 256 ? 1.0 : bn == 192 ? 0.95 : 0.8);
    if (cost < best_cost * 0.97) {  // prefer the wider tile unless the gain is clear
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

// A figure of merit of a one-wave tile, near its time in microseconds, at most one CTA per SM.  Terms: launch and drain;
// MMAs; operand bytes through the SM's load path; one barrier hand-over per ring stage; epilogue columns; CTAs to place;
// pairing.  An MMA takes half a cycle per column, but no less than it needs to read A and to start: 25 cycles for 64 rows
// and 16 to 32 columns, 40 for 128 rows (measured; a few rows are therefore cut into tiles of 64).  The weights are those
// whose choice was best over 770 shapes and all their tiles (M 16 - 4096, N 256 - 4096, K 256 - 4096, weights from HBM,
// dependent launches in a graph); on 300 others it takes 1.007 of the time of the best tile on average, 1.04 in 19
// of 20.
static float one_wave_cost(const GemmTile &t, int64_t M, int64_t N, int num_kb, int sms) {
  const int64_t m_tiles = (M + t.box_m * t.cg - 1) / (t.box_m * t.cg), n_tiles = (N + t.bn - 1) / t.bn;
  const int64_t ctas = m_tiles * n_tiles * t.cg;
  if (ctas > sms) return 1e30f;
  const int steps = (num_kb + t.depth - 1) / t.depth;
  const int rows = M < t.box_m ? static_cast<int>(M) : t.box_m;
  const float bn = static_cast<float>(t.bn);
  const float start = t.cg == 2 ? 35.f + 0.15f * bn : t.mma_m == 64 ? 21.7f + 0.17f * bn : 31.5f + 0.25f * bn;
  const float mma = num_kb * 4 * fmaxf(start, 0.5f * bn) / 1900.f;
  const float bytes = steps * t.depth * static_cast<float>(rows + t.bn / t.cg) * 128.f / 1e5f;  // (a stage is filled whole)
  float us = 2.55f + 2.38f * mma + 0.282f * bytes + 0.118f * steps + 0.00855f * bn +
             0.836f * static_cast<float>(ctas) / static_cast<float>(sms);
  if (t.cg == 2) us += 2.38f;
  // Rows that are no multiple of eight values are stored one by one, about a nanosecond each: 260 such shapes 1.006 of the best
  // tile's time, 1.126 without this term (366 x 337 x 64 7.2 -> 3.9 us, 1739 x 59 x 32 fp32 4.7 -> 3.1).
  if (N % 8) us += static_cast<float>(rows * std::min<int64_t>(t.bn, N)) / 1024.f;
  return us;
}

// The fastest one-wave tile for a problem of at most one 128 x 128 tile per SM.
static GemmTile choose_one_wave(int64_t M, int64_t N, int64_t K, int sms) {
  const int num_kb = static_cast<int>((K + 63) / 64);
  GemmTile best;
  float best_us = 1e30f;
  for (int cg = 1; cg <= 2; ++cg)
    for (int most : {32, 64, 128}) {
      if (most < 128 && cg == 2) continue;
      if (most > 32 && most >= 2 * M) continue;
      // Boxes as high as an equal share of the rows, in whole swizzle groups: rows out of bounds are slow to fill (75 x 2304 x 768 in
      // tiles of 64 and 11 rows 4.9 us, in two of 40 3.7).
      const int64_t shares = (M + most * cg - 1) / (most * cg) * cg;
      const int box_m = static_cast<int>(((M + shares - 1) / shares + 7) / 8 * 8), mma_m = cg == 1 && box_m <= 64 ? 64 : 128;
      for (int bn : {16, 32, 48, 64, 96, 128, 192, 256}) {
        if (cg == 2 && bn < 64) continue;
        // k-blocks that come one box at a time: 16 columns a box lose (51 x 2264 x 1528 7.5 us, with 32 columns 6.2; 18 x 2280 x
        // 1424 6.3 and 5.3; 160 shapes 1.044 of the best tile's time on average with them, 1.033 without)
        if (bn == 16 && K % 64) continue;
        for (int depth : {4, 2, 1}) {
          if (depth > num_kb) continue;
          const int steps = (num_kb + depth - 1) / depth, stage = depth * (box_m + bn / cg) * 128;
          // all of an SM's shared memory: the ring has to cover the latency of operands that come out
          // of L2 at 60 - 100 bytes per cycle.  Half of it, so that the next kernel's CTA fits beside
          // this one, loses more than that overlap wins: 2048 x 1024 x 4096 31.7 -> 22.0 us,
          // 1000 x 1024 x 4096 25.8 -> 18.0, 99 x 768 x 3072 11.7 -> 10.5; a 12-layer pass over 99 tokens,
          // where every kernel is of this kind, 501 -> 450 us.
          int stages = (220 * 1024 - (mma_m - box_m) * 128) / stage;
          if (stages > steps) stages = steps;
          if (stages > 16) stages = 16;
          if (stages < 1 || (stages < 2 && steps > 1)) continue;
          GemmTile t;
          t.one_wave = true, t.cg = cg, t.box_m = box_m, t.mma_m = mma_m, t.bn = bn, t.depth = depth, t.stages = stages;
          const float us = one_wave_cost(t, M, N, num_kb, sms);
          if (us < best_us) best_us = us, best = t;
        }
      }
    }
  return best;
}

GemmTile choose_gemm_tile(int64_t M, int64_t N, int64_t K, int sms) {
  // the choice takes a few microseconds: kept per shape (a plan, not a result)
  struct Entry {
    int64_t M = -1, N = -1, K = -1;
    int sms = 0;
    GemmTile tile;
  };
  static thread_local Entry cache[64];
  Entry &e = cache[(static_cast<uint64_t>(M) * 0x9E3779B97F4A7C15ull ^ static_cast<uint64_t>(N) * 0xC2B2AE3D27D4EB4Full ^
                    static_cast<uint64_t>(K) * 0x165667B19E3779F9ull) >> 58];
  if (e.M == M && e.N == N && e.K == K && e.sms == sms) return e.tile;
  GemmTile t;
  // One wave: up to one 128 x 128 tile per SM.  One-wave / persistent, us, at the line: 991 x 2304 x 768 with residual 7.2 / 7.4,
  // 676 x 3072 x 768 6.6 / 6.9, 2841 x 768 x 768 6.5 / 6.8, 2433 x 768 x 768 with residual 7.10 / 7.04; beyond it the persistent
  // kernel takes 0.94 of the best one-wave tile's time.
  const bool forced = getenv("MDC_GEMM_BN") || getenv("MDC_GEMM_CTA_GROUP");
  if (!forced && ((M + 127) / 128) * ((N + 127) / 128) <= sms)
    t = choose_one_wave(M, N, K, sms);
  // A long K in tiles of 128 columns goes to the persistent kernel where its pairs of 256 x 128 come in one round.  One-wave /
  // persistent, us: 2341 x 768 x 3072 14.9 / 13.6, 1711 x 1024 x 3712 17.3 / 15.6, 1718 x 1024 x 4096 18.3 / 16.8, 2978 x 768 x 1920 11.2 /
  // 10.5; below K = 1400 0.98 of the time instead, and with tiles of 96 columns 1.0, of 64 0.88.  It is the kernel and not the cost
  // above: no tile of the one-wave kernel does as well.  2341 x 768 x 3072 in pairs with 4, 2 and 1 k-blocks to a stage 14.9, 16.2, 20.5,
  // in single CTAs with 2 and 1 15.2, 15.6 (192 columns 17.5 and more).  Why its stages of one k-block turn slower than the
  // persistent kernel's is not known.
  if (t.one_wave && t.bn >= 128 && K >= 1400 && M > gemm::BM && ((M + 255) / 256) * ((N + 127) / 128) <= sms / 2) {
    t = GemmTile();
    t.cg = 2, t.bn = 128;
  } else if (!t.one_wave) {
    t.cg = choose_cta_group(M);
    t.bn = choose_bn(M, N, t.cg, sms);
  }
  e.M = M, e.N = N, e.K = K, e.sms = sms, e.tile = t;
  return t;
}

// persistent grid: one worker (CTA or CTA pair) per tile up to the number the device holds
static int gemm_grid(const GemmParams &p, int sms) {
  const int cg = p.cta_group;
  const int64_t tiles = static_cast<int64_t>((p.num_m_blocks + cg - 1) / cg) * p.num_n_blocks;
  if (tiles > 0x7fffffff) return -1;
  const int64_t max_workers = sms / cg;
  if (tiles <= max_workers) return static_cast<int>(tiles * cg);
  // The kernel takes ceil(tiles / workers) rounds whatever the last round holds.  Use the
  // fewest workers that still finish in that many rounds: the SMs left idle draw no power,
  // which the power-capped tensor cores of the others turn into clock (MDC_GEMM_EVEN_WAVES=0
  // uses every SM).
  static const bool even = !(getenv("MDC_GEMM_EVEN_WAVES") && atoi(getenv("MDC_GEMM_EVEN_WAVES")) == 0);
  const int64_t rounds = (tiles + max_workers - 1) / max_workers;
  const int64_t workers = even ? (tiles + rounds - 1) / rounds : max_workers;
  return static_cast<int>(workers * cg);
}

// The whole of mgpuMatmulEx16 after the argument checks: tile choice, tensor maps, launch.
// Shared by every entry point that ends in this Gemm; allocates nothing.
static void matmul16_launch(const char *who, const void *a, const void *w_nk, const float *bias, const void *residual,
                            void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype, int32_t out_dtype,
                            int32_t act, bool w_ready, cudaStream_t s) {
  const DeviceInfo &di = device_info();
  char msg[160];
  auto failf = [&](const char *what) {
    snprintf(msg, sizeof(msg), "%s: %s", who, what);
    fail(msg);
  };
  uint32_t *err = device_error_slot();
  if (!err) return;

  const GemmTile tile = choose_gemm_tile(M, N, Kp, di.sms);
  if (tile.one_wave) {
    gemm_one_wave_launch(tile, a, w_nk, bias, residual, out, M, N, Kp, dtype, out_dtype, act, w_ready, s);
    return;
  }
  const int cta_group = tile.cg, bn = tile.bn;
  CUtensorMap ta, tb;
  if (!encode_tmap_2d(&ta, a, dtype, static_cast<uint64_t>(Kp), static_cast<uint64_t>(M),
                      static_cast<uint64_t>(Kp) * 2, gemm::BK, gemm::BM) ||
      !encode_tmap_2d(&tb, w_nk, dtype, static_cast<uint64_t>(Kp), static_cast<uint64_t>(N),
                      static_cast<uint64_t>(Kp) * 2, gemm::BK, bn / cta_group))
    return;

  GemmParams p;
  p.cta_group = cta_group;
  p.bn = bn;
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(Kp);
  p.bias = bias;
  p.residual = residual;
  p.out = out;
  p.rows = row_access(N, out, dtype_size(out_dtype), residual, bias);
  p.num_m_blocks = static_cast<int>((M + gemm::BM - 1) / gemm::BM);
  p.num_n_blocks = static_cast<int>((N + bn - 1) / bn);
  p.err = err;
  const int grid = gemm_grid(p, di.sms);
  if (grid <= 0) { failf("too many tiles"); return; }

  if (dtype == MGPU_DTYPE_F16) {
    if (out_dtype == MGPU_DTYPE_F16) launch_gemm_rows<__half, __half>(ta, tb, p, dtype, out_dtype, grid, act, s);
    else if (out_dtype == MGPU_DTYPE_F32) launch_gemm_rows<__half, float>(ta, tb, p, dtype, out_dtype, grid, act, s);
    else failf("output type must be the operand type or F32");
  } else {
    if (out_dtype == MGPU_DTYPE_BF16) launch_gemm_rows<__nv_bfloat16, __nv_bfloat16>(ta, tb, p, dtype, out_dtype, grid, act, s);
    else if (out_dtype == MGPU_DTYPE_F32) launch_gemm_rows<__nv_bfloat16, float>(ta, tb, p, dtype, out_dtype, grid, act, s);
    else failf("output type must be the operand type or F32");
  }
}
}  // namespace mdc

using namespace mdc;

namespace mdc {
void matmul16(const void *a, const void *w_nk, const float *bias, const void *residual, void *out, int64_t M, int64_t N,
              int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act, bool w_ready, void *stream) {
  if (M <= 0 || N <= 0) return;
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  if (!dtype_is16(dtype)) { fail("mgpuMatmulEx16: dtype must be F16 or BF16"); return; }
  if (Kp <= 0 || (Kp & 7)) { fail("mgpuMatmulEx16: K must be a positive multiple of 8"); return; }
  if (M > 0x7fffffff || N > 0x7fffffff || Kp > 0x7fffffff) { fail("mgpuMatmulEx16: shape too large"); return; }
  if ((reinterpret_cast<uintptr_t>(a) & 15u) || (reinterpret_cast<uintptr_t>(w_nk) & 15u)) {
    fail("mgpuMatmulEx16: operands must be 16-byte aligned");
    return;
  }
  matmul16_launch("mgpuMatmulEx16", a, w_nk, bias, residual, out, M, N, Kp, dtype, out_dtype, act, w_ready, as_stream(stream));
}
}  // namespace mdc

MDC_API void mgpuMatmulEx16(const void *a, const void *w_nk, const float *bias, const void *residual,
                            void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype,
                            int32_t out_dtype, int32_t act, void *stream) {
  matmul16(a, w_nk, bias, residual, out, M, N, Kp, dtype, out_dtype, act, false, stream);
}

MDC_API uint32_t mgpuOpsCheckDeviceStatus(void *stream) {
  uint32_t *err = device_error_slot();  // an address look-up; allocates nothing
  if (!err) return 0xffffffffu;
  uint32_t h = 0;
  if (!check_cuda(cudaMemcpyAsync(&h, err, sizeof(h), cudaMemcpyDeviceToHost, as_stream(stream)), "read device status"))
    return 0xffffffffu;
  if (!check_cuda(cudaStreamSynchronize(as_stream(stream)), "cudaStreamSynchronize")) return 0xffffffffu;
  if (h != 0) {
    char msg[96];
    snprintf(msg, sizeof(msg), "a tensor-core kernel gave up waiting (code 0x%08x)", h);
    fail(msg);
    cudaMemsetAsync(err, 0, sizeof(uint32_t), as_stream(stream));
  }
  return h;
}

// =========================================================================================
// mgpuMatmulNoAlloc: mgpuMatmul for callers that must not allocate device memory.
//
// mgpuMatmul needs two temporaries (the 16-bit copies of the input and of the transposed
// weight) and takes them from the runtime's device pool, which calls cudaMalloc whenever the
// pool has no fitting block.  Some callers cannot afford that call: a serving loop whose
// latency budget has no room for the device-wide synchronisation cudaMalloc implies, or a
// process in which another component has reserved all device memory up front so that any
// further allocation fails.  For them this entry point does the same computation with the
// temporaries placed in a fixed array that is part of the library image.
//
// * The array is kNoAllocScratchBytes (16 MiB) of device memory per GPU that loads the
//   library, held until the process exits whether the entry point is used or not.
// * Limit: roundup256(M * Kp * 2) + roundup256(N * Kp * 2) <= 16 MiB with Kp = K rounded
//   up to 8 (for example M x N x K = 1024 x 768 x 4096, or 2048 x 512 x 3072).  Larger problems are
//   rejected with the sticky status set and nothing launched.
// * The first call on a device looks the array's device address up
//   (cudaGetSymbolAddress); make that first call before starting any stream capture.
// * All calls on a device share the one array, which keeps whatever the last call left in
//   it.  Everything a call reads from it is written by that call first (the padded operand
//   copies), but two calls that overlap on the GPU (different streams without an ordering
//   between them) race on it: order them.
// * While profiling is off (mgpuOpsProfileBegin creates CUDA events), no cudaMalloc /
//   cudaFree / pool call and no other allocating routine runs on this path.  A kernel that
//   gives up a bounded wait reports through the same status word as every other entry point
//   (mgpuOpsCheckDeviceStatus, which allocates nothing either).
// =========================================================================================
namespace mdc {
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// host-side cache of the array's device address, per device ordinal
static unsigned char *g_noalloc_ptr[kMaxDevices] = {nullptr};
}  // namespace mdc

MDC_API void mgpuMatmulNoAlloc(float *input, float *weight, float *bias, float *output, int64_t M,
                               int64_t N, int64_t K, void *stream) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0) { fail("mgpuMatmulNoAlloc: K must be positive"); return; }
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  if (M > 0x7fffffff || N > 0x7fffffff || K > 0x7fffffff) { fail("mgpuMatmulNoAlloc: shape too large"); return; }
  const int64_t Kp = (K + 7) / 8 * 8;
  auto up256 = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t a_bytes = up256(static_cast<size_t>(M) * Kp * 2), w_bytes = up256(static_cast<size_t>(N) * Kp * 2);
  if (a_bytes + w_bytes > kNoAllocScratchBytes) {
    char msg[200];
    snprintf(msg, sizeof(msg),
             "mgpuMatmulNoAlloc: %lld x %lld x %lld needs %zu bytes of scratch, the fixed array holds %zu",
             (long long)M, (long long)N, (long long)K, a_bytes + w_bytes, kNoAllocScratchBytes);
    fail(msg);
    return;
  }
  if (di.device < 0 || di.device >= kMaxDevices) { fail("mgpuMatmulNoAlloc: device ordinal out of range"); return; }
  // set-up, once per device, with that device current: the array's name is only a host-side
  // handle; kernels need the address the runtime resolves for this device
  if (!g_noalloc_ptr[di.device]) {
    void *sym = nullptr;
    if (!check_cuda(cudaGetSymbolAddress(&sym, g_noalloc_scratch), "cudaGetSymbolAddress(scratch)")) return;
    g_noalloc_ptr[di.device] = static_cast<unsigned char *>(sym);
  }
  unsigned char *base = g_noalloc_ptr[di.device];
  void *a16 = base;
  void *w16 = base + a_bytes;
  cudaStream_t s = as_stream(stream);
  OperandList list;
  if (gemm_takes_few_rows(M, N, K, weight, output, di.sms)) {
    if (few_rows_convert(input, output, M, N, K, di.sms)) {
      gemm_few_rows(nullptr, input, weight, bias, output, M, N, K, s);
      return;
    }
    list.cast(input, a16, M, K, Kp);
    list.launch(MGPU_DTYPE_F16, stream, true);
    gemm_few_rows(a16, input, weight, bias, output, M, N, K, s);
    return;
  }
  list.pack(weight, w16, K, N);
  list.cast(input, a16, M, K, Kp);
  list.launch(MGPU_DTYPE_F16, stream);
  matmul16_launch("mgpuMatmulNoAlloc", a16, w16, bias, nullptr, output, M, N, Kp, MGPU_DTYPE_F16, MGPU_DTYPE_F32,
                  MGPU_ACT_NONE, false, s);
}
