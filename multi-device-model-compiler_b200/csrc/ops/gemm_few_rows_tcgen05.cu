// Tensor-core Gemm for a few rows against an fp32 weight as the caller has it: out[M, N] = A[M, Kp] . W[K, N]
// + bias[N], M <= 64, A fp16, W fp32 rounded to fp16 on its way into shared memory, fp32 accumulation.
//
// With few rows every weight is used once, by one CTA, so a 16-bit copy in memory would only be written
// to be read back, and this kernel is bound by the bytes of W (4 K N) or, where those are few, by
// latency.  Eight warps read W straight into registers, 16 vector loads of a thread in flight (64 KB an
// SM); a warp fills a ring stage of 128 k x 16 columns or 64 k x 32 by itself, converting to core
// matrices of 8 columns x 8 k.  A comes by TMA, converted by a launch ahead; W and the bias do not wait for it: that
// kernel lets this one start after its own wait, so what is older than it is complete.  Where A is small (kConvert,
// few_rows_convert) eight more warps read and round it here instead, and there is no launch ahead: 16 x 768 x 768 6.1 ->
// 4.9 us a call, 16 x 256 x 256 6.1 -> 3.7.
//
// The accumulator has 64 rows: an MMA of 128 rows and 16 or 32 columns takes 40 cycles, one of 64 rows 25.  A's box is as high
// as there are rows, and the ring leaves L1 to the loads in flight (RING_SMEM).  Whole calls out of memory, with 128 rows, boxes of
// 32 or 64 and a ring of 220 KB / now, one after another from the host (in a graph): 16 x 1000 x 2048 13.0 / 9.2 us (12.8 / 8.0),
// 1 x 1000 x 2048 12.2 / 7.4 (11.8 / 7.0), 64 x 1000 x 2048 13.1 / 9.5 (12.9 / 9.2), 8 x 2000 x 4000 18.8 / 11.6 (18.5 / 11.3), 16 x
// 4096 x 4096 22.1 / 19.1 (21.9 / 19.0; 3.5 TB/s), 16 x 1000 x 512 4.6 / 4.4 (4.35 / 4.13).  Weights that are converted first
// instead: gemm_plan.h.
//
// K order: one sum over K in steps of 16, as in the other Gemm kernels; a row's bits do not depend on
// which of them takes a call.
#include "gemm_common.cuh"
#include "gemm_plan.h"
#include "ops_common.h"

namespace mdc {

namespace fewrows {
constexpr int LOAD_WARPS = 8;
// with the input converted here, as many warps again for it
constexpr int threads(bool convert) { return 64 + LOAD_WARPS * (convert ? 64 : 32); }
// What the ring may take.  Every load of W in flight holds its line in L1, 64 KB an SM, so L1 has to keep that much: with
// 200 KB of ring 16 x 384 x 3968 takes 17.5 us, with 160 KB 11.4, with 128 KB 10.6, and less gains nothing (16 x 1088 x 6144 24.9,
// 16.9, 15.9).  64 rows need 170 KB for a stage a warp.
constexpr int RING_SMEM = 128 * 1024, MAX_SMEM = 172 * 1024;
// an MMA reads 64 rows of A whatever the box holds
constexpr int MMA_M = 64;
constexpr int fixed_bytes(int box_m) { return 1024 + (MMA_M - box_m) * 128; }
// Columns in groups of eight, k in groups of eight: 128-byte core matrices.  They lie 144 bytes apart along the
// columns, which puts the eight 16-byte stores of a quarter-warp on different banks.
constexpr int SBO = 144;
template <int BN>
struct Cfg {
  static constexpr int STAGE_K = 2048 / BN;                      // a warp's 16 loads of 4 values per lane
  static constexpr int LBO = BN == 16 ? 288 : 4 * SBO;           // bytes from one group of eight k to the next
  static constexpr int B_BYTES = STAGE_K / 8 * LBO;              // 4608
  static constexpr int stage_bytes(int box_m) { return STAGE_K / 64 * box_m * 128 + B_BYTES; }
  static constexpr int stages(int box_m) {
    const int n = (RING_SMEM - fixed_bytes(box_m)) / stage_bytes(box_m);
    return n < LOAD_WARPS ? LOAD_WARPS : n;
  }
};
constexpr int MAX_STAGES = Cfg<32>::stages(8);  // the lowest boxes and the shorter stages: 21; with 16 columns 18
static_assert(Cfg<16>::stages(8) <= MAX_STAGES, "a barrier for every stage");
// Warp w fills stages' worth w, w + 8, ... of K and waits for its stage's previous use by parity alone: with fewer
// stages than warps one would be two uses ahead and pass.
template <int BN>
constexpr bool ring_holds_every_warp = Cfg<BN>::stages(8) >= LOAD_WARPS && Cfg<BN>::stages(MMA_M) >= LOAD_WARPS;
static_assert(ring_holds_every_warp<16> && ring_holds_every_warp<32>, "a stage for every loading warp");
static_assert(fixed_bytes(MMA_M) + Cfg<16>::stages(MMA_M) * Cfg<16>::stage_bytes(MMA_M) <= MAX_SMEM, "the largest ring fits");
}  // namespace fewrows

struct FewRowsParams {
  const float *x;  // kConvert: the input, M x K
  const float *w, *bias;
  float *out;
  int M, N, K;
  int box_m, stages, steps;  // rows of A's box, a multiple of 8; steps: stages' worth of K
  int w_vec, out_vec;        // rows of W / of out and the bias in 16-byte vectors
  int x_vec;                 // rows of x
  uint32_t *err;
};

template <int BN, bool kConvert>
__global__ void __launch_bounds__(fewrows::threads(kConvert), 1)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmap_a, const FewRowsParams p) {
  using namespace fewrows;
  using namespace ptx;
  using C = Cfg<BN>;
  constexpr int KBS = C::STAGE_K / 64;  // 64-wide k-blocks of A per stage
  extern __shared__ uint8_t smem_dyn[];
  __shared__ uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_bar;
  __shared__ uint32_t tmem_slot, abort_flag_s;
  volatile uint32_t *abort_flag = &abort_flag_s;
  uint8_t *a_s = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~static_cast<uintptr_t>(1023));
  const int a_kb = p.box_m * 128, a_bytes = KBS * a_kb;
  // what an MMA reads beyond the last stage's A must not be W's part
  uint8_t *b_s = a_s + p.stages * a_bytes + (MMA_M - p.box_m) * 128;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int col0 = blockIdx.x * BN;

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    if (!kConvert) tma_prefetch_desc(&tmap_a);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 2);  // A's bytes, or the warp that brings them, and the warp that brings W
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 32);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_launch_dependents();  // after this CTA holds its tensor memory (see gemm_tcgen05.cu)
  if (kConvert) pdl_wait();  // no conversion ahead that would have waited

  if (kConvert && warp == 0) {
    // nothing to fetch
  } else if (warp == 0) {
    // ------------------------------ A ------------------------------
    pdl_wait();
    int stage = 0;
    uint32_t phase = 0, looked = 0;
    for (int i = 0; i < p.steps; ++i) {
      if (!mbar_wait_looked(looked, &empty_bar[stage], phase ^ 1, abort_flag)) {
        atomicCAS(p.err, 0u, 0x91000000u | static_cast<uint32_t>(stage));
        break;
      }
      const int next = stage + 1 == p.stages ? 0 : stage + 1;
      looked = mbar_look(&empty_bar[next], next ? phase ^ 1 : phase);
      if (elect_one()) {
        mbar_arrive_expect_tx(&full_bar[stage], static_cast<uint32_t>(a_bytes));
#pragma unroll
        for (int kb = 0; kb < KBS; ++kb)
          tma_load_2d(a_s + stage * a_bytes + kb * a_kb, &tmap_a, &full_bar[stage], (i * KBS + kb) * 64, 0);
      }
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    const uint32_t idesc = make_idesc_f16(MMA_M, BN, false, false, false);
    const uint64_t a0 = make_smem_desc_sw128(smem_u32(a_s), 16, 1024);
    // no swizzle (see make_smem_desc_sw128 for the fields)
    const uint64_t b0 = static_cast<uint64_t>(smem_u32(b_s) >> 4) | static_cast<uint64_t>(C::LBO / 16) << 16 |
                        static_cast<uint64_t>(SBO / 16) << 32 | static_cast<uint64_t>(1) << 46;
    int stage = 0;
    uint32_t phase = 0, looked = 0;
    bool ok = true;
    for (int i = 0; i < p.steps; ++i) {
      if (!mbar_wait_looked(looked, &full_bar[stage], phase, abort_flag)) {
        atomicCAS(p.err, 0u, 0x92000000u | static_cast<uint32_t>(stage));
        ok = false;
        break;
      }
      tc_fence_after();
      const int next = stage + 1 == p.stages ? 0 : stage + 1;
      looked = mbar_look(&full_bar[next], next ? phase : phase ^ 1);
      const uint64_t ad = a0 + static_cast<uint64_t>(stage * (a_bytes >> 4)), bd = b0 + static_cast<uint64_t>(stage * (C::B_BYTES >> 4));
#pragma unroll
      for (int kb = 0; kb < KBS; ++kb)
        umma_f16_ss_kblocks<1, 1, 2 * C::LBO / 16>(tmem_base, kblock_desc(ad + static_cast<uint64_t>(kb * (a_kb >> 4)),
                                                                         bd + static_cast<uint64_t>(kb * (8 * C::LBO >> 4))),
                                                  idesc, (i | kb) != 0 ? 1u : 0u);
      umma_commit_warp(&empty_bar[stage]);
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    if (ok) umma_commit_warp(&acc_bar);
  } else if (kConvert && warp >= 2 + LOAD_WARPS) {
    // ------------------------------ A out of the fp32 input ------------------------------
    // A warp fills a stage's worth of rows by itself, in pieces of 16 rows x 64 k (eight lanes a row, four rows a load),
    // two pieces' loads in flight.
    const int aw = warp - 2 - LOAD_WARPS, chunk = lane & 7;
    const int pieces = (p.M + 15) / 16 * KBS;
    auto load = [&](int i, int piece, float4 (&v)[4][2]) __attribute__((always_inline)) {
      const int k = i * C::STAGE_K + piece % KBS * 64 + chunk * 8;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = piece / KBS * 16 + r * 4 + (lane >> 3);
        const float *src = p.x + static_cast<int64_t>(m) * p.K + k;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
          const int left = m < p.M ? p.K - k - 4 * h : 0;  // values of the row from here on
          if (p.x_vec) {
            if (left > 0) q = __ldg(reinterpret_cast<const float4 *>(src + 4 * h));
          } else {
            if (left > 0) q.x = __ldg(src + 4 * h);
            if (left > 1) q.y = __ldg(src + 4 * h + 1);
            if (left > 2) q.z = __ldg(src + 4 * h + 2);
            if (left > 3) q.w = __ldg(src + 4 * h + 3);
          }
          v[r][h] = q;
        }
      }
    };
    auto store = [&](int stage, int piece, const float4 (&v)[4][2]) __attribute__((always_inline)) {
      uint8_t *dst = a_s + stage * a_bytes + piece % KBS * a_kb;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = piece / KBS * 16 + r * 4 + (lane >> 3);
        const float4 lo = v[r][0], hi = v[r][1];
        if (m < p.M)  // 128-byte swizzle: 16-byte chunk c of row m lies at c ^ (m % 8)
          *reinterpret_cast<uint4 *>(dst + m * 128 + ((chunk ^ (m & 7)) << 4)) =
              make_uint4(pack_pair<__half>(lo.x, lo.y), pack_pair<__half>(lo.z, lo.w), pack_pair<__half>(hi.x, hi.y), pack_pair<__half>(hi.z, hi.w));
      }
    };
    for (int i = aw; i < p.steps; i += LOAD_WARPS) {
      const int stage = i % p.stages;
      const uint32_t phase = static_cast<uint32_t>(i / p.stages) & 1u;
      bool gone = false;
      for (int piece = 0; piece < pieces; piece += 2) {
        float4 va[4][2], vb[4][2];
        load(i, piece, va);
        if (piece + 1 < pieces) load(i, piece + 1, vb);
        // the loads are in flight; only now does the stage have to be free
        if (piece == 0 && !mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
          if (lane == 0) atomicCAS(p.err, 0u, 0x94000000u | static_cast<uint32_t>(stage));
          gone = true;
          break;
        }
        store(stage, piece, va);
        if (piece + 1 < pieces) store(stage, piece + 1, vb);
      }
      if (gone) break;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
    }
  } else {
    // ------------------------------ W, then the epilogue ------------------------------
    const int lw = warp - 2;
    constexpr int LANES_N = BN / 4;                 // lanes side by side in a row of W
    constexpr int OCTETS = 32 / LANES_N;            // groups of eight k that a warp covers per pass of eight loads
    const int n = (lane % LANES_N) * 4, octet = lane / LANES_N;
    const int gcol = col0 + n;
    bool ok = true;
    for (int i = lw; i < p.steps; i += LOAD_WARPS) {
      float4 v[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int k = i * C::STAGE_K + (h * OCTETS + octet) * 8 + e;
          float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
          const float *src = p.w + static_cast<int64_t>(k) * p.N + gcol;
          if (k < p.K) {
            if (p.w_vec) {
              if (gcol < p.N) q = __ldcs(reinterpret_cast<const float4 *>(src));
            } else {
              if (gcol < p.N) q.x = __ldcs(src);
              if (gcol + 1 < p.N) q.y = __ldcs(src + 1);
              if (gcol + 2 < p.N) q.z = __ldcs(src + 2);
              if (gcol + 3 < p.N) q.w = __ldcs(src + 3);
            }
          }
          v[h][e] = q;
        }
      const int stage = i % p.stages;
      const uint32_t phase = static_cast<uint32_t>(i / p.stages) & 1u;
      if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag)) {
        atomicCAS(p.err, 0u, 0x90000000u | static_cast<uint32_t>(stage));
        ok = false;
        break;
      }
      uint8_t *dst = b_s + stage * C::B_BYTES;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = j == 0 ? v[h][e].x : j == 1 ? v[h][e].y : j == 2 ? v[h][e].z : v[h][e].w;
          const uint4 q = make_uint4(pack_pair<__half>(f[0], f[1]), pack_pair<__half>(f[2], f[3]),
                                     pack_pair<__half>(f[4], f[5]), pack_pair<__half>(f[6], f[7]));
          *reinterpret_cast<uint4 *>(dst + (h * OCTETS + octet) * C::LBO + ((n + j) >> 3) * SBO + ((n + j) & 7) * 16) = q;
        }
      fence_proxy_async_smem();  // the tensor core reads the stage through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
    }
    const int quarter = warp & 3;
    if (ok && quarter * 16 < p.M) {
      // the two warps of a lane quarter take 16 columns each; 16 columns in all are the first one's
      const int c0 = (lw >> 2) * 16;
      const int row = quarter * 16 + lane, cols = p.N - (col0 + c0);
      if (c0 < BN && cols > 0) {
        float b[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) b[j] = p.bias && j < cols ? __ldg(p.bias + col0 + c0 + j) : 0.f;
        if (!mbar_wait_warp(&acc_bar, 0, abort_flag)) {
          atomicCAS(p.err, 0u, 0x93000000u);
        } else {
          tc_fence_after();
          uint32_t acc[16];
          tmem_ld_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(c0), acc);
          tmem_ld_wait_regs(acc);
#pragma unroll
          for (int j = 0; j < 16; ++j) b[j] += __uint_as_float(acc[j]);
          if (lane < 16 && row < p.M) {  // an accumulator of 64 rows has 16 in each quarter of the lanes
            float *dst = p.out + static_cast<int64_t>(row) * p.N + col0 + c0;
            if (p.out_vec) {
#pragma unroll
              for (int j = 0; j < 16; j += 4)
                if (j < cols) *reinterpret_cast<float4 *>(dst + j) = make_float4(b[j], b[j + 1], b[j + 2], b[j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (j < cols) dst[j] = b[j];
            }
          }
        }
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
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 32);
}

template <int BN, bool kConvert>
static void launch_few_rows(const CUtensorMap &ta, FewRowsParams &p, cudaStream_t s) {
  using C = fewrows::Cfg<BN>;
  auto kern = gemm_few_rows_kernel<BN, kConvert>;
  static bool set_on[64] = {false};  // the attribute is per device
  const int dev = device_info().device;
  bool &set = set_on[(dev >= 0 && dev < 64) ? dev : 0];
  if (!set) {
    if (!check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fewrows::MAX_SMEM), "cudaFuncSetAttribute(gemm few rows)"))
      return;
    set = true;
  }
  p.steps = (p.K + C::STAGE_K - 1) / C::STAGE_K;
  p.stages = p.steps < C::stages(p.box_m) ? p.steps : C::stages(p.box_m);  // fewer only where none is used twice
  const size_t smem = static_cast<size_t>(fewrows::fixed_bytes(p.box_m)) + static_cast<size_t>(p.stages) * C::stage_bytes(p.box_m);
  {
    ProfileScope prof(kCatGemm, s);
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>((p.N + BN - 1) / BN)), dim3(fewrows::threads(kConvert)), smem, s, 1, ta, p),
               "launch gemm few rows");
  }
  launched("gemm_few_rows_kernel");
}

void gemm_few_rows(const void *a16, const float *x, const float *w, const float *bias, float *out, int64_t M, int64_t N, int64_t K,
                   cudaStream_t s) {
  const DeviceInfo &di = device_info();
  uint32_t *err = device_error_slot();
  if (!err) return;
  const uint64_t Kp = static_cast<uint64_t>((K + 7) / 8 * 8);
  FewRowsParams p;
  p.x = x, p.w = w, p.bias = bias, p.out = out;
  p.M = static_cast<int>(M), p.N = static_cast<int>(N), p.K = static_cast<int>(K);
  p.box_m = static_cast<int>((M + 7) / 8 * 8);
  p.w_vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
  p.out_vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  p.x_vec = K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  p.err = err;
  CUtensorMap ta = {};
  if (a16 && !encode_tmap_2d(&ta, a16, MGPU_DTYPE_F16, Kp, static_cast<uint64_t>(M), Kp * 2, 64, static_cast<uint32_t>(p.box_m))) return;
  const bool narrow = few_rows_columns(N, di.sms) == 16;
  if (a16) narrow ? launch_few_rows<16, false>(ta, p, s) : launch_few_rows<32, false>(ta, p, s);
  else narrow ? launch_few_rows<16, true>(ta, p, s) : launch_few_rows<32, true>(ta, p, s);
}

}  // namespace mdc
