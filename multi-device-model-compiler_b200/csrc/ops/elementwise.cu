// Entry points for the HBM-bound elementwise ops: Add / bias / activation (fp32), element
// type casts and the one-time weight packing (cast + transpose) for the tensor-core Gemm.
#include <vector>

#include "elementwise_kernels.cuh"
#include "gemm_common.cuh"
#include "ops_common.h"

namespace mdc {

std::atomic<uint64_t> g_launch_count{0};
static std::atomic<uint64_t> g_pack_count{0};

bool pdl_enabled() {
  static const bool on = [] {
    const char *e = getenv("MDC_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

bool g_profiling = false;
namespace {
struct ProfileSpan {
  int cat;
  cudaEvent_t begin, end;
};
std::vector<ProfileSpan> g_spans;
std::vector<cudaEvent_t> g_spare_events;
cudaEvent_t timing_event() {
  if (!g_spare_events.empty()) {
    cudaEvent_t e = g_spare_events.back();
    g_spare_events.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}
}  // namespace

void profile_mark(int category, cudaStream_t stream, bool begin) {
  if (begin) {
    ProfileSpan sp{category, timing_event(), timing_event()};
    cudaEventRecord(sp.begin, stream);
    g_spans.push_back(sp);
  } else if (!g_spans.empty()) {
    cudaEventRecord(g_spans.back().end, stream);
  }
}

const DeviceInfo &device_info() {
  static thread_local DeviceInfo info;
  int dev = -1;
  if (!check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) {
    info = DeviceInfo();
    return info;
  }
  // Everything the runtime library hands out (pool blocks, streams, tensor maps) belongs to the
  // device it selected for this thread; an op queued while another device is current would
  // mix the two.  Refuse instead: devices are chosen with mgpuSetDefaultDevice.
  const int rt_dev = mgpuGetDefaultDevice();
  if (rt_dev >= 0 && rt_dev != dev) {
    char msg[160];
    snprintf(msg, sizeof(msg),
             "the thread's current CUDA device (%d) is not the device the runtime selected for it (%d); "
             "choose devices with mgpuSetDefaultDevice", dev, rt_dev);
    fail(msg);
    info = DeviceInfo();
    return info;
  }
  if (info.ok && info.device == dev) return info;  // cached for the thread's current device
  info = DeviceInfo();
  cudaDeviceProp p;
  if (!check_cuda(cudaGetDeviceProperties(&p, dev), "cudaGetDeviceProperties")) return info;
  info.device = dev;
  info.sms = p.multiProcessorCount;
  info.cc_major = p.major;
  info.cc_minor = p.minor;
  if (p.major != 10) {
    fail("this library is built for sm_100a (Blackwell B200) only");
    return info;
  }
  info.ok = true;
  return info;
}

// ---- casts -------------------------------------------------------------------------
template <typename T>
struct Vec8;  // eight 16-bit elements = 16 bytes
template <>
struct Vec8<__half> {
  __half2 v[4];
};
template <>
struct Vec8<__nv_bfloat16> {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ __half2 pack2(float a, float b, __half) { return __floats2half2_rn(a, b); }
__device__ __forceinline__ __nv_bfloat162 pack2(float a, float b, __nv_bfloat16) {
  return __floats2bfloat162_rn(a, b);
}
__device__ __forceinline__ float2 unpack2(__half2 v) { return __half22float2(v); }
__device__ __forceinline__ float2 unpack2(__nv_bfloat162 v) { return __bfloat1622float2(v); }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f32(float v) { return v; }
template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }

// fp32 -> 16-bit: two float4 in, one 16-byte store out per item.
template <typename T16>
__global__ void __launch_bounds__(kEwBlock)
cast_f32_to_16(const float *__restrict__ src, T16 *__restrict__ dst, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t nthreads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if (aligned16(src) && aligned16(dst)) {
    const int64_t nvec = n >> 3;
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    Vec8<T16> *d8 = reinterpret_cast<Vec8<T16> *>(dst);
    for (int64_t i = tid; i < nvec; i += nthreads) {
      const float4 a = __ldcs(s4 + 2 * i), b = __ldcs(s4 + 2 * i + 1);
      Vec8<T16> o;
      o.v[0] = pack2(a.x, a.y, T16());
      o.v[1] = pack2(a.z, a.w, T16());
      o.v[2] = pack2(b.x, b.y, T16());
      o.v[3] = pack2(b.z, b.w, T16());
      d8[i] = o;
    }
    for (int64_t j = (nvec << 3) + tid; j < n; j += nthreads) dst[j] = from_f32<T16>(src[j]);
  } else {
    for (int64_t j = tid; j < n; j += nthreads) dst[j] = from_f32<T16>(src[j]);
  }
}

template <typename T16>
__global__ void __launch_bounds__(kEwBlock)
cast_16_to_f32(const T16 *__restrict__ src, float *__restrict__ dst, int64_t n) {
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t nthreads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if (aligned16(src) && aligned16(dst)) {
    const int64_t nvec = n >> 3;
    const Vec8<T16> *s8 = reinterpret_cast<const Vec8<T16> *>(src);
    float4 *d4 = reinterpret_cast<float4 *>(dst);
    for (int64_t i = tid; i < nvec; i += nthreads) {
      const Vec8<T16> v = s8[i];
      const float2 a = unpack2(v.v[0]), b = unpack2(v.v[1]), c = unpack2(v.v[2]), d = unpack2(v.v[3]);
      __stcs(d4 + 2 * i, make_float4(a.x, a.y, b.x, b.y));
      __stcs(d4 + 2 * i + 1, make_float4(c.x, c.y, d.x, d.y));
    }
    for (int64_t j = (nvec << 3) + tid; j < n; j += nthreads) dst[j] = to_f32(src[j]);
  } else {
    for (int64_t j = tid; j < n; j += nthreads) dst[j] = to_f32(src[j]);
  }
}

template <typename TS, typename TD>
__global__ void __launch_bounds__(kEwBlock)
cast_generic(const TS *__restrict__ src, TD *__restrict__ dst, int64_t n) {
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t nthreads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t j = tid; j < n; j += nthreads) dst[j] = from_f32<TD>(to_f32(src[j]));
}

// fp32 [R, C] -> 16-bit [R, Cp], columns C..Cp-1 zero (row padding for the Gemm's A operand
// when C is not a multiple of 8).
template <typename T16>
__global__ void __launch_bounds__(kEwBlock)
cast_pad_rows(const float *__restrict__ src, T16 *__restrict__ dst, int64_t R, int64_t C, int64_t Cp) {
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t nthreads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t n = R * Cp;
  for (int64_t j = tid; j < n; j += nthreads) {
    const int64_t r = j / Cp, c = j - r * Cp;
    dst[j] = from_f32<T16>(c < C ? src[r * C + c] : 0.f);
  }
}

// All operands of a call in one launch; a block belongs to one job.
//   cast: kCastItems elements of a contiguous array, or kPadItems of rows that are padded.
//   pack: weight fp32 [K, N] (N contiguous) -> 16-bit [N, Kp] (K contiguous), zero padded to Kp, in tiles of
//         64 x 64.  A lane reads 16 values of its column, all in flight, one line or two per warp and k, and
//         writes one whole sector; through shared memory (16-byte reads, 16-byte writes of eight values)
//         the five operands of an 8 x 256 token layer, 1024 wide, took 2.9 us longer (98.6 -> 95.7 us a call).
// Bound by HBM bytes (6 per element).  One launch instead of one per operand: the tail of one
// job is filled by the next and the launch gaps go: a 1024-wide
// context layer with 2048 tokens (five operands) 130 -> 118 us a call; 35 x 3086 x 3392 Gemm, whose rows
// need padding, 50 -> 38 us (with the one-wave Gemm).
constexpr int64_t kCastItems = OperandList::kCastItems, kPadItems = OperandList::kPadItems;
struct OperandJobs {
  OperandList::Job j[OperandList::kMax];
  int n, late;
};

// kOdd: there is a weight among them whose packed rows are an odd multiple of 16 bytes (compiled apart: it
// costs registers, and 5 % of a 4096 x 1001 weight's time).
template <typename T16, bool kOdd>
__global__ void __launch_bounds__(kEwBlock, 8) prepare_operands_kernel(const OperandJobs jobs) {
  static_assert(kEwBlock == OperandList::kThreads, "the 64 x 64 tiles are walked by 256 threads");
  if (!jobs.late) pdl_launch_dependents();
  pdl_wait();
  if (jobs.late) pdl_launch_dependents();
  OperandList::Job job = jobs.j[0];
#pragma unroll
  for (int i = 1; i < OperandList::kMax; ++i)
    if (i < jobs.n && blockIdx.x >= jobs.j[i].first_block) job = jobs.j[i];
  const int64_t b = blockIdx.x - job.first_block;
  T16 *out = static_cast<T16 *>(job.dst);
  if (job.tiles_n == 0) {
    const int64_t n = job.rows * job.pitch, base = b * (job.vec_ok ? kCastItems : kPadItems);
    if (job.vec_ok) {
      const float4 *s4 = reinterpret_cast<const float4 *>(job.src);
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t i = base + (u * kEwBlock + threadIdx.x) * 8;
        if (i + 7 < n) v[2 * u] = __ldcs(s4 + i / 4), v[2 * u + 1] = __ldcs(s4 + i / 4 + 1);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t i = base + (u * kEwBlock + threadIdx.x) * 8;
        if (i + 7 < n) {
          Vec8<T16> o;
          o.v[0] = pack2(v[2 * u].x, v[2 * u].y, T16());
          o.v[1] = pack2(v[2 * u].z, v[2 * u].w, T16());
          o.v[2] = pack2(v[2 * u + 1].x, v[2 * u + 1].y, T16());
          o.v[3] = pack2(v[2 * u + 1].z, v[2 * u + 1].w, T16());
          *reinterpret_cast<Vec8<T16> *>(out + i) = o;
        } else {
          for (int64_t j = i; j < n; ++j) out[j] = from_f32<T16>(job.src[j]);
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t j = base + u * kEwBlock + threadIdx.x;
        if (j >= n) break;
        const int64_t r = n <= 0x7fffffff ? static_cast<uint32_t>(j) / static_cast<uint32_t>(job.pitch) : j / job.pitch;
        const int64_t c = j - r * job.pitch;
        out[j] = from_f32<T16>(c < job.cols ? job.src[r * job.cols + c] : 0.f);
      }
    }
    return;
  }
  // warp: 32 columns x 16 k, a lane's values one 32-byte sector of its column's packed row
  const int64_t K = job.rows, N = job.cols, Kp = job.pitch;
  const uint32_t b32 = static_cast<uint32_t>(b), tk = b32 / static_cast<uint32_t>(job.tiles_n);
  const int64_t k0 = static_cast<int64_t>(tk) * 64 + (threadIdx.x >> 6) * 16;
  const int64_t n = static_cast<int64_t>(b32 - tk * job.tiles_n) * 64 + (threadIdx.x & 63);
  const bool odd_pitch = kOdd && Kp % 16 != 0;
  if (!odd_pitch && (n >= N || k0 >= Kp)) return;
  const float *w = job.src + k0 * N + n;
  int live = K - k0 < 16 ? static_cast<int>(K - k0) : 16;  // at most 0 in the padding
  const int room = !kOdd ? 16 : n >= N ? 0 : Kp - k0 < 16 ? static_cast<int>(Kp - k0) : 16;  // of an odd row: 16, 8 or none
  if (kOdd && room <= 0) live = 0;
  float v[16];
  if (live == 16) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __ldcs(w + j * N);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = j < live ? __ldcs(w + j * N) : 0.f;
  }
  uint32_t o[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = pack_pair<T16>(v[2 * e], v[2 * e + 1]);
  T16 *dst = out + n * Kp + k0;
  const uint4 lo = make_uint4(o[0], o[1], o[2], o[3]), hi = make_uint4(o[4], o[5], o[6], o[7]);
  if (!odd_pitch) {
    if (job.vec_ok) {
      st_global_32B(dst, o);
    } else {
      *reinterpret_cast<uint4 *>(dst) = lo;
      *reinterpret_cast<uint4 *>(dst + 8) = hi;
    }
    return;
  }
  // Every second row starts inside a sector.  Its groups hand their upper halves on, so that these rows too are
  // written in whole sectors but for the ends of the tile.  With half sectors throughout 2048 x 1024 x 1000 took
  // 22.1 us a call (20.4 now) and 3000 x 3000 x 3000 72.8 (71.9), the latter's conversion by itself 23.0 (21.0).
  // Lanes of such rows reading 8 k further down instead: the weight alone as fast, but the calls 21.0 and 78 us one
  // after another, as lines that two lanes share did not stay in what L1 the Gemm ahead left.
  __shared__ uint4 upper[4][32];  // of two neighbouring columns one has such a row
  uint4 *mine = &upper[threadIdx.x >> 6][(threadIdx.x & 63) >> 1];
  const bool in_sector = (reinterpret_cast<uintptr_t>(dst) & 31u) != 0;
  if (in_sector) *mine = hi;
  __syncthreads();
  if (room <= 0) return;
  if (!in_sector) {
    if (room == 16) st_global_32B(dst, o);
    else *reinterpret_cast<uint4 *>(dst) = lo;
    return;
  }
  if (threadIdx.x >= 64) {
    const uint4 before = *(mine - 32);
    const uint32_t q[8] = {before.x, before.y, before.z, before.w, lo.x, lo.y, lo.z, lo.w};
    st_global_32B(dst - 8, q);
  } else {
    *reinterpret_cast<uint4 *>(dst) = lo;
  }
  if (threadIdx.x >= 192 && room == 16) *reinterpret_cast<uint4 *>(dst + 8) = hi;
}

void OperandList::launch(int32_t dtype, void *stream, bool late) {
  if (n == 0) return;
  if (overflow || blocks > 0x7fffffff) {
    fail(overflow ? "operand conversion: more operands than a call may have" : "operand conversion: shape too large");
    clear();
    return;
  }
  OperandJobs a;
  for (int i = 0; i < kMax; ++i) a.j[i] = jobs[i < n ? i : 0];
  a.n = n, a.late = late ? 1 : 0;
  cudaStream_t s = as_stream(stream);
  ProfileScope prof(kCatElementwise, s);
  bool odd = false;
  uint64_t packs = 0;
  for (int i = 0; i < n; ++i)
    if (jobs[i].tiles_n != 0) ++packs, odd |= jobs[i].pitch % 16 != 0;
  g_pack_count.fetch_add(packs, std::memory_order_relaxed);
  auto launch = [&](auto kern) {
    check_cuda(launch_chain(kern, dim3(static_cast<unsigned>(blocks)), dim3(kEwBlock), 0, s, 1, a), "launch prepare_operands");
  };
  if (dtype == MGPU_DTYPE_F16) odd ? launch(prepare_operands_kernel<__half, true>) : launch(prepare_operands_kernel<__half, false>);
  else odd ? launch(prepare_operands_kernel<__nv_bfloat16, true>) : launch(prepare_operands_kernel<__nv_bfloat16, false>);
  launched("mdc_prepare_operands");
  clear();
}

}  // namespace mdc

using namespace mdc;

MDC_API uint64_t mgpuOpsLaunchCount(void) { return g_launch_count.load(); }
MDC_API uint64_t mgpuOpsWeightPackCount(void) { return g_pack_count.load(); }

MDC_API void mgpuOpsProfileBegin(void) {
  g_spans.clear();
  g_profiling = true;
}

// Like mgpuOpsProfileEnd, but returns every launch separately, in launch order: its
// category and its device time.  Returns the number of launches written (at most `capacity`).
MDC_API int64_t mgpuOpsProfileEndSpans(int32_t *category, float *ms, int64_t capacity) {
  g_profiling = false;
  int64_t n = 0;
  for (ProfileSpan &sp : g_spans) {
    float t = 0.f;
    if (cudaEventSynchronize(sp.end) == cudaSuccess && cudaEventElapsedTime(&t, sp.begin, sp.end) == cudaSuccess) {
      if (n < capacity) {
        if (category) category[n] = sp.cat;
        if (ms) ms[n] = t;
        ++n;
      }
    } else {
      (void)cudaGetLastError();
    }
    g_spare_events.push_back(sp.begin);
    g_spare_events.push_back(sp.end);
  }
  g_spans.clear();
  return n;
}

MDC_API void mgpuOpsProfileEnd(double *ms_per_category, uint64_t *launches_per_category) {
  g_profiling = false;
  for (int c = 0; c < kNumCategories; ++c) {
    if (ms_per_category) ms_per_category[c] = 0.0;
    if (launches_per_category) launches_per_category[c] = 0;
  }
  for (ProfileSpan &sp : g_spans) {
    float ms = 0.f;
    if (cudaEventSynchronize(sp.end) == cudaSuccess && cudaEventElapsedTime(&ms, sp.begin, sp.end) == cudaSuccess) {
      if (ms_per_category) ms_per_category[sp.cat] += ms;
      if (launches_per_category) launches_per_category[sp.cat] += 1;
    } else {
      (void)cudaGetLastError();
    }
    g_spare_events.push_back(sp.begin);
    g_spare_events.push_back(sp.end);
  }
  g_spans.clear();
}

MDC_API void mgpuAdd(const float *a, const float *b, float *c, int64_t n, void *stream) {
  if (n <= 0) return;
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  ProfileScope prof(kCatElementwise, as_stream(stream));
  check_cuda(launch_chain(mdc_add_f32, dim3(ew_grid((n + 3) / 4, di.sms)), dim3(kEwBlock), 0, as_stream(stream), 1, a, b, c, n), "launch add");
  launched("mdc_add_f32");
}

MDC_API void mgpuBiasAdd(const float *x, const float *bias, float *y, int64_t rows, int64_t cols,
                         void *stream) {
  if (rows <= 0 || cols <= 0) return;
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  check_cuda(launch_chain(mdc_bias_add_f32, dim3(ew_grid((rows * cols + 3) / 4, di.sms)), dim3(kEwBlock), 0, as_stream(stream), 1,
                          x, bias, y, rows, cols), "launch bias add");
  launched("mdc_bias_add_f32");
}

MDC_API void mgpuActivation(const float *x, float *y, int64_t n, int32_t act, void *stream) {
  if (n <= 0) return;
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  const int grid = ew_grid((n + 3) / 4, di.sms);
  cudaStream_t s = as_stream(stream);
  switch (act) {
  case MGPU_ACT_RELU:
    check_cuda(launch_chain(mdc_relu_f32, dim3(grid), dim3(kEwBlock), 0, s, 1, x, y, n), "launch activation");
    break;
  case MGPU_ACT_GELU_ERF:
    check_cuda(launch_chain(mdc_gelu_erf_f32, dim3(grid), dim3(kEwBlock), 0, s, 1, x, y, n), "launch activation");
    break;
  case MGPU_ACT_GELU_TANH:
    check_cuda(launch_chain(mdc_gelu_tanh_f32, dim3(grid), dim3(kEwBlock), 0, s, 1, x, y, n), "launch activation");
    break;
  case MGPU_ACT_NONE:
    if (x != y) check_cuda(cudaMemcpyAsync(y, x, n * sizeof(float), cudaMemcpyDeviceToDevice, s), "copy");
    return;
  default:
    fail("mgpuActivation: unknown activation");
    return;
  }
  launched("mdc_activation");
}

MDC_API void mgpuCast(const void *src, int32_t sd, void *dst, int32_t dd, int64_t n, void *stream) {
  if (n <= 0) return;
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  cudaStream_t s = as_stream(stream);
  const int grid = ew_grid((n + 7) / 8, di.sms);
  ProfileScope prof(kCatElementwise, s);
  if (sd == dd) {
    if (src != dst)
      check_cuda(cudaMemcpyAsync(dst, src, n * dtype_size(sd), cudaMemcpyDeviceToDevice, s), "copy");
    return;
  }
  if (sd == MGPU_DTYPE_F32 && dd == MGPU_DTYPE_F16)
    check_cuda(launch_chain(cast_f32_to_16<__half>, dim3(grid), dim3(kEwBlock), 0, s, 1, (const float *)src, (__half *)dst, n), "launch cast");
  else if (sd == MGPU_DTYPE_F32 && dd == MGPU_DTYPE_BF16)
    check_cuda(launch_chain(cast_f32_to_16<__nv_bfloat16>, dim3(grid), dim3(kEwBlock), 0, s, 1, (const float *)src, (__nv_bfloat16 *)dst, n), "launch cast");
  else if (sd == MGPU_DTYPE_F16 && dd == MGPU_DTYPE_F32)
    cast_16_to_f32<__half><<<grid, kEwBlock, 0, s>>>((const __half *)src, (float *)dst, n);
  else if (sd == MGPU_DTYPE_BF16 && dd == MGPU_DTYPE_F32)
    cast_16_to_f32<__nv_bfloat16><<<grid, kEwBlock, 0, s>>>((const __nv_bfloat16 *)src, (float *)dst, n);
  else if (sd == MGPU_DTYPE_F16 && dd == MGPU_DTYPE_BF16)
    cast_generic<__half, __nv_bfloat16><<<grid, kEwBlock, 0, s>>>((const __half *)src, (__nv_bfloat16 *)dst, n);
  else if (sd == MGPU_DTYPE_BF16 && dd == MGPU_DTYPE_F16)
    cast_generic<__nv_bfloat16, __half><<<grid, kEwBlock, 0, s>>>((const __nv_bfloat16 *)src, (__half *)dst, n);
  else {
    fail("mgpuCast: unknown element type");
    return;
  }
  launched("mdc_cast");
}

namespace mdc {
// fp32 [R,C] -> 16-bit [R,Cp]; plain cast when C == Cp.
void cast_rows_padded(const float *src, void *dst, int64_t R, int64_t C, int64_t Cp, int32_t dtype,
                      cudaStream_t s) {
  if (C == Cp) {
    mgpuCast(src, MGPU_DTYPE_F32, dst, dtype, R * C, s);
    return;
  }
  const DeviceInfo &di = device_info();
  if (!di.ok) return;
  const int grid = ew_grid(R * Cp, di.sms);
  if (dtype == MGPU_DTYPE_F16)
    cast_pad_rows<__half><<<grid, kEwBlock, 0, s>>>(src, (__half *)dst, R, C, Cp);
  else
    cast_pad_rows<__nv_bfloat16><<<grid, kEwBlock, 0, s>>>(src, (__nv_bfloat16 *)dst, R, C, Cp);
  launched("mdc_cast_pad_rows");
}
}  // namespace mdc

MDC_API void mgpuPackWeight(const float *w, void *packed, int64_t K, int64_t N, int32_t dtype,
                            void *stream) {
  if (K <= 0 || N <= 0) return;
  if (!dtype_is16(dtype)) {
    fail("mgpuPackWeight: dtype must be F16 or BF16");
    return;
  }
  if (!device_info().ok) return;
  if (reinterpret_cast<uintptr_t>(packed) & 15u) { fail("mgpuPackWeight: the packed buffer must be 16-byte aligned"); return; }
  OperandList list;
  list.pack(w, packed, K, N);
  list.launch(dtype, stream);
}
