// Shared host-side helpers of the operator library: status reporting through the runtime
// library's sticky error, launch accounting, device queries and the element-type enum.
#pragma once

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "mdc_gpu_ops.h"
#include "mdc_gpu_runtime.h"
#include "operand_list.h"
#ifdef __CUDACC__
#include "pdl.cuh"
#endif

#define MDC_API extern "C" __attribute__((visibility("default")))
#define MDC_CXX_API __attribute__((visibility("default")))

namespace mdc {

extern std::atomic<uint64_t> g_launch_count;

inline bool check_cuda(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return true;
  char msg[256];
  snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorName(e));
  mgpuSetLastError(static_cast<int32_t>(e), msg);
  (void)cudaGetLastError();
  return false;
}

inline void fail(const char *what) { mgpuSetLastError(-1, what); }

// Call after every <<<>>> launch: counts it and turns a launch failure into the status.
inline bool launched(const char *what) {
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return check_cuda(cudaGetLastError(), what);
}

struct DeviceInfo {
  int device = -1;
  int sms = 0;
  int cc_major = 0, cc_minor = 0;
  bool ok = false;
};
// Properties of the current device; ok == false (with the status set) if there is no
// usable CUDA device or it is not compute capability 10.x.
const DeviceInfo &device_info();

inline size_t dtype_size(int32_t dtype) { return dtype == MGPU_DTYPE_F32 ? 4 : 2; }
inline bool dtype_is16(int32_t dtype) { return dtype == MGPU_DTYPE_F16 || dtype == MGPU_DTYPE_BF16; }

inline cudaStream_t as_stream(void *s) { return static_cast<cudaStream_t>(s); }

// Launch helper for the kernels of the layer chain.  With programmatic dependent launch the
// front end may set the next kernel up (and start its CTAs on SMs the previous kernel has
// already left) while the previous kernel drains; each such kernel calls pdl_wait() (device,
// pdl.cuh) before it touches global memory, which orders it after the whole
// previous grid.  Three kernels read ahead of their wait.  The one-wave Gemm: weights that the host knows to be complete
// (w_ready).  gemm_few_rows behind a conversion, and conv_halo_kernel behind the packing of its filter where it makes no copy:
// what is older than that launch (the weight; input, bias and residual), because it triggers only after its own wait.
// MDC_PDL=0 turns the attribute off (plain stream order).
bool pdl_enabled();
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                int cluster_x, Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attrs[2];
  unsigned n = 0;
  if (pdl_enabled()) {
    attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster_x > 1) {
    attrs[n].id = cudaLaunchAttributeClusterDimension;
    attrs[n].val.clusterDim.x = static_cast<unsigned>(cluster_x);
    attrs[n].val.clusterDim.y = 1;
    attrs[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// A tiled tensor map of fp16, bf16 or fp32 elements; dim and box innermost first, stride in bytes from the second dimension
// on.  False where it is not encoded, by this call's own verdict, whatever the status says; the status then says so, unless
// the caller has another way (`report` false).
inline bool encode_tmap(CUtensorMap *map, int32_t dtype, uint32_t rank, const void *base, const uint64_t *dim,
                        const uint64_t *stride, const uint32_t *box, CUtensorMapSwizzle swizzle, bool report = true) {
  const uint32_t ones[5] = {1, 1, 1, 1, 1};
  const int type = dtype == MGPU_DTYPE_BF16  ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                   : dtype == MGPU_DTYPE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                             : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const int32_t e = mgpuTensorMapTryEncodeTiled(map, type, rank, const_cast<void *>(base), dim, stride, box, ones,
                                                CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (e != 0 && report) mgpuSetLastError(e, "cuTensorMapEncodeTiled");
  return e == 0;
}
// The same for rows of a matrix, 128-byte swizzled.
inline bool encode_tmap_2d(CUtensorMap *map, const void *base, int32_t dtype, uint64_t inner, uint64_t outer,
                           uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, bool report = true) {
  const uint64_t dim[2] = {inner, outer};
  const uint32_t box[2] = {box_inner, box_outer};
  return encode_tmap(map, dtype, 2, base, dim, &row_stride_bytes, box, CU_TENSOR_MAP_SWIZZLE_128B, report);
}

// Optional per-launch timing: while profiling is on (mgpuOpsProfileBegin), every launch
// site brackets its kernel with two CUDA events on the launching stream; mgpuOpsProfileEnd
// sums the elapsed times per kernel category.  Off by default (no events, no overhead).
enum ProfileCategory : int { kCatGemm = 0, kCatAttention = 1, kCatLayerNorm = 2, kCatElementwise = 3, kNumCategories = 4 };
extern bool g_profiling;
void profile_mark(int category, cudaStream_t stream, bool begin);
struct ProfileScope {
  int cat;
  cudaStream_t stream;
  ProfileScope(int c, cudaStream_t s) : cat(c), stream(s) {
    if (g_profiling) profile_mark(cat, stream, true);
  }
  ~ProfileScope() {
    if (g_profiling) profile_mark(cat, stream, false);
  }
};

// fp32 [R, C] -> 16-bit [R, Cp] with zero padding of the columns C..Cp (elementwise.cu)
void cast_rows_padded(const float *src, void *dst, int64_t R, int64_t C, int64_t Cp, int32_t dtype, cudaStream_t s);

// mgpuMatmulEx16; w_ready: the weight was complete before this call (it does not come from a kernel
// still queued), so the kernel may read it ahead of its dependency on the previous one.
void matmul16(const void *a, const void *w_nk, const float *bias, const void *residual, void *out, int64_t M, int64_t N,
              int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act, bool w_ready, void *stream);

// Packed 16-bit [N, Kp] form of an fp32 [K, N] weight, from the constant cache when the weight
// is a copy of a registered constant (defined in ops_init.cu).  A weight that is not is added to
// `list`; it is packed once that is launched.
void *packed_weight(const float *w, int64_t K, int64_t N, int32_t dtype, void *stream, bool *cached, OperandList *list);

// Device slot the tensor-core kernels write a non-zero code into when one of their bounded
// waits gives up; checked (and turned into the status) by mgpuOpsCheckDeviceStatus().
uint32_t *device_error_slot();

}  // namespace mdc

// Reads the device error slot (synchronises the stream); 0 = no kernel reported a problem.
MDC_API uint32_t mgpuOpsCheckDeviceStatus(void *stream);
