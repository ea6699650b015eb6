// Shared helpers for the sm_100a kernel library: error reporting, dtype
// dispatch and scalar load/store with conversion.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "xdlb200.h"

namespace xb {

// Thread-local reason of the last rejected call (returned by xb_last_error()).
int fail(int code, const char* fmt, ...);
void clear_error();

#define XB_REQUIRE(cond, code, ...)              \
  do {                                           \
    if (!(cond)) return xb::fail(code, __VA_ARGS__); \
  } while (0)

#define XB_CUDA(call)                                                            \
  do {                                                                           \
    cudaError_t e__ = (call);                                                    \
    if (e__ != cudaSuccess)                                                      \
      return xb::fail(XB_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e__)); \
  } while (0)

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(XB_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
  return 0;
}

inline size_t dtype_size(int dt) {
  switch (dt) {
    case XB_F32: case XB_I32: return 4;
    case XB_I64: return 8;
    case XB_F16: case XB_BF16: return 2;
    default: return 0;
  }
}

// Programmatic dependent launch: a kernel launched with launch_dependent may begin while the kernel before it in the stream
// still runs, as soon as every block of that one has released it (pdl_release) or ended. pdl_wait waits until the kernel
// before has completed and its writes are visible; what stands above it (barriers, tensor memory) and the launch itself
// overlap the tail of the kernel before. The rules, for every kernel launched so:
//  - Every thread passes pdl_wait, before its first access to global memory and before any exit. A kernel that could end
//    without having waited would let the kernel after the next one start on data that are not there yet.
//  - pdl_release comes after the kernel's own tensor memory has been allocated. A kernel that allocates above its pdl_wait
//    holds columns while it waits; if the kernel it waits for still had to allocate, neither would go on.
//  - A kernel that runs for long releases late (or not at all: its end does). Blocks that wait for it hold registers and
//    shared memory that the kernels of other streams could run on. Two streams of 74 DIN requests: 365 us a step with every
//    release at the kernel's beginning, 351 with those of the tensor-core kernels and recurrences at their end; one stream
//    348 and 345. Short kernels use pdl_begin.
// One pooling call after another (10 240 lists): 14.3 -> 11.1 us; DIN on 2 tiles: 48 -> 43; DIEN on 128 tiles: 370 -> 360.
template <typename... KArgs, typename... Args>
inline void launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = at; cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);       // an error is found by check_launch
}
__device__ __forceinline__ void pdl_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void pdl_release() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_release();
}

// Number of SMs of the current device (cached per device).
int sm_count();

// A launch attribute such as cudaFuncAttributeMaxDynamicSharedMemorySize belongs to one device, and one process
// may serve several (one workspace per device, blaze/blaze/api/cpp_api/predictor_manager_impl.cc:142-177): this
// remembers, per launcher, on which devices the attribute was set. Safe for concurrent serving threads: two
// threads that both find the bit clear both set the (idempotent) attribute.
struct PerDeviceOnce {
  std::atomic<uint64_t> bits{0};
  // true when the caller still has to do the set-up on the current device (ordinal above 63: always)
  bool needed(int* dev) {
    *dev = 0;
    if (cudaGetDevice(dev) != cudaSuccess || *dev < 0 || *dev >= 64) { *dev = -1; return true; }
    return ((bits.load(std::memory_order_acquire) >> *dev) & 1u) == 0;
  }
  void done(int dev) {
    if (dev >= 0) bits.fetch_or(uint64_t(1) << dev, std::memory_order_release);
  }
};
#define XB_SET_MAX_SMEM_ONCE(once, bytes, ...)                                                        \
  do {                                                                                                \
    int dev__;                                                                                        \
    if ((once).needed(&dev__)) {                                                                      \
      const void* fns__[] = {__VA_ARGS__};                                                            \
      for (const void* f__ : fns__)                                                                   \
        XB_CUDA(cudaFuncSetAttribute(f__, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))); \
      (once).done(dev__);                                                                             \
    }                                                                                                 \
  } while (0)

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Load/store through a runtime dtype (used by the low-rate glue kernels).
__device__ __forceinline__ float load_as_f32(const void* p, int64_t i, int dt) {
  if (dt == XB_F32) return reinterpret_cast<const float*>(p)[i];
  if (dt == XB_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  if (dt == XB_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  if (dt == XB_I32) return (float)reinterpret_cast<const int32_t*>(p)[i];
  return 0.f;
}
__device__ __forceinline__ void store_from_f32(void* p, int64_t i, int dt, float v) {
  if (dt == XB_F32) reinterpret_cast<float*>(p)[i] = v;
  else if (dt == XB_F16) reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
  else if (dt == XB_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else if (dt == XB_I32) reinterpret_cast<int32_t*>(p)[i] = (int32_t)v;
}

// Activation epilogues, restating blaze/blaze/math/activation.h:36-68.
struct EpiParams {
  int kind;            // XB_EPI_*
  const float* a;      // prelu slopes / dice gamma
  const float* b;      // dice mean
  const float* c;      // dice var
  int count;           // prelu slope count
  int nosqrt;
};

__device__ __forceinline__ float dice_rstd(float var, int nosqrt) {
  return nosqrt ? 1.f / var : 1.f / sqrtf(var + 1e-8f);
}
__device__ __forceinline__ float act_dice(float x, float gamma, float mean, float rstd) {
  float p = 1.f / (1.f + __expf(-(x - mean) * rstd));
  return (1.f - p) * gamma * x + p * x;
}
__device__ __forceinline__ float act_prelu(float x, float w) {
  return x * ((x > 0.f ? 1.f : 0.f) + (x < 0.f ? w : 0.f));
}
__device__ __forceinline__ float act_sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }

}  // namespace xb
