// Shared helpers for the sm_100a kernels of the quantized-linear path.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/xqt_b200.h"

namespace xqt_b200 {

// Every entry point returns a cudaError_t as int, cudaErrorInvalidValue for a
// request it cannot serve; nothing is thrown across the C boundary.
#define XQT_REQUIRE(cond)                        \
  do {                                           \
    if (!(cond)) return (int)cudaErrorInvalidValue; \
  } while (0)

#define XQT_CUDA(call)                           \
  do {                                           \
    cudaError_t err__ = (call);                  \
    if (err__ != cudaSuccess) return (int)err__; \
  } while (0)

inline int launch_status() { return (int)cudaGetLastError(); }

// Opt a kernel in to more than 48 KiB of dynamic shared memory.  The attribute belongs to the
// (function, device) pair, so it is set once per device the process launches on, with that device
// current.
#define XQT_SMEM_OPT_IN(kern, bytes)                                                                    \
  do {                                                                                                  \
    static bool configured__[64] = {};                                                                  \
    int dev__ = 0;                                                                                      \
    XQT_CUDA(cudaGetDevice(&dev__));                                                                    \
    if (dev__ < 0 || dev__ >= 64 || !configured__[dev__]) {                                             \
      XQT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes)));  \
      if (dev__ >= 0 && dev__ < 64) configured__[dev__] = true;                                         \
    }                                                                                                   \
  } while (0)

// SMs of the current device, asked for once per device (the query costs about 0.2 us of host time per launch).
inline int sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    cached[dev] = v;
  }
  return cached[dev];
}

// Launch with programmatic stream serialisation: the kernel may start while the one before it in the stream drains.  It
// has to execute griddepcontrol.wait (in every CTA) before it touches memory that an earlier kernel writes or reads, unless the
// caller vouches that it was complete before the launch.
template <typename... Params, typename... Args>
inline int launch_pdl_cluster(void (*kern)(Params...), dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  XQT_CUDA(cudaLaunchKernelEx(&cfg, kern, Params(args)...));
  return launch_status();
}
template <typename... Params, typename... Args>
inline int launch_pdl(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_pdl_cluster(kern, grid, block, 1, smem, stream, args...);
}

// Clusters of two CTAs of `Kern` that are resident together with a CTA per SM, asked for once per kernel and device.
template <auto Kern>
inline int resident_pairs(int threads, size_t smem) {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() / 2;
  if (cached[dev] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() & ~1));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int v = 0;
    if (cudaOccupancyMaxActiveClusters(&v, Kern, &cfg) != cudaSuccess || v <= 0) v = sm_count() / 2;
    cached[dev] = v < sm_count() / 2 ? v : sm_count() / 2;
  }
  return cached[dev];
}

__host__ __device__ constexpr int ceil_div(int a, int b) { return (a + b - 1) / b; }

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Read element i of a scale / zero-point array whose dtype is only known at run
// time (fp16, bf16 or fp32, XQT_B200_FP16/BF16/FP32).
__device__ __forceinline__ float load_param(const void* base, int dtype, size_t i) {
  if (dtype == XQT_B200_FP32) return reinterpret_cast<const float*>(base)[i];
  if (dtype == XQT_B200_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[i]);
  return __half2float(reinterpret_cast<const __half*>(base)[i]);
}

// The same in two steps, so that a prefetch does not wait for its own data: the raw bits now, the value when needed.
__device__ __forceinline__ uint32_t load_param_bits(const void* base, int dtype, size_t i) {
  if (dtype == XQT_B200_FP32) return reinterpret_cast<const uint32_t*>(base)[i];
  return reinterpret_cast<const unsigned short*>(base)[i];
}
__device__ __forceinline__ float param_from_bits(uint32_t bits, int dtype) {
  if (dtype == XQT_B200_FP32) return __uint_as_float(bits);
  if (dtype == XQT_B200_BF16) return __uint_as_float(bits << 16);
  return __half2float(__ushort_as_half((unsigned short)bits));
}

__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + __expf(-v)); }

}  // namespace xqt_b200
