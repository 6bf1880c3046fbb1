// Device helpers shared by the memory-bound kernels: warp/block reductions, typed loads/stores,
// grid sizing.  Parity: src/cuda/common.cuh:30-137 of the reference (warp_sum/block_sum,
// blocks_for, Num<T> load/store); written for 32-wide warps only.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "once_per_device.h"

namespace nx {

constexpr int kNumSmsB200 = 148;

// Lets a following kernel that was launched with the programmatic-serialization attribute (the tensor-core GEMM)
// begin its prologue early; that kernel still waits for this grid to complete before it reads anything.  A no-op
// when the next launch is an ordinary one.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The other side: blocks until the grids in front have completed and their memory is visible.  A kernel launched by `launch_pdl`
// passes this before it touches anything that a kernel in front may have written, and before its own first write.
__device__ __forceinline__ void pdl_dependency() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A launch that may begin while the kernel in front of it drains (its blocks are placed and its constants set up by then): in a
// chain of short kernels, as decoding is, about half a microsecond per launch.  For kernels that call `pdl_dependency` only.
template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...) == cudaSuccess) return 0;
  (void)cudaGetLastError();
  return -2;
}
// Allows a kernel `bytes` of dynamic shared memory on the current device, once; in a function that returns 0 or an error:
// NX_ALLOW_SMEM((kernel), bytes)
template <typename... KArgs>
inline int allow_smem(OncePerDevice& once, void (*kern)(KArgs...), int bytes) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -2;
  return once(dev, [&](int) { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : -2; });
}
#define NX_ALLOW_SMEM(KERN_, BYTES_)                               \
  do {                                                             \
    static ::nx::OncePerDevice nx_once;                            \
    if (::nx::allow_smem(nx_once, KERN_, BYTES_) != 0) return -2;  \
  } while (0)
// The launch in a function that returns 0 or an error: NX_PDL((kernel), grid, threads, shared memory, stream, arguments ...)
#define NX_PDL(KERN_, GRID_, BLOCK_, SMEM_, ST_, ...)                                                  \
  do {                                                                                                 \
    if (::nx::launch_pdl(KERN_, dim3(GRID_), dim3(BLOCK_), SMEM_, ST_, __VA_ARGS__) != 0) return -2;    \
  } while (0)

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide reductions; `scratch` holds 32 values of T in shared memory.  Every thread gets the
// result.  Safe to call repeatedly with the same scratch.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  T r = (lane < nwarps) ? scratch[lane] : T(0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = (lane < nwarps) ? scratch[lane] : -INFINITY;
  return warp_max(r);
}

inline int blocks_for(int64_t n, int threads, int max_blocks = kNumSmsB200 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return static_cast<int>(b);
}

#define NX_GRID_STRIDE(i, n)                                                                       \
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < (n);          \
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)

template <typename T>
struct Num;
template <>
struct Num<float> {
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
};
template <>
struct Num<__nv_bfloat16> {
  static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
};
template <>
struct Num<__half> {
  static __device__ __forceinline__ float load(const __half* p) { return __half2float(*p); }
  static __device__ __forceinline__ void store(__half* p, float v) { *p = __float2half_rn(v); }
};

// dtype codes follow NxDType in nx_api.h: 0 bf16, 1 f32, 2 f16.
__device__ __forceinline__ float load_as_float(const void* base, int dtype, int64_t i) {
  if (dtype == 1) return reinterpret_cast<const float*>(base)[i];
  if (dtype == 0) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[i]);
  return __half2float(reinterpret_cast<const __half*>(base)[i]);
}
__device__ __forceinline__ void store_from_float(void* base, int dtype, int64_t i, float v) {
  if (dtype == 1)
    reinterpret_cast<float*>(base)[i] = v;
  else if (dtype == 0)
    reinterpret_cast<__nv_bfloat16*>(base)[i] = __float2bfloat16_rn(v);
  else
    reinterpret_cast<__half*>(base)[i] = __float2half_rn(v);
}

inline int launch_status() { return cudaGetLastError() == cudaSuccess ? 0 : -2; }

}  // namespace nx
