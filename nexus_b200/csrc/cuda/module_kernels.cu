// Elementwise passes of the autograd operators: backward of an activation, the product with a scalar that lives on the device,
// rotary embedding of the queries and keys inside packed rows.  All bound by memory; 16 bytes per access, one launch where the
// tensor library took a chain of conversions and FP32 copies (activation backward: 6 launches; rotation of queries and keys:
// 10 forward and 14 backward).
#include "common.cuh"
#include "nx_api_kernels.h"
#include "sm100_ptx.cuh"

#include <algorithm>

namespace {
using namespace nx;

template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = Num<T>::load(e + j);
  }
}
template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint4 q;
    T* e = reinterpret_cast<T*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) Num<T>::store(e + j, v[j]);
    *reinterpret_cast<uint4*>(p) = q;
  }
}

// FP32 to the last bits: the pass is bound by memory, the approximate forms of the GEMM epilogues (tanh to 5e-4) would only lose
// them.  GELU: t = sigmoid(2 u) = (1 + tanh u) / 2, so that 1 - tanh^2 u = 4 t (1 - t) has no cancellation.
__device__ __forceinline__ float sigmoid_exact(float x) { return __fdividef(1.0f, 1.0f + expf(-x)); }
__device__ __forceinline__ float act_grad(float x, float dy, int act) {
  if (act == NX_ACT_GELU) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f, x2 = x * x;
    const float t = sigmoid_exact(2.0f * k0 * (x + k1 * x * x2));
    return dy * (t + 2.0f * x * t * (1.0f - t) * k0 * (1.0f + 3.0f * k1 * x2));
  }
  if (act == NX_ACT_SILU) {
    const float s = sigmoid_exact(x);
    return dy * (s * (1.0f + x * (1.0f - s)));
  }
  return x <= 0.0f ? 0.0f : dy;  // relu
}

// out = dy * act'(x); `vec` pieces of eight, then single elements
template <typename T>
__global__ void __launch_bounds__(256) act_bwd_kernel(const T* __restrict__ x, const T* __restrict__ dy, T* __restrict__ out, int64_t n,
                                                      int64_t vec, int act) {
  pdl_trigger();
  NX_GRID_STRIDE(i, vec) {
    float a[8], d[8];
    load8(x + i * 8, a);
    load8(dy + i * 8, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = act_grad(a[j], d[j], act);
    store8(out + i * 8, d);
  }
  for (int64_t i = vec * 8 + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    Num<T>::store(out + i, act_grad(Num<T>::load(x + i), Num<T>::load(dy + i), act));
}

// out = in * (*factor)
template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(const T* __restrict__ in, const float* __restrict__ factor, T* __restrict__ out, int64_t n,
                                                    int64_t vec) {
  pdl_trigger();
  const float f = *factor;
  NX_GRID_STRIDE(i, vec) {
    float a[8];
    load8(in + i * 8, a);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] *= f;
    store8(out + i * 8, a);
  }
  for (int64_t i = vec * 8 + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    Num<T>::store(out + i, Num<T>::load(in + i) * f);
}

// Rotate-half embedding of the first `heads` heads of every row; position of row r: r % seq_len.  Columns past 2 * half are
// copied.  A piece: eight elements of the first half and the eight they turn with, or eight copied ones.  x and y may be the
// same rows.
__global__ void __launch_bounds__(256) rope_rows_kernel(const __nv_bfloat16* x, int64_t ldx, __nv_bfloat16* y, int64_t ldy,
                                                        const float* __restrict__ cos_t, const float* __restrict__ sin_t, int rows, int seq_len,
                                                        int heads, int D, int half, float sign) {
  pdl_trigger();
  const uint32_t turn = half >> 3, per = turn + ((D - 2 * half) >> 3), row_pieces = per * heads;
  const uint32_t total = row_pieces * static_cast<uint32_t>(rows);
  for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < total; i += gridDim.x * 256u) {
    const uint32_t r = i / row_pieces, in_row = i - r * row_pieces, h = in_row / per, j = in_row - h * per;
    const __nv_bfloat16* xr = x + r * ldx + h * D;
    __nv_bfloat16* yr = y + r * ldy + h * D;
    if (j >= turn) {
      const int c = 2 * half + (j - turn) * 8;
      *reinterpret_cast<uint4*>(yr + c) = *reinterpret_cast<const uint4*>(xr + c);
      continue;
    }
    const int64_t at = static_cast<int64_t>(r % static_cast<uint32_t>(seq_len)) * half + j * 8;
    float a[8], b[8], c[8], s[8], o[8];
    load8(xr + j * 8, a);
    load8(xr + half + j * 8, b);
    load8(cos_t + at, c);
    load8(sin_t + at, s);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      s[e] *= sign;
      // products and sums rounded one by one, as the chain of FP32 operators does: the same bits
      o[e] = __fsub_rn(__fmul_rn(a[e], c[e]), __fmul_rn(b[e], s[e]));
      b[e] = __fadd_rn(__fmul_rn(b[e], c[e]), __fmul_rn(a[e], s[e]));
    }
    store8(yr + j * 8, o);
    store8(yr + half + j * 8, b);
  }
}

bool on16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

}  // namespace

extern "C" int nx_act_bwd(const void* x, const void* dy, void* out, int dtype, int64_t n, int act, nx_stream_t stream) {
  if (n <= 0) return n == 0 ? 0 : -1;
  if (act != NX_ACT_GELU && act != NX_ACT_SILU && act != NX_ACT_RELU) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t vec = on16(x, dy, out) ? n / 8 : 0;
  const int blocks = blocks_for(vec > 0 ? vec : n, 256);
#define NX_ACT_BWD(T_) act_bwd_kernel<T_><<<blocks, 256, 0, st>>>(static_cast<const T_*>(x), static_cast<const T_*>(dy), static_cast<T_*>(out), n, vec, act)
  if (dtype == NX_BF16) NX_ACT_BWD(__nv_bfloat16);
  else if (dtype == NX_F16) NX_ACT_BWD(__half);
  else return -1;
#undef NX_ACT_BWD
  return launch_status();
}

extern "C" int nx_scale(const void* in, const float* factor, void* out, int dtype, int64_t n, nx_stream_t stream) {
  if (n <= 0) return n == 0 ? 0 : -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t vec = on16(in, out, out) ? n / 8 : 0;
  const int blocks = blocks_for(vec > 0 ? vec : n, 256);
#define NX_SCALE(T_) scale_kernel<T_><<<blocks, 256, 0, st>>>(static_cast<const T_*>(in), factor, static_cast<T_*>(out), n, vec)
  if (dtype == NX_BF16) NX_SCALE(__nv_bfloat16);
  else if (dtype == NX_F32) NX_SCALE(float);
  else return -1;
#undef NX_SCALE
  return launch_status();
}

extern "C" int nx_rope_rows(const void* x, int64_t ldx, void* y, int64_t ldy, const float* cos_t, const float* sin_t, int rows, int seq_len,
                            int heads, int head_dim, int half, int inverse, nx_stream_t stream) {
  if (rows <= 0 || seq_len <= 0 || heads <= 0 || half <= 0 || 2 * half > head_dim) return -1;
  if ((half & 7) || (head_dim & 7) || (ldx & 7) || (ldy & 7) || !on16(x, y, y) || !on16(cos_t, sin_t, sin_t)) return -1;
  const int64_t total = static_cast<int64_t>(rows) * heads * (head_dim - half) / 8;
  if (total >= (int64_t{1} << 31)) return -1;
  rope_rows_kernel<<<blocks_for(total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy, cos_t, sin_t, rows, seq_len, heads, head_dim, half,
      inverse ? -1.0f : 1.0f);
  return launch_status();
}
