// y[m][n] = act(x[m][:] . w[n][:] + bias[n]) + residual[m][n] for few rows: decode steps and short verification runs.  Bound by
// reading the weights once; at these sizes that means loads in flight, and the launches and passes around them.  Two forms, each of
// which gives a row the same bits in any batch that it takes:
//
// Up to 16 rows, `skinny_kernel`: a warp has C columns, its lanes stride along K; FP32 sums on the CUDA cores, reduced by a fixed
// butterfly.  The weights of the next steps and the rows of x are in registers before they are needed, the weights of a loaded
// model even before the kernel in front has finished.  C columns share the loads and conversions of the rows of x, which took
// more issue slots than the products.
//
// Up to 64 rows, `few_rows_kernel`: the weights go straight from memory into the registers of `mma.sync` (16 columns of w per
// warp, 16 bytes per thread and row), kAhead chunks of 32 reduction elements ahead; the rows of x pass through shared memory once
// per block of 64 columns; K is split over the CTAs of a cluster, whose partial sums meet through distributed shared memory in a
// fixed order, so there is no workspace and no second launch.  The split depends on n and k alone, and each column of the MMA is a
// row of x.  Within a chunk the four threads of a quad hold 8 consecutive elements of K each, in w and in x alike; the MMA then
// sums the elements in another order than they lie in memory, the same one for both operands.  64 rows, against the split
// tcgen05 product and its reduction pass: 7.2 and 12.4 us at 1600 x 1600, 12.1 and 17.0 at 4800 x 1600, 6.5 and 13.8 at
// 3072 x 768, but 20.1 and 15.9 at 1600 x 6400 and 76 and 39 (unsplit) at 50304 x 1600: `mma.sync` runs out of throughput.
#include "common.cuh"
#include "mixer_common.cuh"
#include "nx_api_infer.h"
#include "sm100_ptx.cuh"

#include <algorithm>

namespace {
using namespace nx;

constexpr int kSkinnyRows = 16, kFewRows = 64;
constexpr int kCols = 64;             // columns of a few-rows block: 4 warps of 16
constexpr int kStageK = 128;          // elements of K per shared-memory stage of x
constexpr int kStages = 3;
constexpr int kPitch = kStageK * 2 + 64;  // bytes; = 64 mod 128: the 16-byte reads of a quarter-warp (two rows) meet no bank twice
constexpr int kRedPitch = kCols + 4;      // floats
constexpr int kAhead = 8;                 // chunks of w in a few-rows warp's registers

struct FewRowsArgs {
  const __nv_bfloat16 *x, *w, *bias;
  const void* residual;
  void* y;
  int64_t ldx, ldw, ldr, ldy;
  int m, n, k, act, k_per;  // k_per: elements of K per CTA of the cluster, a multiple of 32
  int vec;                  // y and residual rows take 4-element accesses
  int w_const;              // w is written by no kernel that may still run: it is read before the grid dependency
};

__device__ __forceinline__ uint4 ld_weights(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ float apply_act(float v, int act) {
  if (act == NX_ACT_GELU) return gelu_tanh_f(v);
  if (act == NX_ACT_RELU) return fmaxf(v, 0.0f);
  if (act == NX_ACT_SILU) return silu_f(v);
  if (act == NX_ACT_RELU2) return fmaxf(v, 0.0f) * fmaxf(v, 0.0f);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& q, float (&v)[8]) {
  unpack_bf16x2(q.x, v[0], v[1]);
  unpack_bf16x2(q.y, v[2], v[3]);
  unpack_bf16x2(q.z, v[4], v[5]);
  unpack_bf16x2(q.w, v[6], v[7]);
}

// M rows (the last one repeated where there are fewer), C columns per warp, 4 warps per block.  A step is 256 elements of K.
template <int M, int C, typename YT>
__global__ void __launch_bounds__(128, M > 8 ? 2 : (M > 2 ? 3 : 5)) skinny_kernel(const FewRowsArgs a) {
  constexpr int kW = M <= 2 ? 8 : (C == 4 ? 2 : 4);   // steps of weights in registers
  constexpr int kX = M == 1 ? 4 : (M == 2 ? 2 : 1);   // steps of x
  const int lane = threadIdx.x & 31, col0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * C;
  pdl_trigger();
  if (col0 >= a.n) return;
  const __nv_bfloat16* w[C];
#pragma unroll
  for (int c = 0; c < C; ++c) w[c] = a.w + static_cast<int64_t>(min(col0 + c, a.n - 1)) * a.ldw + lane * 8;
  uint4 wr[kW][C], xr[kX][M];
  auto fetch_w = [&](int slot, int k) {
#pragma unroll
    for (int c = 0; c < C; ++c) wr[slot][c] = k + lane * 8 < a.k ? ld_weights(w[c] + k) : make_uint4(0u, 0u, 0u, 0u);
  };
  auto load_x = [&](int i, int k) {
    return k + lane * 8 < a.k ? *reinterpret_cast<const uint4*>(a.x + min(i, a.m - 1) * a.ldx + k + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
  };
  if (!a.w_const) pdl_dependency();
#pragma unroll
  for (int s = 0; s < kW; ++s) fetch_w(s, s * 256);
  if (a.w_const) pdl_dependency();
#pragma unroll
  for (int s = 0; s < kX; ++s)
#pragma unroll
    for (int i = 0; i < M; ++i) xr[s][i] = load_x(i, s * 256);
  // lane i * C + c finishes row i of column c: its residual is on the way while the products run
  static_assert(M * C <= 32, "a lane per result");
  const int my_row = lane / C, my_col = col0 + lane % C;
  const bool mine = my_row < a.m && my_col < a.n;
  const float bias = a.bias != nullptr && my_col < a.n ? __bfloat162float(a.bias[my_col]) : 0.0f;
  const float res = a.residual != nullptr && mine ? Num<YT>::load(static_cast<const YT*>(a.residual) + my_row * a.ldr + my_col) : 0.0f;
  float acc[M][C];
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[i][c] = 0.0f;
  for (int k0 = 0; k0 < a.k; k0 += kW * 256) {
#pragma unroll
    for (int s = 0; s < kW; ++s) {
      const int k = k0 + s * 256;
      if (k >= a.k) break;
      const bool in = k + lane * 8 < a.k;
      float wv[C][8];
#pragma unroll
      for (int c = 0; c < C; ++c) unpack8(wr[s][c], wv[c]);
      fetch_w(s, k + kW * 256);
#pragma unroll
      for (int i = 0; i < M; ++i) {
        float xv[8];
        unpack8(xr[s % kX][i], xv);
        xr[s % kX][i] = load_x(i, k + kX * 256);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          float t = 0.0f;
#pragma unroll
          for (int j = 0; j < 8; ++j) t += xv[j] * wv[c][j];
          if (in) acc[i][c] += t;
        }
      }
    }
  }
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float t = acc[i][c];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == i * C + c) sum = t;
    }
  if (!mine) return;
  float v = apply_act(sum + bias, a.act);
  if (a.residual != nullptr) v += res;
  Num<YT>::store(static_cast<YT*>(a.y) + my_row * a.ldy + my_col, v);
}

// The same sums of exactly M rows with a column per warp and no prefetch of its own: many small warps per SM instead.  kSpread: lane i
// finishes row i, otherwise lane 0 finishes them all, which takes fewer registers for some M (M = 12 and 16: 48 against 54, so that an
// SM holds a block more; with the arguments in a struct 16 rows of 6400 x 1600 took 32.7 us in place of 28.9).
template <int M, bool kSpread, typename YT>
__global__ void __launch_bounds__(256)
skinny_wide_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, const __nv_bfloat16* __restrict__ w, int64_t ldw,
                   const __nv_bfloat16* __restrict__ bias, const YT* residual, int64_t ldr, YT* y, int64_t ldy, int n, int k, int act) {
  const int col = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if constexpr (kSpread) {
    pdl_trigger();
    pdl_dependency();
  }
  if (col >= n) return;
  float acc[M];
#pragma unroll
  for (int i = 0; i < M; ++i) acc[i] = 0.0f;
  const __nv_bfloat16* wr = w + static_cast<int64_t>(col) * ldw;
  for (int c = lane * 8; c < k; c += 256) {
    float wv[8];
    unpack8(*reinterpret_cast<const uint4*>(wr + c), wv);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      float xv[8];
      unpack8(*reinterpret_cast<const uint4*>(x + i * ldx + c), xv);
      float t = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) t += xv[j] * wv[j];
      acc[i] += t;
    }
  }
  if constexpr (kSpread) {
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      float t = acc[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == i) sum = t;
    }
    if (lane >= M) return;
    float v = apply_act(sum + (bias != nullptr ? __bfloat162float(bias[col]) : 0.0f), act);
    if (residual != nullptr) v += Num<YT>::load(residual + lane * ldr + col);
    Num<YT>::store(y + lane * ldy + col, v);
  } else {
#pragma unroll
    for (int i = 0; i < M; ++i) {
      float t = acc[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      acc[i] = t;
    }
    if (lane != 0) return;
    const float b = bias != nullptr ? __bfloat162float(bias[col]) : 0.0f;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      float v = apply_act(acc[i] + b, act);
      if (residual != nullptr) v += Num<YT>::load(residual + i * ldr + col);
      Num<YT>::store(y + i * ldy + col, v);
    }
  }
}

template <int M, int C, typename YT>
int launch_skinny_as(const FewRowsArgs& a, cudaStream_t st) {
  return launch_pdl(skinny_kernel<M, C, YT>, dim3(static_cast<unsigned>((a.n + 4 * C - 1) / (4 * C))), dim3(128), 0, st, a);
}
// Whether lanes finish a row each (1, 2, 13 and 15 rows: always; 11: never, 1 to 5 % faster).  One lane finishes them all where the
// registers that saves end the grid a wave earlier (4800 x 1600, spread and one lane: 25.0 and 24.2 us with 16 rows; 5120 x 1600 21.8
// and 19.7 with 12; 6400 x 1600 20.2 and 18.6 with 9), and for the row counts whose loop comes out the faster with it: 12 and 14
// where the loop outweighs the finish (k = 3072: 2 to 8 %; at k = 768 spread is 3 to 5 % faster), 10, 14 and 16 where the blocks
// nearly fill their one wave (5120 x 1280 with 10 rows 12.7 and 12.3, 3072 x 768 with 14 8.1 and 7.9, 3840 x 3072 with 16 33.3 and 31.7).
template <int M, typename YT>
bool spread_finish(unsigned blocks, int k) {
  if ((M == 12 || M == 14) && k > 1536) return false;
  auto per_wave = [](auto kern) {
    int per_sm = 0;
    const bool ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0) == cudaSuccess && per_sm > 0;
    return static_cast<unsigned>((ok ? per_sm : 4) * kNumSmsB200);
  };
  static const unsigned one = per_wave(skinny_wide_kernel<M, false, YT>), each = per_wave(skinny_wide_kernel<M, true, YT>);
  const unsigned waves = (blocks + one - 1) / one;
  if (waves < (blocks + each - 1) / each) return false;
  return !(waves == 1 && ((M == 10 && blocks > 4 * kNumSmsB200) || (M == 14 && blocks > 2 * kNumSmsB200) || (M == 16 && k > 2048 && blocks > 400)));
}
template <int M, typename YT>
int launch_wide(const FewRowsArgs& a, cudaStream_t st) {
  const dim3 grid(static_cast<unsigned>((a.n + 7) / 8)), block(256);
  const YT* res = static_cast<const YT*>(a.residual);
  YT* y = static_cast<YT*>(a.y);
  // One row alone is a dependent launch (4128 x 1024: 3.9 -> 3.5 us): with more rows the blocks that wait take warps from the grid in
  // front (4800 x 1600, dependent and plain: 8.0 and 7.1 us with 2 rows, 27.7 and 25.5 with 16).
  if constexpr (M == 1) {
    return launch_pdl(skinny_wide_kernel<M, true, YT>, grid, block, 0, st, a.x, a.ldx, a.w, a.ldw, a.bias, res, a.ldr, y, a.ldy, a.n, a.k, a.act);
  } else {
    auto kern = skinny_wide_kernel<M, M != 11, YT>;
    if constexpr (M != 2 && M != 11 && M != 13 && M != 15) {
      if (!spread_finish<M, YT>(grid.x, a.k)) kern = skinny_wide_kernel<M, false, YT>;
    }
    kern<<<grid, block, 0, st>>>(a.x, a.ldx, a.w, a.ldw, a.bias, res, a.ldr, y, a.ldy, a.n, a.k, a.act);
    return launch_status();
  }
}
template <typename YT>
int launch_skinny(const FewRowsArgs& a, cudaStream_t st) {
  // 3 to 8 rows: columns per warp share what a row costs besides its products, but there have to be warps enough to have most of
  // the matrix requested at once (sixteen per SM at four columns, eight at two).  8 rows, one column per warp without prefetch and
  // now: 15.5 -> 8.8 us at 768 x 3072, 31.3 -> 17.3 at 1600 x 6400, 38.7 -> 33.3 at 32000 x 1024.
  const bool four = a.n >= 4 * 16 * kNumSmsB200, two = a.n >= 2 * 8 * kNumSmsB200;
  // 1, 2 and 9 to 16 rows: prefetch while the columns do not fill the machine with warps by themselves (one row: 6.4 -> 5.3 us at
  // 1024 x 4096, but 15.6 without against 25.9 us at 50304 x 768; 12 rows: 19.2 -> 9.0 us at 768 x 3072, but 12.4 against 14.5 at
  // 4800 x 1024).  With 13 and more rows two of its blocks fill an SM's registers, so that it ends where a second wave would begin
  // (columns without and with prefetch, 13 rows: 7.1 and 5.5 us at 1184 x 1024, 7.6 and 9.9 at 1600 x 1024); 16 rows of a long K
  // bear that a little longer (17.6 -> 14.6 us at 1600 x 1600).  11 rows take the instance of 12.
  const int alone_above = kNumSmsB200 * (a.m == 1 || a.m == 2 ? 20 : (a.m == 11 ? 12 : (a.m < 13 ? 16 : 8)));
  const bool many = a.n > alone_above && !(a.m == 16 && a.k >= 1600 && a.n <= 1600);
#define NX_WIDE(M_) if (many && a.m == M_) return launch_wide<M_, YT>(a, st);
  NX_WIDE(1) NX_WIDE(2) NX_WIDE(9) NX_WIDE(10) NX_WIDE(11) NX_WIDE(12) NX_WIDE(13) NX_WIDE(14) NX_WIDE(15) NX_WIDE(16)
#undef NX_WIDE
#define NX_SK(M_)                                                  \
  if (a.m <= M_) {                                                 \
    if constexpr (M_ > 2 && M_ <= 8) {                             \
      if (four) return launch_skinny_as<M_, 4, YT>(a, st);         \
      if (two) return launch_skinny_as<M_, 2, YT>(a, st);          \
    }                                                              \
    return launch_skinny_as<M_, 1, YT>(a, st);                     \
  }
  NX_SK(1) NX_SK(2) NX_SK(3) NX_SK(4) NX_SK(6) NX_SK(8) NX_SK(12) NX_SK(16)
#undef NX_SK
  return -1;
}

// MT: row tiles of 8.  Grid: (CTAs of the cluster, blocks of 64 columns).
template <int MT, typename YT>
__global__ void __launch_bounds__(128) few_rows_kernel(const FewRowsArgs a) {
  constexpr int kRows = MT * 8, kPer = kStageK / 32;
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x, parts = gridDim.x, n0 = blockIdx.y * kCols;
  const int k_begin = min(rank * a.k_per, a.k), k_end = min(k_begin + a.k_per, a.k);
  const int chunks = (k_end - k_begin + 31) / 32;
  pdl_trigger();

  // columns past the end repeat the last one; their sums are not stored
  const __nv_bfloat16* w0 = a.w + static_cast<int64_t>(min(n0 + warp * 16 + g, a.n - 1)) * a.ldw + k_begin + t * 8;
  const __nv_bfloat16* w1 = a.w + static_cast<int64_t>(min(n0 + warp * 16 + g + 8, a.n - 1)) * a.ldw + k_begin + t * 8;
  uint4 wr[kAhead][2];
  auto fetch = [&](int slot, int c) {
    const bool in = k_begin + c * 32 + t * 8 < k_end;  // k is a multiple of 8: a piece is inside as a whole or not at all
    wr[slot][0] = in ? ld_weights(w0 + c * 32) : make_uint4(0u, 0u, 0u, 0u);
    wr[slot][1] = in ? ld_weights(w1 + c * 32) : make_uint4(0u, 0u, 0u, 0u);
  };
  if (!a.w_const) pdl_dependency();
#pragma unroll
  for (int i = 0; i < kAhead; ++i) fetch(i, i);
  if (a.w_const) pdl_dependency();

  const int stages = (chunks * 32 + kStageK - 1) / kStageK;
  auto stage_x = [&](int st) {  // kStageK elements of every row; rows past m and elements past the end are zeros
    uint8_t* dst = smem + (st % kStages) * kRows * kPitch;
    const int kb = k_begin + st * kStageK;
    for (int i = threadIdx.x; i < kRows * (kStageK / 8); i += 128) {
      const int r = i / (kStageK / 8), c = i % (kStageK / 8);
      uint8_t* d = dst + r * kPitch + c * 16;
      if (r < a.m && kb + c * 8 < k_end) cp_async16(d, a.x + r * a.ldx + kb + c * 8);
      else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
    }
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < stages) stage_x(s);
    cp_async_commit();
  }
  float acc[MT][4];
#pragma unroll
  for (int j = 0; j < MT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.0f;

  for (int st = 0; st < stages; st += kAhead / kPer) {
#pragma unroll
    for (int u = 0; u < kAhead / kPer; ++u) {  // the register slots stay compile-time constants
      if (st + u < stages) {
        cp_async_wait<kStages - 2>();
        __syncthreads();                    // stage st + u has landed, and every warp has left the one that is refilled
        if (st + u + kStages - 1 < stages) stage_x(st + u + kStages - 1);
        cp_async_commit();
        const uint8_t* xs = smem + ((st + u) % kStages) * kRows * kPitch;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
          const int c = (st + u) * kPer + q, slot = u * kPer + q;
          if (c < chunks) {
            const uint4 p0 = wr[slot][0], p1 = wr[slot][1];
            if (c + kAhead < chunks) fetch(slot, c + kAhead);
            const uint32_t a0[4] = {p0.x, p1.x, p0.y, p1.y}, a1[4] = {p0.z, p1.z, p0.w, p1.w};
#pragma unroll
            for (int j = 0; j < MT; ++j) {
              const uint4 b = *reinterpret_cast<const uint4*>(xs + (j * 8 + g) * kPitch + q * 64 + t * 16);
              mma_bf16(acc[j], a0, b.x, b.y);
              mma_bf16(acc[j], a1, b.z, b.w);
            }
          }
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // partial sums [row][column]; this memory was the stages of x
  float* red = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int j = 0; j < MT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) red[(j * 8 + 2 * t + (e & 1)) * kRedPitch + warp * 16 + g + (e >> 1) * 8] = acc[j][e];
  if (parts > 1) cluster_sync_all();
  else __syncthreads();
  const uint32_t base = smem_u32(red);
  for (int i = rank * 128 + threadIdx.x; i < a.m * (kCols / 4); i += parts * 128) {
    const int row = i / (kCols / 4), c4 = (i % (kCols / 4)) * 4, col = n0 + c4;
    if (col >= a.n) continue;
    const uint32_t at = base + static_cast<uint32_t>(row * kRedPitch + c4) * 4u;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    float4 p[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < parts) p[s] = ld_cluster4(parts > 1 ? mapa_shared(at, s) : at);
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < parts) { v[0] += p[s].x; v[1] += p[s].y; v[2] += p[s].z; v[3] += p[s].w; }
    const YT* res = a.residual != nullptr ? static_cast<const YT*>(a.residual) + row * a.ldr + col : nullptr;
    YT* y = static_cast<YT*>(a.y) + row * a.ldy + col;
    const int valid = min(4, a.n - col);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < valid) v[e] = apply_act(v[e] + (a.bias != nullptr ? __bfloat162float(a.bias[col + e]) : 0.0f), a.act);
    if (a.vec && valid == 4) {
      if constexpr (sizeof(YT) == 4) {
        if (res != nullptr) {
          const float4 q = *reinterpret_cast<const float4*>(res);
          v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
        }
        *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        if (res != nullptr) {
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] += __bfloat162float(res[e]);
        }
        *reinterpret_cast<uint2*>(y) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      }
    } else {
      for (int e = 0; e < valid; ++e) Num<YT>::store(y + e, v[e] + (res != nullptr ? Num<YT>::load(res + e) : 0.0f));
    }
  }
  if (parts > 1) cluster_sync_all();  // no CTA leaves while another may still read its sums
}

template <int MT, typename YT>
int launch_few(const FewRowsArgs& a, int parts, cudaStream_t st) {
  constexpr int smem = std::max(kStages * MT * 8 * kPitch, MT * 8 * kRedPitch * 4);
  auto kern = few_rows_kernel<MT, YT>;
  NX_ALLOW_SMEM(kern, smem);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(parts);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(parts), static_cast<unsigned>((a.n + kCols - 1) / kCols));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess ? 0 : ((void)cudaGetLastError(), -2);
}

// CTAs of a cluster along K: enough to have the weights of the whole matrix requested at once (two CTAs per SM), at least 64 elements
// of K each, but no more than are resident at 64 rows (three per SM): a second wave cost 12.6 us against 7.9 at 64 rows of
// 4128 x 1024, 15.6 against 13.9 at 8192 x 1024.
int few_rows_parts(int n, int k) {
  const int blocks = (n + kCols - 1) / kCols;
  int parts = 1;
  while (parts < 8 && blocks * parts < 2 * kNumSmsB200 && 2 * blocks * parts <= 3 * kNumSmsB200 && k >= 2 * parts * 64) parts *= 2;
  return parts;
}
int few_rows_chain(int k, int parts) { return ((k + parts - 1) / parts + 31) / 32 * 32; }

}  // namespace

extern "C" int nx_skinny_max_rows(void) { return kFewRows; }

extern "C" int nx_few_rows_chain(int n, int k) { return n > 0 && k > 0 ? few_rows_chain(k, few_rows_parts(n, k)) : -1; }

extern "C" int nx_skinny_gemm(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* bias, const void* residual,
                              int64_t ldr, void* y, int64_t ldy, int out_dtype, int m, int n, int k, int act, int w_const,
                              nx_stream_t stream) {
  if (m < 1 || m > kFewRows || n <= 0 || k <= 0 || (k & 7) || (ldx & 7) || (ldw & 7)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return -1;
  if (out_dtype != NX_BF16 && out_dtype != NX_F32) return -1;
  FewRowsArgs a{};
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.w = static_cast<const __nv_bfloat16*>(w);
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.residual = residual;
  a.y = y;
  a.ldx = ldx; a.ldw = ldw; a.ldr = ldr; a.ldy = ldy;
  a.m = m; a.n = n; a.k = k; a.act = act; a.w_const = w_const;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (m <= kSkinnyRows) return out_dtype == NX_F32 ? launch_skinny<float>(a, st) : launch_skinny<__nv_bfloat16>(a, st);
  const uintptr_t align = out_dtype == NX_F32 ? 15 : 7;
  a.vec = !(reinterpret_cast<uintptr_t>(y) & align) && !(ldy & 3) &&
          (residual == nullptr || (!(reinterpret_cast<uintptr_t>(residual) & align) && !(ldr & 3)));
  if ((n + kCols - 1) / kCols > 65535) return -1;
  const int parts = few_rows_parts(n, k);
  a.k_per = few_rows_chain(k, parts);
#define NX_FEW(MT_) return out_dtype == NX_F32 ? launch_few<MT_, float>(a, parts, st) : launch_few<MT_, __nv_bfloat16>(a, parts, st)
  if (m <= 32) NX_FEW(4);
  NX_FEW(8);
#undef NX_FEW
}
