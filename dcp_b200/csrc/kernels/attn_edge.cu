// Passes over memory at the edges of an attention call, all bound by HBM bandwidth: 16-byte accesses and
// several of them in flight per thread.
//
//  pad_cast_rows   rows of d channels (fp32 / fp16 / bf16) -> bf16 rows of 128, zero-padded
//  cut_cast_rows   rows of 128 (fp32 accumulators or bf16) -> rows of d channels in the caller's type
//  attn_bwd_prep   delta = rowsum(dO * O) and cleared dQ / dKV accumulators, one launch; also from rows in the caller's form,
//                  with dO converted on the way
//
// The two row kernels take up to two tensors per launch (Q and KV, O and dO, dQ and dKV).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "attn_levels.cuh"
#include "entries.h"
#include "launch.cuh"

namespace dcpk {

static constexpr int kEdgeHeadDim = 128;
static constexpr int kEdgeThreads = 256;
static constexpr int kEdgeBlocks = 148 * 8;   // every SM full (2048 threads)
// Passes over up to so many chunks of 16 bytes (about 10 us) begin while the kernel before them ends.  Longer ones gain
// nothing from it (6168 tokens of 32 heads, forward and backward, 1008 -> 1010 us; 121987 tokens 41.4 -> 41.9 ms).
// Passes over levels of dQ are plain launches: overlapped, both took longer (2048 tokens, 8 / 2 heads, forward and
// backward in a graph, 88 and 93 us; four sequences of 300 to 2100 tokens 119 and 122).
static constexpr size_t kSmallPass = size_t(1) << 21;

__device__ __forceinline__ void load8(const float* p, float* f) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(v[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ void load8(const __half* p, float* f) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __half2* v = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __half22float2(v[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ void store8(float* p, const float* f) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* f) {
  uint4 raw;
  __nv_bfloat162* v = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = raw;
}
__device__ __forceinline__ void store8(__half* p, const float* f) {
  uint4 raw;
  __half2* v = reinterpret_cast<__half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = raw;
}

// chunk = 8 channels; `c` runs over rows * 16 chunks of the padded side
template <typename T>
__device__ __forceinline__ void pad_chunk(const T* src, __nv_bfloat16* dst, size_t c, int d8) {
  const size_t row = c >> 4;
  const int k = int(c & 15);
  float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (k < d8) load8(src + (row * d8 + k) * 8, f);
  store8(dst + c * 8, f);
}
template <typename T>
__global__ void __launch_bounds__(kEdgeThreads) pad_cast_kernel(const T* __restrict__ src0, __nv_bfloat16* __restrict__ dst0,
                                                                size_t n0, const T* __restrict__ src1,
                                                                __nv_bfloat16* __restrict__ dst1, size_t n1, int d8) {
  const size_t stride = size_t(gridDim.x) * kEdgeThreads;
  grid_let_next();
  grid_wait();
  for (size_t c = size_t(blockIdx.x) * kEdgeThreads + threadIdx.x; c < n0 + n1; c += stride) {
    if (c < n0) pad_chunk(src0, dst0, c, d8);
    else pad_chunk(src1, dst1, c - n0, d8);
  }
}

// `c` runs over rows * d / 8 chunks of the narrow side
template <typename S, typename T>
__device__ __forceinline__ void cut_chunk(const S* src, T* dst, size_t c, int d8) {
  const size_t row = d8 == 16 ? c >> 4 : c / d8;
  float f[8];
  load8(src + row * kEdgeHeadDim + (c - row * d8) * 8, f);
  store8(dst + c * 8, f);
}
template <typename S, typename T>
__global__ void __launch_bounds__(kEdgeThreads) cut_cast_kernel(const S* __restrict__ src0, T* __restrict__ dst0, size_t n0,
                                                                const S* __restrict__ src1, T* __restrict__ dst1, size_t n1,
                                                                int d8) {
  const size_t stride = size_t(gridDim.x) * kEdgeThreads;
  grid_let_next();
  grid_wait();
  for (size_t c = size_t(blockIdx.x) * kEdgeThreads + threadIdx.x; c < n0 + n1; c += stride) {
    if (c < n0) cut_chunk(src0, dst0, c, d8);
    else cut_chunk(src1, dst1, c - n0, d8);
  }
}

// The same of dQ and dKV where dQ has levels, which are added on the way.  The first `row_blocks` blocks take dQ,
// kLevelRows rows each.  As a launch of its own the sum took 13 us of 135 (42 MB of levels and 16 of dQ; four sequences
// of 300 to 2100 tokens, 8 / 2 heads).
template <typename T>
__global__ void __launch_bounds__(kEdgeThreads)
cut_cast_levels_kernel(const __grid_constant__ DqLevels lv, const float* __restrict__ dq, T* __restrict__ gq,
                       const float* __restrict__ dkv, T* __restrict__ gkv, size_t n_kv, int d8, int row_blocks) {
  __shared__ RowLevels present;
  grid_let_next();
  grid_wait();
  if (int(blockIdx.x) >= row_blocks) {
    const size_t stride = size_t(gridDim.x - row_blocks) * kEdgeThreads;
    for (size_t c = size_t(blockIdx.x - row_blocks) * kEdgeThreads + threadIdx.x; c < n_kv; c += stride)
      cut_chunk(dkv, gkv, c, d8);
    return;
  }
  const int row0 = blockIdx.x * kLevelRows, per_row = lv.hq * d8;
  find_levels(lv, row0, present);
  for (int c = threadIdx.x; c < kLevelRows * per_row; c += kEdgeThreads) {
    const int r = c / per_row, k = c % d8;
    if (row0 + r >= lv.q_rows) break;
    const size_t head_row = size_t(row0 + r) * lv.hq + c % per_row / d8;
    const float4* src = reinterpret_cast<const float4*>(dq + head_row * kEdgeHeadDim + 8 * k);
    const uint64_t above = levels_above(present, r);
    float4 a = src[0], b = src[1];
    add_levels(lv, above, head_row * lv.pitch + 8 * k, a);
    add_levels(lv, above, head_row * lv.pitch + 8 * k + 4, b);
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    store8(gq + (head_row * d8 + k) * 8, f);
  }
}

// delta[h][row] = sum_d dO[row][h][d] * O[row][h][d]: sixteen lanes per (row, head), 16 bytes each of both
// operands, four (row, head) pairs in flight per thread; then the grid clears the two accumulators.
// One warp per pair with 8-byte loads read at 3.7 TB/s and the two fills were launches of their own.
template <bool kLevels>
__global__ void __launch_bounds__(kEdgeThreads) attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o,
                                                                     const __nv_bfloat16* __restrict__ d_o,
                                                                     float* __restrict__ delta, int n_rows, int hq,
                                                                     int stat_stride, float4* __restrict__ zero0, size_t nz0,
                                                                     float4* __restrict__ zero1, size_t nz1,
                                                                     const __grid_constant__ DqLevels levels) {
  const size_t tid = size_t(blockIdx.x) * kEdgeThreads + threadIdx.x, n_thr = size_t(gridDim.x) * kEdgeThreads;
  const int sub = threadIdx.x & 15;
  const size_t n_items = size_t(n_rows) * hq, step = n_thr >> 4;
  grid_let_next();
  grid_wait();
  // the trip count depends on the block only, so the shuffles below see whole warps
  for (size_t base = size_t(blockIdx.x) * (kEdgeThreads / 16); base < n_items; base += 4 * step) {
    uint4 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t item = base + u * step + (threadIdx.x >> 4);
      a[u] = b[u] = make_uint4(0, 0, 0, 0);
      if (item < n_items) {
        a[u] = *reinterpret_cast<const uint4*>(o + item * kEdgeHeadDim + sub * 8);
        b[u] = *reinterpret_cast<const uint4*>(d_o + item * kEdgeHeadDim + sub * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t item = base + u * step + (threadIdx.x >> 4);
      const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&a[u]), *y = reinterpret_cast<const __nv_bfloat162*>(&b[u]);
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 p = __bfloat1622float2(x[i]), q = __bfloat1622float2(y[i]);
        acc += p.x * q.x + p.y * q.y;
      }
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
      if (sub == 0 && item < n_items) delta[(item % hq) * size_t(stat_stride) + item / hq] = acc;
    }
  }
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (size_t i = tid; i < nz0; i += n_thr) zero0[i] = z;
  for (size_t i = tid; i < nz1; i += n_thr) zero1[i] = z;
  if constexpr (kLevels) {
    __shared__ RowLevels present;
    for (int row0 = blockIdx.x * kLevelRows; row0 < levels.q_rows; row0 += gridDim.x * kLevelRows)
      clear_levels(levels, row0, present);
  }
}

// The same for gradients in the caller's form (rows of d8 chunks of 8 channels): dO also goes to the arena's rows,
// rounded to bf16 and zero-padded, and delta is that of the rounded values.  As a pass that converts O and dO and the
// one above it took 22 us for 7680 tokens of 8 heads with 64 fp32 channels.
template <typename T, bool kLevels>
__global__ void __launch_bounds__(kEdgeThreads) attn_bwd_prep_cast_kernel(const T* __restrict__ o, const T* __restrict__ d_o, int d8,
                                                                          __nv_bfloat16* __restrict__ rows, float* __restrict__ delta,
                                                                          int n_rows, int hq, int stat_stride,
                                                                          float4* __restrict__ zero0, size_t nz0,
                                                                          float4* __restrict__ zero1, size_t nz1,
                                                                          const __grid_constant__ DqLevels levels) {
  constexpr int kInFlight = 2;
  const size_t tid = size_t(blockIdx.x) * kEdgeThreads + threadIdx.x, n_thr = size_t(gridDim.x) * kEdgeThreads;
  const int sub = threadIdx.x & 15;
  const size_t n_items = size_t(n_rows) * hq, step = n_thr >> 4;
  grid_let_next();
  grid_wait();
  // the trip count depends on the block only, so the shuffles below see whole warps
  for (size_t base = size_t(blockIdx.x) * (kEdgeThreads / 16); base < n_items; base += kInFlight * step) {
    float a[kInFlight][8], b[kInFlight][8];
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const size_t item = base + u * step + (threadIdx.x >> 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[u][i] = b[u][i] = 0.f;
      if (item < n_items && sub < d8) {
        load8(o + (item * d8 + sub) * 8, a[u]);
        load8(d_o + (item * d8 + sub) * 8, b[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const size_t item = base + u * step + (threadIdx.x >> 4);
      if (item < n_items) store8(rows + item * kEdgeHeadDim + sub * 8, b[u]);
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        acc += __bfloat162float(__float2bfloat16_rn(a[u][2 * i])) * __bfloat162float(__float2bfloat16_rn(b[u][2 * i])) +
               __bfloat162float(__float2bfloat16_rn(a[u][2 * i + 1])) * __bfloat162float(__float2bfloat16_rn(b[u][2 * i + 1]));
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
      if (sub == 0 && item < n_items) delta[(item % hq) * size_t(stat_stride) + item / hq] = acc;
    }
  }
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (size_t i = tid; i < nz0; i += n_thr) zero0[i] = z;
  for (size_t i = tid; i < nz1; i += n_thr) zero1[i] = z;
  if constexpr (kLevels) {
    __shared__ RowLevels present;
    for (int row0 = blockIdx.x * kLevelRows; row0 < levels.q_rows; row0 += gridDim.x * kLevelRows)
      clear_levels(levels, row0, present);
  }
}

static int edge_grid(size_t chunks) {
  const size_t b = (chunks + kEdgeThreads - 1) / kEdgeThreads;
  return int(b < size_t(kEdgeBlocks) ? b : size_t(kEdgeBlocks));
}

template <typename T>
static void launch_pad(const void* s0, void* d0, size_t n0, const void* s1, void* d1, size_t n1, int d8, cudaStream_t st) {
  launch_overlapped(pad_cast_kernel<T>, edge_grid(n0 + n1), kEdgeThreads, 0, st, 1, n0 + n1 <= kSmallPass, static_cast<const T*>(s0),
                    static_cast<__nv_bfloat16*>(d0), n0, static_cast<const T*>(s1), static_cast<__nv_bfloat16*>(d1), n1, d8);
}
template <typename S, typename T>
static void launch_cut(const void* s0, void* d0, size_t n0, const void* s1, void* d1, size_t n1, int d8, cudaStream_t st) {
  launch_overlapped(cut_cast_kernel<S, T>, edge_grid(n0 + n1), kEdgeThreads, 0, st, 1, n0 + n1 <= kSmallPass,
                    static_cast<const S*>(s0), static_cast<T*>(d0), n0, static_cast<const S*>(s1), static_cast<T*>(d1), n1, d8);
}

}  // namespace dcpk

using namespace dcpk;

// element types: 0 fp32, 1 fp16, 2 bf16.  rows0 / rows1: rows of the two tensors (0: absent), d: channels per row
// (multiple of 8, at most 128).  All pointers 16-byte aligned.
extern "C" int dcpk_pad_cast_rows(int type, const void* src0, void* dst0, long rows0, const void* src1, void* dst1,
                                  long rows1, int d, void* stream) {
  if (rows0 < 0 || rows1 < 0 || d <= 0 || d % 8 || d > kEdgeHeadDim) return -3;
  if (rows0 + rows1 == 0) return 0;
  const size_t n0 = size_t(rows0) * 16, n1 = size_t(rows1) * 16;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (type == 0) launch_pad<float>(src0, dst0, n0, src1, dst1, n1, d / 8, st);
  else if (type == 1) launch_pad<__half>(src0, dst0, n0, src1, dst1, n1, d / 8, st);
  else if (type == 2) launch_pad<__nv_bfloat16>(src0, dst0, n0, src1, dst1, n1, d / 8, st);
  else return -3;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// src_f32: the rows of 128 are fp32 (1) or bf16 (0)
extern "C" int dcpk_cut_cast_rows(int src_f32, int type, const void* src0, void* dst0, long rows0, const void* src1,
                                  void* dst1, long rows1, int d, void* stream) {
  if (rows0 < 0 || rows1 < 0 || d <= 0 || d % 8 || d > kEdgeHeadDim || type < 0 || type > 2) return -3;
  if (rows0 + rows1 == 0) return 0;
  const int d8 = d / 8;
  const size_t n0 = size_t(rows0) * d8, n1 = size_t(rows1) * d8;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (src_f32) {
    if (type == 0) launch_cut<float, float>(src0, dst0, n0, src1, dst1, n1, d8, st);
    else if (type == 1) launch_cut<float, __half>(src0, dst0, n0, src1, dst1, n1, d8, st);
    else launch_cut<float, __nv_bfloat16>(src0, dst0, n0, src1, dst1, n1, d8, st);
  } else {
    if (type == 0) launch_cut<__nv_bfloat16, float>(src0, dst0, n0, src1, dst1, n1, d8, st);
    else if (type == 1) launch_cut<__nv_bfloat16, __half>(src0, dst0, n0, src1, dst1, n1, d8, st);
    else launch_cut<__nv_bfloat16, __nv_bfloat16>(src0, dst0, n0, src1, dst1, n1, d8, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// The gradients of a call whose dQ has levels (these with items, workspace and the rest of dcpk_attn_bwd's call): dq
// fp32 [levels->q_rows, levels->hq, 128] and dkv fp32 [rows1, 128] -> rows of d channels of element type `type`.
extern "C" int dcpk_cut_cast_gradients(int type, const DcpkDqLevels* levels, const float* dq, void* gq, const float* dkv, void* gkv,
                                       long rows1, int d, void* stream) {
  if (!levels || !levels->workspace || levels->n_levels < 2 || rows1 < 0 || d <= 0 || d % 8 || d > kEdgeHeadDim ||
      d > levels->channels || type < 0 || type > 2)
    return -3;
  const int d8 = d / 8, row_blocks = (levels->q_rows + kLevelRows - 1) / kLevelRows;
  const size_t n_kv = size_t(rows1) * d8;
  auto launch = [&](auto kernel, auto* as) {
    using T = std::remove_pointer_t<decltype(as)>;
    return launch_overlapped(kernel, unsigned(row_blocks + edge_grid(n_kv)), kEdgeThreads, 0, static_cast<cudaStream_t>(stream), 1, false,
                             make_levels(levels), dq, static_cast<T*>(gq), dkv, static_cast<T*>(gkv), n_kv, d8, row_blocks);
  };
  if (type == 0) launch(cut_cast_levels_kernel<float>, static_cast<float*>(nullptr));
  else if (type == 1) launch(cut_cast_levels_kernel<__half>, static_cast<__half*>(nullptr));
  else launch(cut_cast_levels_kernel<__nv_bfloat16>, static_cast<__nv_bfloat16*>(nullptr));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// o, d_o: bf16 [n_rows, hq, 128]; delta fp32 [hq, stat_stride]; zero0 / zero1: fp32 buffers of nz0 / nz1 elements
// (multiples of 4); levels (may be null): of the dQ of the backward that follows, cleared where it will add to them
extern "C" int dcpk_attn_bwd_prep(const void* o, const void* d_o, float* delta, int n_rows, int hq, int stat_stride,
                                  float* zero0, long nz0, float* zero1, long nz1, const DcpkDqLevels* levels, void* stream) {
  if (n_rows < 0 || hq <= 0 || n_rows > stat_stride || nz0 % 4 || nz1 % 4 || nz0 < 0 || nz1 < 0) return -3;
  const size_t work = size_t(n_rows) * hq * 16 + size_t(nz0 + nz1) / 4;
  if (work == 0) return 0;
  const bool clear = levels && levels->workspace;
  launch_overlapped(
      clear ? attn_bwd_prep_kernel<true> : attn_bwd_prep_kernel<false>, edge_grid(work), kEdgeThreads, 0,
      static_cast<cudaStream_t>(stream), 1, work <= kSmallPass && !clear,
      static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), delta, n_rows, hq, stat_stride,
      reinterpret_cast<float4*>(zero0), size_t(nz0) / 4, reinterpret_cast<float4*>(zero1), size_t(nz1) / 4, make_levels(levels));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// o, d_o: [n_rows, hq, d] of an element type as above; d_o_rows: bf16 [n_rows, hq, 128]; the rest as dcpk_attn_bwd_prep
extern "C" int dcpk_attn_bwd_prep_cast(int type, const void* o, const void* d_o, int d, void* d_o_rows, float* delta, int n_rows, int hq,
                                       int stat_stride, float* zero0, long nz0, float* zero1, long nz1,
                                       const DcpkDqLevels* levels, void* stream) {
  if (n_rows < 0 || hq <= 0 || n_rows > stat_stride || nz0 % 4 || nz1 % 4 || nz0 < 0 || nz1 < 0 || d <= 0 || d % 8 ||
      d > kEdgeHeadDim || type < 0 || type > 2)
    return -3;
  const size_t work = size_t(n_rows) * hq * 16 + size_t(nz0 + nz1) / 4;
  if (work == 0) return 0;
  const bool clear = levels && levels->workspace;
  auto launch = [&](auto* as) {
    using T = std::remove_pointer_t<decltype(as)>;
    return launch_overlapped(clear ? attn_bwd_prep_cast_kernel<T, true> : attn_bwd_prep_cast_kernel<T, false>,
                             edge_grid(work), kEdgeThreads, 0, static_cast<cudaStream_t>(stream), 1,
                             work <= kSmallPass && !clear, static_cast<const T*>(o), static_cast<const T*>(d_o), d / 8,
                             static_cast<__nv_bfloat16*>(d_o_rows), delta, n_rows, hq, stat_stride,
                             reinterpret_cast<float4*>(zero0), size_t(nz0) / 4, reinterpret_cast<float4*>(zero1),
                             size_t(nz1) / 4, make_levels(levels));
  };
  if (type == 0) launch(static_cast<float*>(nullptr));
  else if (type == 1) launch(static_cast<__half*>(nullptr));
  else launch(static_cast<__nv_bfloat16*>(nullptr));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
