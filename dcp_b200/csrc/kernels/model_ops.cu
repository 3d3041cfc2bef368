// Memory-bound transformer ops in bf16 with fp32 math, written for HBM3e: 16-byte vector
// accesses, one pass over the data wherever the math allows, and layout changes fused into
// the op that touches the data anyway.
//
//  rmsnorm_fwd / rmsnorm_bwd      y = x * rsqrt(mean(x^2) + eps) * w
//  qkv_rope_split_fwd             packed QKV projection -> rotary on q,k -> attention arenas
//  qkv_rope_pack_bwd              fp32 dQ / dKV accumulators -> inverse rotary -> packed bf16 dQKV
//  swiglu_fwd / swiglu_bwd        y = silu(gate) * up on a [T, 2F] gate|up tensor
//  cross_entropy_fwd_bwd          per-row loss and in-place dlogits in one kernel
//
// The reference takes these from Megatron-LM / TransformerEngine / apex
// (benchmark/mlm/pretrain_gpt.py:143-167, benchmark/mlm/monkey_patch.py:158-251).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

namespace dcpk {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
  return v;
}
template <int kWarps>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = lane < kWarps ? scratch[lane] : 0.f;
  return warp_sum(t);
}
template <int kWarps>
__device__ __forceinline__ float block_max(float v, float* scratch) {
  v = warp_max(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = lane < kWarps ? scratch[lane] : -INFINITY;
  return warp_max(t);
}
__device__ __forceinline__ void unpack8(const uint4& raw, float* f) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x; f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 raw;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return raw;
}

// ------------------------------------------------------------------ RMSNorm
// one CTA of 128 threads per row; hidden must be a multiple of 1024 (8 per vector x 128 threads)
template <int kVecs>
__global__ void __launch_bounds__(128) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                                          int hidden, float eps) {
  __shared__ float scratch[4];
  const size_t row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * hidden);
  float v[kVecs][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    unpack8(xr[threadIdx.x + i * 128], v[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
  }
  ss = block_sum<4>(ss, scratch);
  const float r = rsqrtf(ss / hidden + eps);
  if (threadIdx.x == 0) rstd[row] = r;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + row * hidden);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    float wv[8];
    unpack8(wr[threadIdx.x + i * 128], wv);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] = v[i][j] * r * wv[j];
    yr[threadIdx.x + i * 128] = pack8(v[i]);
  }
}

// persistent CTAs: each walks rows blockIdx.x, +gridDim.x, ... and keeps its dW slice in registers.  kResidual is a
// template parameter: tested at run time it cost rows of 8192 (255 registers) 6 % (16384 rows: 186 -> 199 us)
template <int kVecs, bool kResidual>
__global__ void __launch_bounds__(128) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          const __nv_bfloat16* __restrict__ dy,
                                                          const float* __restrict__ rstd,
                                                          __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                                                          const __nv_bfloat16* __restrict__ residual, int n_rows, int hidden) {
  __shared__ float scratch[4];
  float wv[kVecs][8], dwv[kVecs][8];
  const uint4* wr = reinterpret_cast<const uint4*>(w);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    unpack8(wr[threadIdx.x + i * 128], wv[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) dwv[i][j] = 0.f;
  }
  for (size_t row = blockIdx.x; row < size_t(n_rows); row += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * hidden);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + row * hidden);
    const float r = rstd[row];
    float xh[kVecs][8], g[kVecs][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      unpack8(xr[threadIdx.x + i * 128], xh[i]);
      unpack8(gr[threadIdx.x + i * 128], g[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[i][j] *= r;
        dwv[i][j] += g[i][j] * xh[i][j];
        g[i][j] *= wv[i][j];
        dot += g[i][j] * xh[i][j];
      }
    }
    dot = block_sum<4>(dot, scratch) / hidden;
    uint4* dxr = reinterpret_cast<uint4*>(dx + row * hidden);
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) g[i][j] = r * (g[i][j] - xh[i][j] * dot);
      if (kResidual) {   // the gradient that by-passed the norm, added before the one rounding
        float add[8];
        unpack8(reinterpret_cast<const uint4*>(residual + row * hidden)[threadIdx.x + i * 128], add);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[i][j] += add[j];
      }
      dxr[threadIdx.x + i * 128] = pack8(g[i]);
    }
  }
  // one vector reduction per four channels (a quarter of the scalar atomics, which bound this kernel)
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dw + (threadIdx.x + i * 128) * 8 + j),
                   "f"(dwv[i][j]), "f"(dwv[i][j + 1]), "f"(dwv[i][j + 2]), "f"(dwv[i][j + 3])
                   : "memory");
}

// ------------------------------------------------------------------ QKV split + rotary
// qkv: [T, (hq + 2*hkv) * 128] packed as q heads | k heads | v heads.  cos/sin: [T, 64].
// rotate-half convention: (x1, x2) -> (x1 cos - x2 sin, x2 cos + x1 sin), x1 = x[:64], x2 = x[64:].
// eight lanes per (token, head): lane s of the group owns channels 8s .. 8s+7 of each half, so every
// global access is a 16-byte vector (a warp moves four heads).
__global__ void qkv_rope_split_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ cs,
                                          const float* __restrict__ sn, __nv_bfloat16* __restrict__ q_out,
                                          __nv_bfloat16* __restrict__ kv_out, int n_tok, int hq, int hkv,
                                          int q_row0, int kv_row0) {
  const int heads = hq + 2 * hkv;
  const long item = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  if (item >= long(n_tok) * heads) return;
  const int t = int(item / heads), h = int(item % heads);
  const __nv_bfloat16* src = qkv + (size_t(t) * heads + h) * 128;
  __nv_bfloat16* dst;
  if (h < hq) dst = q_out + (size_t(q_row0 + t) * hq + h) * 128;
  else if (h < hq + hkv) dst = kv_out + ((size_t(kv_row0 + t) * 2 + 0) * hkv + (h - hq)) * 128;
  else dst = kv_out + ((size_t(kv_row0 + t) * 2 + 1) * hkv + (h - hq - hkv)) * 128;
  const uint4 a = *reinterpret_cast<const uint4*>(src + 8 * sub);
  const uint4 b = *reinterpret_cast<const uint4*>(src + 64 + 8 * sub);
  if (h < hq + hkv) {
    float x1[8], x2[8], c[8], sv[8], o1[8], o2[8];
    unpack8(a, x1); unpack8(b, x2);
    *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cs + size_t(t) * 64 + 8 * sub);
    *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cs + size_t(t) * 64 + 8 * sub + 4);
    *reinterpret_cast<float4*>(sv) = *reinterpret_cast<const float4*>(sn + size_t(t) * 64 + 8 * sub);
    *reinterpret_cast<float4*>(sv + 4) = *reinterpret_cast<const float4*>(sn + size_t(t) * 64 + 8 * sub + 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o1[j] = x1[j] * c[j] - x2[j] * sv[j];
      o2[j] = x2[j] * c[j] + x1[j] * sv[j];
    }
    *reinterpret_cast<uint4*>(dst + 8 * sub) = pack8(o1);
    *reinterpret_cast<uint4*>(dst + 64 + 8 * sub) = pack8(o2);
  } else {
    *reinterpret_cast<uint4*>(dst + 8 * sub) = a;
    *reinterpret_cast<uint4*>(dst + 64 + 8 * sub) = b;
  }
}

// dq: fp32 [rows, hq, 128], dkv: fp32 [rows, 2, hkv, 128] -> dqkv bf16 [T, (hq+2hkv)*128] with the
// rotation transposed (sin negated) on the q and k parts.  Same eight-lanes-per-head layout.
__global__ void qkv_rope_pack_bwd_kernel(const float* __restrict__ dq, const float* __restrict__ dkv,
                                         const float* __restrict__ cs, const float* __restrict__ sn,
                                         __nv_bfloat16* __restrict__ dqkv, int n_tok, int hq, int hkv, int q_row0,
                                         int kv_row0) {
  const int heads = hq + 2 * hkv;
  const long item = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  if (item >= long(n_tok) * heads) return;
  const int t = int(item / heads), h = int(item % heads);
  const float* src;
  if (h < hq) src = dq + (size_t(q_row0 + t) * hq + h) * 128;
  else if (h < hq + hkv) src = dkv + ((size_t(kv_row0 + t) * 2 + 0) * hkv + (h - hq)) * 128;
  else src = dkv + ((size_t(kv_row0 + t) * 2 + 1) * hkv + (h - hq - hkv)) * 128;
  __nv_bfloat16* dst = dqkv + (size_t(t) * heads + h) * 128;
  float g1[8], g2[8];
  *reinterpret_cast<float4*>(g1) = *reinterpret_cast<const float4*>(src + 8 * sub);
  *reinterpret_cast<float4*>(g1 + 4) = *reinterpret_cast<const float4*>(src + 8 * sub + 4);
  *reinterpret_cast<float4*>(g2) = *reinterpret_cast<const float4*>(src + 64 + 8 * sub);
  *reinterpret_cast<float4*>(g2 + 4) = *reinterpret_cast<const float4*>(src + 64 + 8 * sub + 4);
  if (h < hq + hkv) {
    float c[8], sv[8], o1[8], o2[8];
    *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cs + size_t(t) * 64 + 8 * sub);
    *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cs + size_t(t) * 64 + 8 * sub + 4);
    *reinterpret_cast<float4*>(sv) = *reinterpret_cast<const float4*>(sn + size_t(t) * 64 + 8 * sub);
    *reinterpret_cast<float4*>(sv + 4) = *reinterpret_cast<const float4*>(sn + size_t(t) * 64 + 8 * sub + 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o1[j] = g1[j] * c[j] + g2[j] * sv[j];
      o2[j] = g2[j] * c[j] - g1[j] * sv[j];
    }
    *reinterpret_cast<uint4*>(dst + 8 * sub) = pack8(o1);
    *reinterpret_cast<uint4*>(dst + 64 + 8 * sub) = pack8(o2);
  } else {
    *reinterpret_cast<uint4*>(dst + 8 * sub) = pack8(g1);
    *reinterpret_cast<uint4*>(dst + 64 + 8 * sub) = pack8(g2);
  }
}

// ------------------------------------------------------------------ SwiGLU
// Bound by HBM; a flat index over the tensor would cost two 64-bit divisions per vector.  kWide: one CTA of 256 threads
// per row (16384 rows, F = 14336: forward 287 -> 243 us, 5.8 TB/s; backward 437 -> 393 us, 6.0 TB/s against the flat
// index; two or four vectors per thread in flight were slower: 259 / 261 and 415 / 434 us).  Otherwise as many rows per
// CTA as fit its threads, and wide rows over several CTAs; see swiglu_launch for the choice.
template <bool kWide>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const uint4* __restrict__ gu, uint4* __restrict__ y, size_t n_rows, int f_vec) {
  const size_t row = kWide ? size_t(blockIdx.x) : size_t(blockIdx.x) * blockDim.y + threadIdx.y;
  if (!kWide && row >= n_rows) return;
  const int first = kWide ? threadIdx.x : blockIdx.y * blockDim.x + threadIdx.x, step = kWide ? 256 : gridDim.y * blockDim.x;
  const uint4* gr = gu + row * 2 * f_vec;
  uint4* yr = y + row * f_vec;
  for (int c = first; c < f_vec; c += step) {
    float g[8], u[8];
    unpack8(gr[c], g);
    unpack8(gr[f_vec + c], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    yr[c] = pack8(g);
  }
}
template <bool kWide>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const uint4* __restrict__ gu, const uint4* __restrict__ dy,
                                                         uint4* __restrict__ dgu, size_t n_rows, int f_vec) {
  const size_t row = kWide ? size_t(blockIdx.x) : size_t(blockIdx.x) * blockDim.y + threadIdx.y;
  if (!kWide && row >= n_rows) return;
  const int first = kWide ? threadIdx.x : blockIdx.y * blockDim.x + threadIdx.x, step = kWide ? 256 : gridDim.y * blockDim.x;
  const uint4* gr = gu + row * 2 * f_vec;
  const uint4* dr = dy + row * f_vec;
  uint4* out = dgu + row * 2 * f_vec;
  for (int c = first; c < f_vec; c += step) {
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(gr[c], g);
    unpack8(gr[f_vec + c], u);
    unpack8(dr[c], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * sg;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (sg + silu * (1.f - sg));
    }
    out[c] = pack8(dg);
    out[f_vec + c] = pack8(du);
  }
}

// ------------------------------------------------------------------ gradients of the head and the embedding
// dst = bf16(src * g) or dst = bf16(dst + bf16(src * g)), g an fp32 scalar on the device: the roundings of an fp32
// product and an accumulation of their own, in one pass
template <bool kAdd>
__global__ void __launch_bounds__(256) scale_rows_kernel(const uint4* __restrict__ src, const float* __restrict__ g,
                                                         uint4* __restrict__ dst, size_t n_vec) {
  const float gv = *g;
  const size_t stride = size_t(gridDim.x) * 256;
  for (size_t i = size_t(blockIdx.x) * 256 + threadIdx.x; i < n_vec; i += stride) {
    float v[8];
    unpack8(src[i], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= gv;
    uint4 out = pack8(v);
    if (kAdd) {
      float a[8];
      unpack8(out, v);
      unpack8(dst[i], a);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += a[j];
      out = pack8(v);
    }
    dst[i] = out;
  }
}

// grad[id] += sum over the tokens with that id of dy[token], fp32 sums.  `ids` sorted, `order` the token at each sorted
// place.  A run of equal ids is cut at every kSegment-th place, and one CTA per (segment, 512 channels) works on it: the
// first place of a segment is the first of a run or a multiple of kSegment.  A run that lies in one segment is added to
// its gradient row at once.  The segments of a longer one leave fp32 sums in `part` (block of kSegment places; 0: from
// the block's start, 1: a run that begins inside it), which embedding_grad_combine_kernel adds in order: one writer per
// gradient row, the same bits in every run, and rows no token names are not touched.
static constexpr int kSegment = 64;

__device__ __forceinline__ void add_rounded(__nv_bfloat16* dst, const float (&acc)[8]) {
  // rounded to bf16 before it is added, as a gradient tensor of its own would be
  uint4* d = reinterpret_cast<uint4*>(dst);
  float old[8], sum[8];
  unpack8(pack8(acc), sum);
  unpack8(*d, old);
#pragma unroll
  for (int e = 0; e < 8; ++e) sum[e] += old[e];
  *d = pack8(sum);
}

__global__ void __launch_bounds__(kSegment) embedding_grad_kernel(const int64_t* __restrict__ ids, const int64_t* __restrict__ order,
                                                                  const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ grad,
                                                                  float* __restrict__ part, int n_tok, int hidden, long vocab) {
  const int i = blockIdx.x, block = i / kSegment, t = threadIdx.x;
  const int64_t id = ids[i];
  const bool first = i == 0 || ids[i - 1] != id;
  if (!(first || i % kSegment == 0) || id < 0 || id >= vocab) return;
  const int stop = min(n_tok, (block + 1) * kSegment);
  // the tokens of the segment, read at once: no gradient row waits for a place and its token first
  __shared__ int64_t token[kSegment];
  const bool in = i + t < stop && ids[i + t] == id;
  if (in) token[t] = order[i + t];
  const int n = __syncthreads_count(in);
  const bool more = stop < n_tok && ids[stop] == id;
  const int c = (blockIdx.y * kSegment + t) * 8;
  if (c >= hidden) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const auto row = [&](int j) { return *reinterpret_cast<const uint4*>(dy + size_t(token[j]) * hidden + c); };
  const auto add = [&](const uint4& raw) {
    float v[8];
    unpack8(raw, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += v[e];
  };
  int j = 0;
  for (; j + 8 <= n; j += 8) {      // eight rows in flight
    uint4 raw[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) raw[k] = row(j + k);
#pragma unroll
    for (int k = 0; k < 8; ++k) add(raw[k]);
  }
#pragma unroll 4
  for (; j < n; ++j) add(row(j));
  if (first && !more) {
    add_rounded(grad + size_t(id) * hidden + c, acc);
  } else {
    float4* dst = reinterpret_cast<float4*>(part + (size_t(block) * 2 + (i % kSegment != 0)) * hidden + c);
    dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
  }
}

// One CTA per (block of places, 512 channels): the run that begins in the block and goes on past its end.  Eight rows of
// 64 threads take every eighth of its sums.
__global__ void __launch_bounds__(512) embedding_grad_combine_kernel(const int64_t* __restrict__ ids, const float* __restrict__ part,
                                                                     __nv_bfloat16* __restrict__ grad, int n_tok, int hidden, long vocab) {
  const int block = blockIdx.x, next = (block + 1) * kSegment;
  if (next >= n_tok) return;
  const int64_t id = ids[next];
  if (ids[next - 1] != id || id < 0 || id >= vocab) return;
  const bool whole = ids[block * kSegment] == id;          // the run covers the block from its start
  if (whole && block > 0 && ids[block * kSegment - 1] == id) return;   // and began before it
  int n = 1;                                               // blocks the run has a sum in
  for (long b = block + 1;; b += 512) {
    const long place = (b + threadIdx.x) * kSegment;
    const int k = __syncthreads_count(place < n_tok && ids[place] == id);
    n += k;
    if (k < 512) break;
  }
  const int lane = threadIdx.x & 63, row = threadIdx.x >> 6, c = (blockIdx.y * 64 + lane) * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  __shared__ float sums[8][64][9];
  if (c < hidden) {
#pragma unroll 4
    for (int k = row; k < n; k += 8) {
      const float4* src = reinterpret_cast<const float4*>(part + (size_t(block + k) * 2 + (k == 0 && !whole)) * hidden + c);
      const float4 x = src[0], y = src[1];
      acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
      acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sums[row][lane][e] = acc[e];
  }
  __syncthreads();
  if (row == 0 && c < hidden) {
    for (int r = 1; r < 8; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += sums[r][lane][e];
    add_rounded(grad + size_t(id) * hidden + c, acc);
  }
}

// ------------------------------------------------------------------ cross entropy (loss + dlogits)
// one CTA per row; vocab must be a multiple of 8.  Rows whose label is < 0 are ignored
// (loss 0, zero gradient).  dlogits overwrite logits: (softmax - onehot) * grad_scale.
// The logits are read twice and overwritten, so the rows under way should stay in L2 until they are read again.  With 256
// threads 1184 rows are under way, with 1024 threads 296: 1024 from 49152 classes on, where 1184 rows fill L2 (4096 rows
// of 128256: 517 -> 471 us, of 65536: 264 -> 248, of 50304: 203 -> 199).  Below that 256 threads, which hide latency across
// rows better (4096 rows of 40008: 164 against 168 us, of 32768: 125 / 139), unless all rows are under way at once
// anyway: then 1024 threads read a row faster (1184 rows of 40008: 53 against 59 us, of 32768: 45 / 47; of 16384 no
// more: 31 / 25).
template <int kThreads>
__global__ void __launch_bounds__(kThreads) cross_entropy_kernel(__nv_bfloat16* __restrict__ logits,
                                                            const int64_t* __restrict__ labels,
                                                            float* __restrict__ loss, int vocab, float grad_scale) {
  __shared__ float scratch[kThreads / 32];
  const size_t row = blockIdx.x;
  uint4* lr = reinterpret_cast<uint4*>(logits + row * vocab);
  const int n_vec = vocab / 8;
  const long label = labels[row];
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < n_vec; i += kThreads) {
    float v[8];
    unpack8(lr[i], v);
    float lm = v[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, v[j]);
    const float nm = fmaxf(m, lm);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += __expf(v[j] - nm);
    s = s * __expf(m - nm) + acc;
    m = nm;
  }
  const float gm = block_max<kThreads / 32>(m, scratch);
  s = block_sum<kThreads / 32>(s * __expf(m - gm), scratch);
  const float lse = gm + __logf(s);
  if (threadIdx.x == 0) {
    float l = 0.f;
    if (label >= 0) l = lse - __bfloat162float(logits[row * vocab + label]);
    loss[row] = l;
  }
  __syncthreads();  // the label logit is read before anyone overwrites it
  const float scale = label >= 0 ? grad_scale : 0.f;
  for (int i = threadIdx.x; i < n_vec; i += kThreads) {
    float v[8];
    unpack8(lr[i], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(v[j] - lse);
      if (long(i) * 8 + j == label) p -= 1.f;
      v[j] = p * scale;
    }
    lr[i] = pack8(v);
  }
}

// ------------------------------------------------------------------ AdamW on a flat shard
__global__ void adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                             const float* __restrict__ grad, __nv_bfloat16* __restrict__ param_bf16, size_t n,
                             float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2,
                             const float* __restrict__ clip_coef) {
  const float clip = clip_coef ? *clip_coef : 1.f;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    const float g = grad[i] * clip;
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    float p = master[i];
    p -= lr * (mi / bc1 / (sqrtf(vi / bc2) + eps) + wd * p);
    m[i] = mi; v[i] = vi; master[i] = p;
    param_bf16[i] = __float2bfloat16(p);
  }
}

}  // namespace dcpk

using namespace dcpk;
#define STREAM static_cast<cudaStream_t>(stream)
#define LAUNCH_OK (cudaGetLastError() == cudaSuccess ? 0 : -5)

extern "C" int dcpk_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int n_rows, int hidden, float eps,
                                void* stream) {
  if (n_rows <= 0) return 0;
  auto X = static_cast<const __nv_bfloat16*>(x); auto W = static_cast<const __nv_bfloat16*>(w);
  auto Y = static_cast<__nv_bfloat16*>(y);
  switch (hidden) {
    case 1024: rmsnorm_fwd_kernel<1><<<n_rows, 128, 0, STREAM>>>(X, W, Y, rstd, hidden, eps); break;
    case 2048: rmsnorm_fwd_kernel<2><<<n_rows, 128, 0, STREAM>>>(X, W, Y, rstd, hidden, eps); break;
    case 4096: rmsnorm_fwd_kernel<4><<<n_rows, 128, 0, STREAM>>>(X, W, Y, rstd, hidden, eps); break;
    case 8192: rmsnorm_fwd_kernel<8><<<n_rows, 128, 0, STREAM>>>(X, W, Y, rstd, hidden, eps); break;
    default: return -3;
  }
  return LAUNCH_OK;
}

// residual: null, or bf16 [n_rows, hidden] that is added to dx
extern "C" int dcpk_rmsnorm_bwd_add(const void* x, const void* w, const void* dy, const float* rstd, void* dx, float* dw,
                                    const void* residual, int n_rows, int hidden, void* stream) {
  if (n_rows <= 0) return 0;
  auto X = static_cast<const __nv_bfloat16*>(x); auto W = static_cast<const __nv_bfloat16*>(w);
  auto G = static_cast<const __nv_bfloat16*>(dy); auto DX = static_cast<__nv_bfloat16*>(dx);
  auto R = static_cast<const __nv_bfloat16*>(residual);
  // Persistent CTAs: at most as many as are resident at once (registers decide), so no CTA waits for a slot while
  // others already finished their share.  Fewer where there are few rows: a CTA's chain of rows grows with rows / CTAs,
  // and the additions to each line of dW with the CTAs, so the best count grows with the root of the rows.  Counts from
  // 32 to 1332 timed at 1 to 16384 rows are best at 6.5 roots (rows of 8192, which take twice as long: 9.3), us against as
  // many CTAs as rows or residents: 256 rows of 1024 10 / 12, 2048 of 1024 17 / 33, 1024 of 4096 18 / 20, 512 of 8192 22 / 23.
  auto launch = [&](auto kernel, float per_root) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, 0) != cudaSuccess || per_sm < 1) per_sm = 2;
    const int root = int(per_root * sqrtf(float(n_rows)) + 0.5f), want = root < 64 ? 64 : root, cap = want < 148 * per_sm ? want : 148 * per_sm;
    kernel<<<n_rows < cap ? n_rows : cap, 128, 0, STREAM>>>(X, W, G, rstd, DX, dw, R, n_rows, hidden);
  };
  const auto sized = [&](auto plain, auto with_residual, float per_root) {
    if (R) launch(with_residual, per_root);
    else launch(plain, per_root);
  };
  switch (hidden) {
    case 1024: sized(rmsnorm_bwd_kernel<1, false>, rmsnorm_bwd_kernel<1, true>, 6.5f); break;
    case 2048: sized(rmsnorm_bwd_kernel<2, false>, rmsnorm_bwd_kernel<2, true>, 6.5f); break;
    case 4096: sized(rmsnorm_bwd_kernel<4, false>, rmsnorm_bwd_kernel<4, true>, 6.5f); break;
    case 8192: sized(rmsnorm_bwd_kernel<8, false>, rmsnorm_bwd_kernel<8, true>, 9.3f); break;
    default: return -3;
  }
  return LAUNCH_OK;
}

extern "C" int dcpk_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, void* dx, float* dw,
                                int n_rows, int hidden, void* stream) {
  return dcpk_rmsnorm_bwd_add(x, w, dy, rstd, dx, dw, nullptr, n_rows, hidden, stream);
}

extern "C" int dcpk_qkv_rope_split_fwd(const void* qkv, const float* cs, const float* sn, void* q_out, void* kv_out,
                                       int n_tok, int hq, int hkv, int q_row0, int kv_row0, void* stream) {
  if (n_tok <= 0) return 0;
  const long items = long(n_tok) * (hq + 2 * hkv);   // eight threads per (token, head)
  const long blocks = (items * 8 + 255) / 256;
  qkv_rope_split_fwd_kernel<<<unsigned(blocks), 256, 0, STREAM>>>(
      static_cast<const __nv_bfloat16*>(qkv), cs, sn, static_cast<__nv_bfloat16*>(q_out),
      static_cast<__nv_bfloat16*>(kv_out), n_tok, hq, hkv, q_row0, kv_row0);
  return LAUNCH_OK;
}

extern "C" int dcpk_qkv_rope_pack_bwd(const float* dq, const float* dkv, const float* cs, const float* sn, void* dqkv,
                                      int n_tok, int hq, int hkv, int q_row0, int kv_row0, void* stream) {
  if (n_tok <= 0) return 0;
  const long items = long(n_tok) * (hq + 2 * hkv);   // eight threads per (token, head)
  const long blocks = (items * 8 + 255) / 256;
  qkv_rope_pack_bwd_kernel<<<unsigned(blocks), 256, 0, STREAM>>>(dq, dkv, cs, sn, static_cast<__nv_bfloat16*>(dqkv),
                                                                  n_tok, hq, hkv, q_row0, kv_row0);
  return LAUNCH_OK;
}

// Grid and block of a SwiGLU pass.  A CTA per row pays when at least half of its 256 threads have work (32768 rows of
// F = 1024, backward: 59 us, two rows per CTA 64) and the rows fill the GPU twice (148 x 8 CTAs at once).  Narrower rows share a CTA (32768 rows of F = 64, forward:
// 25 us with a CTA per row, 10 so), few wide ones are cut into pieces of 256 vectors (64 rows of F = 14336: 14 us / 8).
static bool swiglu_launch(long n_rows, int f_vec, dim3* grid, dim3* block) {
  const long full = 148 * 8 * 2;
  if (f_vec >= 128 && n_rows >= full) {
    *grid = dim3(unsigned(n_rows));
    *block = dim3(256);
    return true;
  }
  const int tx = f_vec < 256 ? f_vec : 256, ty = 256 / tx;
  const long gx = (n_rows + ty - 1) / ty, pieces = (f_vec + tx - 1) / tx, want = (full + gx - 1) / gx;
  *grid = dim3(unsigned(gx), unsigned(pieces < want ? pieces : want));
  *block = dim3(unsigned(tx), unsigned(ty));
  return false;
}

extern "C" int dcpk_swiglu_fwd(const void* gu, void* y, long n_rows, int f, void* stream) {
  if (n_rows <= 0 || f == 0) return 0;
  if (f < 0 || f % 8 != 0 || n_rows / (f >= 1024 ? 1 : 2) > 0x7fffffffl) return -3;   // narrower rows share a CTA
  dim3 grid, block;
  auto kernel = swiglu_launch(n_rows, f / 8, &grid, &block) ? swiglu_fwd_kernel<true> : swiglu_fwd_kernel<false>;
  kernel<<<grid, block, 0, STREAM>>>(static_cast<const uint4*>(gu), static_cast<uint4*>(y), size_t(n_rows), f / 8);
  return LAUNCH_OK;
}

extern "C" int dcpk_swiglu_bwd(const void* gu, const void* dy, void* dgu, long n_rows, int f, void* stream) {
  if (n_rows <= 0 || f == 0) return 0;
  if (f < 0 || f % 8 != 0 || n_rows / (f >= 1024 ? 1 : 2) > 0x7fffffffl) return -3;   // narrower rows share a CTA
  dim3 grid, block;
  auto kernel = swiglu_launch(n_rows, f / 8, &grid, &block) ? swiglu_bwd_kernel<true> : swiglu_bwd_kernel<false>;
  kernel<<<grid, block, 0, STREAM>>>(static_cast<const uint4*>(gu), static_cast<const uint4*>(dy), static_cast<uint4*>(dgu),
                                     size_t(n_rows), f / 8);
  return LAUNCH_OK;
}

// n elements (multiple of 8), both pointers 16-byte aligned; add = 1: accumulate into dst
extern "C" int dcpk_scale_rows(const void* src, const float* g, void* dst, long n, int add, void* stream) {
  if (n <= 0) return 0;
  if (n % 8 != 0) return -3;
  const size_t n_vec = size_t(n) / 8, blocks = (n_vec + 255) / 256;
  const int grid = int(blocks < 148 * 8 ? blocks : 148 * 8);
  if (add) scale_rows_kernel<true><<<grid, 256, 0, STREAM>>>(static_cast<const uint4*>(src), g, static_cast<uint4*>(dst), n_vec);
  else scale_rows_kernel<false><<<grid, 256, 0, STREAM>>>(static_cast<const uint4*>(src), g, static_cast<uint4*>(dst), n_vec);
  return LAUNCH_OK;
}

// part: fp32 [2 * ceil(n_tok / 64), hidden] of scratch, not read before it is written
extern "C" int dcpk_embedding_grad(const void* ids, const void* order, const void* dy, void* grad, float* part, int n_tok, int hidden,
                                   long vocab, void* stream) {
  if (n_tok <= 0) return 0;
  if (hidden % 8 != 0 || hidden <= 0) return -3;
  const unsigned slices = unsigned((hidden + 511) / 512), blocks = unsigned((n_tok + kSegment - 1) / kSegment);
  embedding_grad_kernel<<<dim3(unsigned(n_tok), slices), kSegment, 0, STREAM>>>(
      static_cast<const int64_t*>(ids), static_cast<const int64_t*>(order), static_cast<const __nv_bfloat16*>(dy),
      static_cast<__nv_bfloat16*>(grad), part, n_tok, hidden, vocab);
  if (blocks > 1)
    embedding_grad_combine_kernel<<<dim3(blocks - 1, slices), 512, 0, STREAM>>>(
        static_cast<const int64_t*>(ids), part, static_cast<__nv_bfloat16*>(grad), n_tok, hidden, vocab);
  return LAUNCH_OK;
}

extern "C" int dcpk_cross_entropy(void* logits, const void* labels, float* loss, int n_rows, int vocab, float grad_scale,
                                  void* stream) {
  if (n_rows <= 0) return 0;
  if (vocab % 8 != 0) return -3;
  auto launch = [&](auto kernel, int threads) {
    kernel<<<n_rows, threads, 0, STREAM>>>(static_cast<__nv_bfloat16*>(logits), static_cast<const int64_t*>(labels), loss,
                                           vocab, grad_scale);
  };
  if (vocab >= 49152 || (vocab >= 32768 && n_rows <= 148 * 8)) launch(cross_entropy_kernel<1024>, 1024);
  else launch(cross_entropy_kernel<256>, 256);
  return LAUNCH_OK;
}

extern "C" int dcpk_adamw(float* master, float* m, float* v, const float* grad, void* param_bf16, long n, float lr,
                          float beta1, float beta2, float eps, float wd, int step, const float* clip_coef,
                          void* stream) {
  if (n <= 0) return 0;
  const float bc1 = 1.f - powf(beta1, float(step)), bc2 = 1.f - powf(beta2, float(step));
  adamw_kernel<<<148 * 8, 256, 0, STREAM>>>(master, m, v, grad, static_cast<__nv_bfloat16*>(param_bf16), size_t(n), lr,
                                            beta1, beta2, eps, wd, bc1, bc2, clip_coef);
  return LAUNCH_OK;
}

// ------------------------------------------------------------------ allocation-free RMSNorm backward
// See noalloc.h.  The fp32 weight-gradient accumulator the regular entry point takes from its
// caller lives here, in a file-scope device array, so callers that must not allocate can still
// run the backward pass.
#include "noalloc.h"

static __device__ __align__(256) float g_noalloc_dw_accum[DCPK_NOALLOC_MAX_HIDDEN];

namespace dcpk {
static constexpr int kNoallocMaxDevices = 64;
// device address of g_noalloc_dw_accum per device; in host code the array's name is only a
// handle, the address a kernel can use comes from cudaGetSymbolAddress
static float* g_noalloc_accum_ptr[kNoallocMaxDevices] = {nullptr};

__global__ void dw_accum_to_bf16_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dw, int hidden) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < hidden) dw[i] = __float2bfloat16(acc[i]);
}
}  // namespace dcpk

extern "C" int dcpk_rmsnorm_bwd_noalloc(const void* x, const void* w, const void* dy, const float* rstd, void* dx,
                                        void* dw_bf16, int n_rows, int hidden, void* stream) {
  if (hidden > DCPK_NOALLOC_MAX_HIDDEN || (hidden != 1024 && hidden != 2048 && hidden != 4096 && hidden != 8192)) {
    fprintf(stderr, "dcpk_rmsnorm_bwd_noalloc: hidden=%d is not supported (1024, 2048, 4096 or 8192, at most %d)\n",
            hidden, DCPK_NOALLOC_MAX_HIDDEN);
    return -3;
  }
  if (n_rows < 0) return -3;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices) return -6;
  if (g_noalloc_accum_ptr[dev] == nullptr) {
    float* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_dw_accum) != cudaSuccess || p == nullptr) return -6;
    g_noalloc_accum_ptr[dev] = p;
  }
  float* accum = g_noalloc_accum_ptr[dev];
  // the array keeps what the previous call left: clear the part this call accumulates into
  if (cudaMemsetAsync(accum, 0, size_t(hidden) * sizeof(float), STREAM) != cudaSuccess) return -6;
  if (n_rows > 0) {
    const int rc = dcpk_rmsnorm_bwd(x, w, dy, rstd, dx, accum, n_rows, hidden, stream);
    if (rc != 0) return rc;
  }
  dw_accum_to_bf16_kernel<<<(hidden + 255) / 256, 256, 0, STREAM>>>(accum, static_cast<__nv_bfloat16*>(dw_bf16), hidden);
  return LAUNCH_OK;
}
