// Blockwise range-masked attention backward for sm_100a.
//
// One CTA owns one 128-row KV tile of one KV head and walks a host-built list of 128-query
// tiles that attend to it, once per query head it is responsible for (all heads of the GQA group, or a
// part of them: see heads_per_cta).  Scores are computed in the transposed orientation (lane = key row):
//   S^T  = K  Q^T     (SS UMMA 128x128, K=d)                               -> TMEM
//   dP^T = V  dO^T    (SS)                                                  -> TMEM
//   P^T  = exp2(S^T*c - lse),  dS^T = P^T o (dP^T - delta) * scale          (16 gradient warps)
//   dV  += P^T  dO    (TS, P^T as packed bf16 in the TMEM columns S^T came from)
//   dK  += dS^T Q     (TS, dS^T as packed bf16 in the TMEM columns dP^T came from)
//   dQ   = dS   K     (SS, A = dS^T in shared memory, read MN-major)         -> the TMEM columns of dP^T, behind dK
// TMEM (512 columns): S^T / P^T [0,128)  dP^T / dS^T / dQ [128,256)  dK [256,384)  dV [384,512).
// Per item t the issuer emits  S(t+1) | dK(t) dQ(t) | dP(t+1) | dV(t+1):  the exponentials of t+1 run
// under dK(t) / dQ(t), and dS(t+1) under dV(t+1) and S(t+2).  dK comes before dQ, which overwrites its A
// operand.  With dS^T in TMEM the product dK takes 64 instead of 72 cycles per UMMA and leaves 256 wavefronts per
// item of shared memory to others.  The gradient warps wait twice per item, where it was five times: the statistics
// of the queries arrive on the barriers of S and dP, and dP says that dQ of the item before is done with dS^T.  Both
// together (8192 queries x 16384 keys, one box, long runs): full 5.59 -> 5.41 ms, causal 4.23 -> 4.09, sink + window
// 1.49 -> 1.47; each alone up to 1 %.
// Warps: 0-15 gradient (warp = 32 key rows x 32 queries), 16-23 drain dQ (thread = 64 channels of a query row; a
// [32 queries x 32 channels] fp32 tile per step, added to the accumulator with one tiled TMA
// reduce-add, or to a peer's with a 128-byte bulk reduce-add per row), 24 TMA producer, 25 UMMA issuer, 26
// per-query statistics, 27 idle.  dK/dV stay in TMEM for the CTA's lifetime and are added once,
// through shared memory with tiled TMA reduce-adds (with red.global.add.v4.f32, a row per lane, L2 took 11000 cycles
// for the 128 KB of a key tile, 7000 now: one visit per CTA 15.4 -> 13.1 us per wave, 18944 keys x 1024 queries, 8
// heads, 256 -> 232 us, with 64 channels 180 -> 172; what is left of it is L2's rate of fp32 additions, 20 bytes per
// cycle and SM); the CTAs of a split head group first add their shares up through distributed shared memory, in the
// order of their heads, so that an element has one adder and the same bits in every run (with an atomic addition per
// CTA, three and more of them gave other last bits each time).  dQ is added to by every key tile as it comes, in short
// launches through buffers of at most two additions each, which are summed afterwards (see attn_levels.cuh): these give
// the same bits in every run, the last bits of longer ones differ.
//
// Why 128 x 128: a UMMA with N = 64 occupies the tensor pipe almost as long as one with N = 128 (61 and 72
// cycles with both operands in shared memory, 64 with A in TMEM), so with 64-query items three of the five
// products ran at half rate.  The issuer is one thread, taken by elect.sync: with a test on the lane number
// each UMMA took about 90 cycles to issue (128 x 128 tiles: 839 against 1053 TFLOP/s).  Its descriptors cost an
// addition of 32 bits each, and it asks for operands that are long there while it has something to issue: an answer
// takes 200 cycles and more, behind the exponentials of the warps that share its scheduler (full 5.52 -> 5.45 ms,
// causal 4.18 -> 4.13, sink + window 1.52 -> 1.51 in long runs; 1000 queries x 2100 keys, causal, 101 -> 99 us).
// Handing dS^T to dK before it is stored for dQ costs more registers than it gains time (5.69 ms).  16 gradient warps
// of 32 queries instead of 8 of 64: the unrolled loops of 8 warps did not stay in the instruction cache (5 of
// 13 stall cycles per issue; 0.5 of 19 now).  8 drain warps keep their part of dQ in registers, so the columns
// are free before the shared-memory tile and the L2 have taken it (4 warps with half of it at a time: 7 % slower).
// What bounds it now: an item takes 4100 to 4300 cycles for 2600 of tensor time, and the chain dS(t), dK(t), dQ(t), dQ
// to registers, dP(t+1) is as long, because dP, dS and dQ share 128 TMEM columns.  L2 adds 64 KB of dQ in 2900 cycles
// when all SMs add to tiles that are there (4300 when they are not), and shared memory moves 2048 wavefronts of UMMA
// operands and about 1900 of loads and stores; without the dQ drain an item takes 15 % less.  Not what bounds it: the
// broadcast reads of lse and delta (as a product of their own, three bf16 terms each: 4.85 -> 4.95 ms, and no faster
// with that product left out), the conversions to bf16 (left out: the same), the order of a CTA's queries (reversed:
// the same).  In long runs the power limit holds the clock at 1.3 to 1.6 GHz.  Not tried: a pair of CTAs for 256 keys
// (cta_group::2), which would add half as much to dQ.  It needs Q, dO and K in two layouts, by count 208 KB of shared
// memory per CTA: K and V 32 each, K for dQ 32, Q and dO for S and dP 16 each, for dK and dV 16 each, dS for dQ 32, dQ
// staging 16.
// Measured (8192 queries x 16384 keys, 32 / 8 heads, against 64-query items): full 6.68 -> 4.98 ms (1104 TFLOP/s),
// causal 4.99 -> 3.77 ms (1095), sink + window 1.84 -> 1.38 ms (1009).
//
// The first `n_copy_rows` rows of the grid are fetch CTAs: they compute nothing and bring the next plan
// stage's remote operands (Q, dO, KV rows and the lse / delta statistics of the queries) from peer
// GPUs into this GPU's staging rows (copy_jobs.cuh) while the other CTAs of the same launch work
// through the items; they are scheduled first and retire after about a millisecond.
//
// Reference behaviour covered: the varlen backward the executor calls at
// dcp/runtime/flash_attention/executor.py:1058-1115, plus the blockwise partial sums
// that follow it (dcp/ops/fused_ops.py:1087-1360), which the atomics make unnecessary.
#include <limits.h>
#include <math.h>
#include <stddef.h>

#include <algorithm>

#include "attn_common.cuh"
#include "attn_levels.cuh"
#include "copy_jobs.cuh"
#include "entries.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "smem_limit.h"
#include "tmap.cuh"

namespace dcpk {

static constexpr int kBwdThreads = 896;  // 16 gradient warps, 8 drain warps, TMA producer, UMMA issuer, statistics, 1 idle
static constexpr int kQTile = 128;            // query rows per item
static constexpr int kHalf = 128 * 64 * 2;  // [128 x 64] bf16 half tile, 16 KB

struct BwdItem {  // descriptor + the query head of the current visit
  int q_row, n_rows, head, kv_pos0, mask_row, dq_dev, dq_row, full;
};

struct BwdCta {
  int kv_row;    // arena row of the 128-key tile
  int n_valid;   // valid keys
  int item_off, n_items;
  int dkv_dev, dkv_row;
  int pad0, pad1;
};

__device__ __forceinline__ BwdItem load_item(const BwdItemDesc* descs, int visit, int heads, int head0) {
  const BwdItemDesc d = descs[visit / heads];
  BwdItem it;
  it.q_row = d.q_row; it.n_rows = d.n_rows; it.head = head0 + visit % heads; it.kv_pos0 = d.kv_pos0;
  it.mask_row = d.mask_row; it.dq_dev = d.dq_dev; it.dq_row = d.dq_row; it.full = d.full;
  return it;
}

// table sanity of one item, checked before anything it points at is read
__device__ __forceinline__ bool item_ok(const BwdItem& it, int q_rows, int stat_stride, int n_dst, int n_mask_rows) {
  return !(it.n_rows < 0 || it.n_rows > kQTile || it.q_row < 0 || it.q_row + it.n_rows > q_rows ||
           it.q_row + it.n_rows > stat_stride || it.dq_dev >= n_dst || it.mask_row < 0 ||
           (!it.full && it.mask_row + it.n_rows > n_mask_rows) ||
           (it.dq_dev >= 0 && (it.dq_row < 0 || it.dq_row + it.n_rows > q_rows)));
}

struct BwdPtrs {
  float* dq[kMaxPeers];   // fp32 [rows, hq, d]
  float* dkv[kMaxPeers];  // fp32 [rows, 2, hkv, d]
};

// Exactly 227 KB: two Q tiles (S(t+1) runs before dK(t)), one dO tile (it is read by two adjacent products).
struct __align__(1024) BwdSmem {
  uint8_t k[2 * kHalf];
  uint8_t v[2 * kHalf];
  uint8_t q[2][2 * kHalf];
  uint8_t dout[2 * kHalf];
  uint8_t ds[2 * kHalf];            // dS^T: [128 keys x 128 queries], two halves of 64 queries
  float dq_stage[8][32 * 32];       // per drain warp: [32 queries x 32 channels], 128-byte swizzled
  // per-query statistics in the form the packed-fp32 math consumes them: -lse * log2(e) (-inf for rows
  // past the tile) and -delta * scale; ranges clamped to the key tile, one byte per bound
  alignas(16) float nlse[2][kQTile];
  uint32_t rng[2][kQTile];
  alignas(16) float ndelta[kQTile];
  uint64_t kv_full, q_full[2], q_empty[2], do_full, do_empty, s_full[2], p_ready, dp_full,
      ds_ready, dq_full, dq_drained, acc_full;
  int fast[2];                      // item of the stage needs no masking at all
  uint32_t tmem_base;
  int abort_word;
};

// Optional per-phase cycle counters of CTA (0,0) (set with dcpk_attn_bwd_set_timeline; null = off).
// Layout: [phase][sum of cycles]; phases 0-6 gradient warp 0, 7-15 UMMA warp.  The counters live in
// a separately instantiated kernel (kTL) so the production kernel carries no probe branches; each
// phase includes the cost of one probe (about 110 cycles).
__device__ long long* g_bwd_timeline = nullptr;
static_assert(offsetof(BwdSmem, dout) == 256 * kHeadDim * sizeof(float), "K, V and Q tiles hold a gradient share");
#define TL_ADD(idx, t_prev)                                                        \
  do {                                                                             \
    if constexpr (kTL) if (tl) { long long now_ = clock64(); if (lane == 0 || warp == 25) atomicAdd(reinterpret_cast<unsigned long long*>(tl + (idx)), (unsigned long long)(now_ - (t_prev))); (t_prev) = now_; } \
  } while (0)

__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// row `row` (0-127 dK, 128-255 dV) of a CTA's gradient share: 128 floats, 16-byte pieces swizzled by the row
__device__ __forceinline__ float* share_of(BwdSmem& sm, int row) { return reinterpret_cast<float*>(sm.k) + row * kHeadDim; }

// lane i holds row i of a 32 x 32 bit matrix; afterwards lane i holds column i
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1) {
    const uint32_t low = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~low) | ((y >> j) & low)) : ((x & low) | ((y & low) << j));
  }
  return x;
}

// the 32 keys [key0, key0 + 32) of the tile one query sees, from its packed ranges
__device__ __forceinline__ uint32_t visible_keys(uint32_t rng, int key0) {
  return bits_between(int(rng & 0xff) - key0, int((rng >> 8) & 0xff) - key0) |
         bits_between(int((rng >> 16) & 0xff) - key0, int(rng >> 24) - key0);
}

// P = exp2(S * c - lse) of one key row and 32 queries, in place, and its packed bf16 pairs
template <bool kMasked>
__device__ __forceinline__ void grad_probs(uint32_t* s, uint32_t* packed, const float* nlse, uint64_t sl2_2, uint32_t see) {
  const ulonglong2* nl = reinterpret_cast<const ulonglong2*>(nlse);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const ulonglong2 n = nl[c];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 4 * c + 2 * h;
      const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sl2_2, h ? n.y : n.x);
      float x0, x1;
      unpack_f32x2(x2, x0, x1);
      float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
      if (kMasked) {
        p0 = (see >> e) & 1u ? p0 : 0.f;
        p1 = (see >> (e + 1)) & 1u ? p1 : 0.f;
      }
      s[e] = __float_as_uint(p0); s[e + 1] = __float_as_uint(p1);
      packed[e >> 1] = pack_bf16x2(p0, p1);
    }
  }
}

// dS = P * (dP * scale - delta * scale) of 16 queries, packed bf16 pairs
template <bool kMasked>
__device__ __forceinline__ void grad_scores(const uint32_t* p, const uint32_t* dp, uint32_t* packed, const float* ndelta,
                                            uint64_t scale_2, uint32_t see) {
  const ulonglong2* nd = reinterpret_cast<const ulonglong2*>(ndelta);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const ulonglong2 n = nd[c];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 4 * c + 2 * h;
      const uint64_t g2 = fma_f32x2(pack_f32x2(__uint_as_float(dp[e]), __uint_as_float(dp[e + 1])), scale_2, h ? n.y : n.x);
      float d0, d1;
      unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(p[e]), __uint_as_float(p[e + 1])), g2), d0, d1);
      if (kMasked) {   // a masked pair is an exact zero whatever its dP is
        d0 = (see >> e) & 1u ? d0 : 0.f;
        d1 = (see >> (e + 1)) & 1u ? d1 : 0.f;
      }
      packed[e >> 1] = pack_bf16x2(d0, d1);
    }
  }
}

// kD: channels that are computed.  The arenas' rows have 128; heads of fewer are zero-padded there, and products over
// zeros and accumulators of zeros are left out: for up to 64 channels half of S and dP (K steps), half of dK, dV and dQ
// (N) and of their traffic; for up to 96 a quarter of S, dP and the drain of dQ (N stays 128: an operand that is not
// K-major comes in 64s).  8192 queries x 16384 keys, 32 / 8 heads, causal, against all 128 channels: 64 channels 3.56
// -> 2.61 ms, 96 channels 3.99 -> 3.45 ms; 1000 x 2100: 110 -> 83 us and 122 -> 110 us.
template <bool kTL, int kD>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_kv, const __grid_constant__ CUtensorMap tm_dq,
                const __grid_constant__ CUtensorMap tm_dkv, const __grid_constant__ CUtensorMap tm_levels, int n_levels,
                const BwdCta* __restrict__ ctas, const BwdItemDesc* __restrict__ items, const int4* __restrict__ masks,
                const float* __restrict__ lse, const float* __restrict__ delta, BwdPtrs ptrs, int hq, int hkv,
                int heads_per_cta, int stat_stride, int n_dst, int q_rows, int kv_rows, int n_mask_rows, int n_items_total,
                float scale, const CopyJob* __restrict__ jobs, int n_jobs, const __grid_constant__ CopyCtx copy_ctx,
                int n_copy_rows, int* __restrict__ status) {
  grid_let_next();
  grid_wait();
  if (int(blockIdx.y) < n_copy_rows) {
    // ------------------------------------------------------------ operand fetch for the next stage
    run_copy_jobs(jobs, n_jobs, copy_ctx, blockIdx.y * gridDim.x + blockIdx.x, n_copy_rows * gridDim.x, threadIdx.x,
                  kBwdThreads);
    return;
  }
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BwdSmem& sm = *reinterpret_cast<BwdSmem*>(smem_raw);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // grid = (kv heads x parts of the head group, key tiles): neighbouring CTAs share the item list and the mask rows
  const BwdCta cta = ctas[blockIdx.y - n_copy_rows];
  constexpr int kHalves = kD > 64 ? 2 : 1;   // of 64 channels
  const int group = hq / hkv, parts = group / heads_per_cta;
  const int kv_head = blockIdx.x / parts, head0 = kv_head * group + (blockIdx.x % parts) * heads_per_cta;
  const BwdItemDesc* my_items = items + cta.item_off;
  const int n_items = cta.n_items * heads_per_cta;  // visits
  {
    // table sanity before anything is allocated: a key tile whose gradient rows would fall outside
    // the accumulator, or whose item list runs past the item table, is reported and skipped (items
    // are checked one by one by the warps that read them, mask rows included); shared memory has no room for
    // alignment padding, so its base is checked too
    const bool bad = cta.dkv_dev < 0 || cta.dkv_dev >= n_dst || cta.dkv_row < 0 || cta.n_valid < 0 ||
                     cta.n_valid > 128 || cta.dkv_row + cta.n_valid > kv_rows || cta.kv_row < 0 ||
                     cta.kv_row + cta.n_valid > kv_rows || cta.n_items < 0 || cta.item_off < 0 ||
                     cta.item_off + cta.n_items > n_items_total || (smem_u32(smem_raw) & 1023u);
    if (bad) {
      if (threadIdx.x == 0) atomicExch(status, kStatusBadArgs);
      return;
    }
  }

  if (threadIdx.x == 768) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_kv);
    tma_prefetch_desc(&tm_dq);
    mbar_init(&sm.kv_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.q_full[i], 1); mbar_init(&sm.q_empty[i], 1); mbar_init(&sm.s_full[i], 2); }
    mbar_init(&sm.do_full, 1);
    mbar_init(&sm.do_empty, 1);
    mbar_init(&sm.p_ready, 16);
    mbar_init(&sm.dp_full, 2);
    mbar_init(&sm.ds_ready, 16);
    mbar_init(&sm.dq_full, 1);
    mbar_init(&sm.dq_drained, 8);
    mbar_init(&sm.acc_full, 1);
    sm.abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 25) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  volatile int* abort_word = &sm.abort_word;
  constexpr uint32_t cS = 0, cdP = 128, cdK = 256, cdV = 384;

  long long* tl = (kTL && blockIdx.x == 0 && int(blockIdx.y) == n_copy_rows && (warp == 0 || warp == 25)) ? g_bwd_timeline : nullptr;
  long long tl_t = kTL ? clock64() : 0;
  // registers move from the producer / issuer warpgroup to the drain warps
  // (512 x 72 + 256 x 80 + 128 x 56 = 64512 = 896 x 72, what the block is launched with)
  if (warp >= 24) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 24) {
      // ------------------------------------------------------------ TMA producer
      if (lane == 0) {
        mbar_expect_tx(&sm.kv_full, 2 * kHalves * kHalf);
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {
          tma_load_3d(sm.k + h * kHalf, &tm_kv, &sm.kv_full, 64 * h, kv_head, cta.kv_row);
          tma_load_3d(sm.v + h * kHalf, &tm_kv, &sm.kv_full, 64 * h, hkv + kv_head, cta.kv_row);
        }
      }
      bool ok = true;
      int q_pending[2] = {-1, -1}, do_pending = -1;
      // descriptors are read two visits ahead: a table read never sits between a free buffer and its load
      BwdItem ring[3] = {};
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (i < n_items) ring[i] = load_item(my_items, i, heads_per_cta, head0);
      for (int i = 0; i < n_items && ok; ++i) {
        const int st = i & 1, u = i >> 1;
        const BwdItem itx = ring[0];
        if (i + 2 < n_items) ring[2] = load_item(my_items, i + 2, heads_per_cta, head0);
        if (!item_ok(itx, q_rows, stat_stride, n_dst, n_mask_rows)) {
          sm.abort_word = kStatusBadArgs;  // every waiter unwinds; the code is reported as the status
          ok = false;
          break;
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.q_empty[st], (u & 1) ^ 1, abort_word));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&sm.q_full[st], kHalves * kHalf);
#pragma unroll
          for (int h = 0; h < kHalves; ++h)
            tma_load_3d(sm.q[st] + h * kHalf, &tm_q, &sm.q_full[st], 64 * h, itx.head, itx.q_row);
          q_pending[st] = u & 1;
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.do_empty, (i & 1) ^ 1, abort_word));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(&sm.do_full, kHalves * kHalf);
#pragma unroll
          for (int h = 0; h < kHalves; ++h)
            tma_load_3d(sm.dout + h * kHalf, &tm_do, &sm.do_full, 64 * h, itx.head, itx.q_row);
          do_pending = i & 1;
          // the visit after the next is pulled into L2 now, so that its loads find it there
          const BwdItem& nx = ring[2];
          if (i + 2 < n_items && nx.q_row >= 0 && nx.q_row < q_rows && nx.head < hq) {
#pragma unroll
            for (int h = 0; h < kHalves; ++h) {
              tma_prefetch_l2_3d(&tm_q, 64 * h, nx.head, nx.q_row);
              tma_prefetch_l2_3d(&tm_do, 64 * h, nx.head, nx.q_row);
            }
          }
        }
        ring[0] = ring[1]; ring[1] = ring[2];
      }
      if (!ok && lane == 0) {
        // give copies already in flight a bounded chance to land before the CTA retires
#pragma unroll
        for (int s2 = 0; s2 < 2; ++s2)
          if (q_pending[s2] >= 0)
            for (int spin = 0; spin < 200000 && !mbar_try_wait(&sm.q_full[s2], q_pending[s2]); ++spin) {}
        if (do_pending >= 0)
          for (int spin = 0; spin < 200000 && !mbar_try_wait(&sm.do_full, do_pending); ++spin) {}
      }
    } else if (warp == 26) {
      // ------------------------------------------------------------ per-query statistics
      // The values of a visit are read while the one before it is still being computed, its descriptor one
      // visit earlier still, so no wait of this warp is followed by a trip to global memory.
      struct Stats { float l[4], d[4]; uint32_t rg[4]; int fast; };
      auto fetch = [&](const BwdItem& itx, Stats& s) -> bool {
        if (!item_ok(itx, q_rows, stat_stride, n_dst, n_mask_rows)) return false;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int qi = lane + 32 * h;
          const bool qv = qi < itx.n_rows;
          const size_t si = size_t(itx.head) * stat_stride + itx.q_row + qi;
          s.l[h] = qv ? lse[si] : INFINITY;
          s.d[h] = qv ? delta[si] : 0.f;
          s.rg[h] = 0;
          if (qv && itx.full) {
            s.rg[h] = uint32_t(cta.n_valid) << 8;
          } else if (qv) {
            const int4 m = masks[itx.mask_row + qi];
            const int s0 = min(max(m.x - itx.kv_pos0, 0), 128), e0 = min(max(m.y - itx.kv_pos0, 0), cta.n_valid);
            const int s1 = min(max(m.z - itx.kv_pos0, 0), 128), e1 = min(max(m.w - itx.kv_pos0, 0), cta.n_valid);
            s.rg[h] = uint32_t(s0) | (uint32_t(e0) << 8) | (uint32_t(s1) << 16) | (uint32_t(e1) << 24);
          }
        }
        s.fast = itx.full && itx.n_rows == kQTile && cta.n_valid == 128;
        return true;
      };
      Stats cur{}, nxt{};
      BwdItem it1{};
      bool ok = true;
      if (n_items > 0) ok = fetch(load_item(my_items, 0, heads_per_cta, head0), cur);
      if (n_items > 1) it1 = load_item(my_items, 1, heads_per_cta, head0);
      for (int i = 0; i < n_items && ok; ++i) {
        const int st = i & 1, u = i >> 1;
        if (i + 1 < n_items) ok = fetch(it1, nxt);
        if (i + 2 < n_items) it1 = load_item(my_items, i + 2, heads_per_cta, head0);
        if (!ok) break;   // the TMA producer reports the bad entry
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.q_empty[st], (u & 1) ^ 1, abort_word));
        if (!ok) break;
        if (lane == 0) sm.fast[st] = cur.fast;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          sm.nlse[st][lane + 32 * h] = (cur.l[h] == -INFINITY) ? -INFINITY : -(cur.l[h] * 1.4426950408889634f);
          sm.rng[st][lane + 32 * h] = cur.rg[h];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.s_full[st]);  // release: the stores above are visible to waiters
        // the gradient warps are through with the previous item's delta once its dS is written
        if (i > 0) ok = __all_sync(0xffffffffu, mbar_wait(&sm.ds_ready, (i - 1) & 1, abort_word));
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < 4; ++h) sm.ndelta[lane + 32 * h] = -cur.d[h] * scale;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.dp_full);
        cur = nxt;
      }
    } else if (warp == 25) {
      // ------------------------------------------------------------ UMMA issuer (one thread)
      if (elect_one()) {
        constexpr uint32_t idesc_sdp = make_idesc_bf16(128, 128, 0, 0);
        constexpr uint32_t idesc_acc = make_idesc_bf16(128, 64 * kHalves, 0, 1);
        constexpr uint32_t idesc_dq = make_idesc_bf16(128, 64 * kHalves, 1, 1);
        // descriptors: K-major operands and MN-major ones differ in the leading offset, all others in the address field
        // only
        const uint64_t some = make_sdesc_sw128(0, 16, 1024), some_mn = make_sdesc_sw128(0, kHalf, 1024);
        const uint32_t hi = uint32_t(some >> 32), lo = uint32_t(some), lo_mn = uint32_t(some_mn);
        auto desc = [&](uint32_t low) { return (uint64_t(hi) << 32) | low; };
        const uint32_t k_at = sdesc_addr(sm.k), v_at = sdesc_addr(sm.v), ds_at = sdesc_addr(sm.ds), do_at = sdesc_addr(sm.dout),
                       q_at = sdesc_addr(sm.q[0]);
        constexpr uint32_t kTile = 2 * kHalf >> 4;
        bool ok = mbar_wait(&sm.kv_full, 0, abort_word);
        // D = A B^T, both operands K-major (K = channels)
        auto issue_kk = [&](uint32_t col, uint32_t a_at, uint32_t b_at, uint64_t* done) {
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < kD / 16; ++k) {
            const uint32_t off = (k >> 2) * (kHalf >> 4) + (k & 3) * 2;
            umma_ss(tmem + col, desc(lo + a_at + off), desc(lo + b_at + off), idesc_sdp, k > 0 ? 1u : 0u);
          }
          umma_commit(done);
        };
        auto issue_s = [&](int t, bool there) -> bool {
          if (!there && !mbar_wait(&sm.q_full[t & 1], (t >> 1) & 1, abort_word)) return false;
          TL_ADD(8, tl_t);
          issue_kk(cS, k_at, q_at + (t & 1) * kTile, &sm.s_full[t & 1]);   // P(t-1) was consumed by dV(t-1), issued before
          TL_ADD(12, tl_t);
          return true;
        };
        auto issue_dp = [&](int t, bool there) -> bool {
          if (t > 0 && !mbar_wait(&sm.dq_drained, (t - 1) & 1, abort_word)) return false;
          TL_ADD(10, tl_t);
          if (!there && !mbar_wait(&sm.do_full, t & 1, abort_word)) return false;
          TL_ADD(14, tl_t);
          issue_kk(cdP, v_at, do_at, &sm.dp_full);
          TL_ADD(15, tl_t);
          return true;
        };
        auto issue_dv = [&](int t) -> bool {
          if (!mbar_wait(&sm.p_ready, t & 1, abort_word)) return false;
          TL_ADD(11, tl_t);
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 8; ++k)  // 16 queries per step; P^T: queries 32 i .. 32 i + 31 in columns [32 i, 32 i + 16) of S^T
            umma_ts(tmem + cdV, tmem + cS + (k >> 1) * 32 + (k & 1) * 8, desc(lo_mn + do_at + k * 128), idesc_acc,
                    (t > 0 || k > 0) ? 1u : 0u);
          umma_commit(&sm.do_empty);
          TL_ADD(7, tl_t);
          return true;
        };
        auto issue_dqk = [&](int t) -> bool {
          if (!mbar_wait(&sm.ds_ready, t & 1, abort_word)) return false;
          TL_ADD(9, tl_t);
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 8; ++k)  // 16 queries per step
            umma_ts(tmem + cdK, tmem + cdP + (k >> 1) * 32 + (k & 1) * 8, desc(lo_mn + q_at + (t & 1) * kTile + k * 128), idesc_acc,
                    (t > 0 || k > 0) ? 1u : 0u);
          umma_commit(&sm.q_empty[t & 1]);   // Q(t) is free
#pragma unroll
          for (int k = 0; k < 8; ++k)  // 16 keys per step
            umma_ss(tmem + cdP, desc(lo_mn + ds_at + k * 128), desc(lo_mn + k_at + k * 128), idesc_dq, k > 0 ? 1u : 0u);
          umma_commit(&sm.dq_full);            // and so is the dS^T tile
          TL_ADD(13, tl_t);
          return true;
        };
        if (n_items > 0) {
          ok = ok && issue_s(0, false) && issue_dp(0, false) && issue_dv(0);
          for (int t = 0; t + 1 < n_items && ok; ++t) {
            // an answer takes 200 cycles and more: the operands that are long there are asked for together
            const bool q_there = mbar_test_wait(&sm.q_full[(t + 1) & 1], ((t + 1) >> 1) & 1);
            ok = issue_s(t + 1, q_there);
            if (!ok) break;
            const bool do_there = mbar_test_wait(&sm.do_full, (t + 1) & 1);
            ok = issue_dqk(t) && issue_dp(t + 1, do_there) && issue_dv(t + 1);
          }
          ok = ok && issue_dqk(n_items - 1);
          if (ok) {
            umma_commit(&sm.acc_full);
            mbar_wait(&sm.acc_full, 0, abort_word);   // keep TMEM alive until everything retired
          }
        }
      }
      __syncwarp();
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------ dQ drain: thread = query row
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    // warps 16-19 the first half of the channels, warps 20-23 the others (of 96: 64 and 32)
    constexpr int kMine = kD > 64 ? 2 : 1;   // steps of 32 channels
    const int quad = warp & 3, ch0 = (warp >= 20) * 32 * kMine;
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    bool ok = true;
    BwdItem itx{};
    if (n_items > 0) itx = load_item(my_items, 0, heads_per_cta, head0);
    for (int t = 0; t < n_items && ok; ++t) {
      const BwdItem cur = itx;
      if (t + 1 < n_items) itx = load_item(my_items, t + 1, heads_per_cta, head0);
      const bool any_row = quad * 32 < cur.n_rows && cur.dq_dev >= 0;   // dq_dev < 0: dQ is not wanted
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.dq_full, t & 1, abort_word));
      if (!ok) break;
      tc_fence_after();
      // the warp's part goes to registers as a whole: dP of the next item waits for the columns
      uint32_t reg[32 * kMine];
#pragma unroll
      for (int b = 0; b < kMine; ++b) tmem_ld32(tmem + lane_base + cdP + ch0 + 32 * b, reg + 32 * b);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.dq_drained);
      if (!any_row) continue;
      // this GPU's accumulator takes a swizzled tile with one tiled reduce, any other one 128 bytes of a row per lane
      // (rows past n_rows of the tile hold exact zeros, their probabilities are masked to 0: adding them is harmless)
      float* stage = sm.dq_stage[warp - 16];
      const int swizzle = cur.dq_dev == 0 ? lane & 7 : 0;
#pragma unroll
      for (int b = 0; b < kMine; ++b) {
        if (ch0 + 32 * b >= kD) break;
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // what this lane reduced before has left the buffer
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(stage + lane * 32 + ((c ^ swizzle) << 2)) =
              make_uint4(reg[32 * b + 4 * c], reg[32 * b + 4 * c + 1], reg[32 * b + 4 * c + 2], reg[32 * b + 4 * c + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (cur.dq_dev == 0) {
          if (lane == 0) {
            const int level = dq_level(cur.kv_pos0, n_levels), row = cur.dq_row + quad * 32;
            if (level > 0) tma_reduce_add_3d(&tm_levels, stage, ch0 + b * 32, cur.head, (level - 1) * q_rows + row);
            else tma_reduce_add_3d(&tm_dq, stage, ch0 + b * 32, cur.head, row);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        } else if (quad * 32 + lane < cur.n_rows) {
          float* dq = ptrs.dq[cur.dq_dev] + (size_t(cur.dq_row + quad * 32 + lane) * hq + cur.head) * kHeadDim + ch0 + b * 32;
          asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], 128;"
                       ::"l"(dq), "r"(smem_u32(stage + lane * 32)) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    // no staged dQ tile may still be in flight when the CTA retires (also on the abort path)
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ------------------------------------------------------------ softmax-gradient threads
    // warp w works on TMEM lanes 32*(w&3).. (key rows) and on queries 32*(w>>2)..+31 of every item
    const int quad = warp & 3, hf = warp >> 2;
    const int r = quad * 32 + lane;  // key row inside the tile == TMEM lane
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const uint32_t s_addr = tmem + lane_base + cS + hf * 32, dp_addr = tmem + lane_base + cdP + hf * 32;
    const float sl2 = scale * 1.4426950408889634f;
    const uint64_t sl2_2 = pack_f32x2(sl2, sl2), scale_2 = pack_f32x2(scale, scale);
    uint8_t* ds_row = sm.ds + (hf >> 1) * kHalf + r * 128;
    bool ok = true;
    for (int t = 0; t < n_items && ok; ++t) {
      const int st = t & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.s_full[st], (t >> 1) & 1, abort_word));
      if (!ok) break;
      TL_ADD(0, tl_t);
      // The tile-level "no masking needed" switch is taken once, outside the element loops.  Otherwise
      // every lane turns the ranges of one query into a bit word over the warp's 32 keys, and a bit
      // transpose gives each lane (= key) the 32 queries that see it.
      const bool fast = sm.fast[st];
      uint32_t see = 0;
      if (!fast) see = warp_transpose_bits(visible_keys(sm.rng[st][hf * 32 + lane], quad * 32), lane);
      TL_ADD(1, tl_t);
      tc_fence_after();
      uint32_t p[32];
      tmem_ld32(s_addr, p);
      tmem_wait_ld();
      TL_ADD(2, tl_t);
      {
        uint32_t packed[16];
        if (fast) grad_probs<false>(p, packed, sm.nlse[st] + hf * 32, sl2_2, 0);
        else grad_probs<true>(p, packed, sm.nlse[st] + hf * 32, sl2_2, see);
        tmem_st16(s_addr, packed);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.p_ready);
      TL_ADD(3, tl_t);
      // dP(t) was issued behind dK(t-1) and dQ(t-1), which have finished reading dS^T then
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.dp_full, t & 1, abort_word));
      if (!ok) break;
      TL_ADD(4, tl_t);
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t dp[16], packed[8];
        tmem_ld16(dp_addr + 16 * h, dp);
        tmem_wait_ld();
        if (fast) grad_scores<false>(p + 16 * h, dp, packed, sm.ndelta + hf * 32 + 16 * h, scale_2, 0);
        else grad_scores<true>(p + 16 * h, dp, packed, sm.ndelta + hf * 32 + 16 * h, scale_2, see >> (16 * h));
#pragma unroll
        for (int c = 0; c < 2; ++c)
          *reinterpret_cast<uint4*>(ds_row + ((((hf & 1) * 4 + 2 * h + c) ^ (r & 7)) << 4)) =
              make_uint4(packed[4 * c], packed[4 * c + 1], packed[4 * c + 2], packed[4 * c + 3]);
        tmem_st8(dp_addr + 8 * h, packed);   // over the dP^T columns read above
      }
      tmem_wait_st();
      TL_ADD(5, tl_t);
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.ds_ready);
      TL_ADD(6, tl_t);
    }
    if (ok && n_items > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.acc_full, 0, abort_word));
      if (ok) {
        tc_fence_after();
        // lane = key row; warps 0-7 take dK, warps 8-15 dV, half of the channels each
        constexpr int kMine = kD > 64 ? 2 : 1;   // steps of 32 channels
        const int ch = (hf & 1) * 32 * kMine;
        float* dst = ptrs.dkv[cta.dkv_dev] + ((size_t(cta.dkv_row + r) * 2 + (hf >> 1)) * hkv + kv_head) * kHeadDim + ch;
        const uint32_t acc = tmem + lane_base + (hf >> 1 ? cdV : cdK) + ch;
        // a whole key tile for this GPU's accumulator goes there in boxes of [32 keys x 32 channels], which take the
        // place of K, V and Q; rows that may not be added to, and other GPUs' accumulators, go 16 bytes at a time
        const bool whole = cta.dkv_dev == 0 && cta.n_valid == 128;
#pragma unroll
        for (int c = 0; c < kMine; ++c) {
          if (ch + 32 * c >= kD) break;
          uint32_t reg[32];
          tmem_ld32(acc + 32 * c, reg);
          tmem_wait_ld();
          if (parts > 1) {   // K, V and Q have been read for the last time: their 128 KB take the CTA's share
            float* row = share_of(sm, (hf >> 1) * 128 + r);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(row + (((ch >> 2) + 8 * c + i) ^ (r & 7)) * 4) =
                  make_uint4(reg[4 * i], reg[4 * i + 1], reg[4 * i + 2], reg[4 * i + 3]);
          } else if (whole) {
            uint8_t* box = sm.k + warp * 8192 + c * 4096;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(box + lane * 128 + ((i ^ (lane & 7)) << 4)) =
                  make_uint4(reg[4 * i], reg[4 * i + 1], reg[4 * i + 2], reg[4 * i + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_reduce_add_3d(&tm_dkv, box, ch + 32 * c, (hf >> 1) * hkv + kv_head, cta.dkv_row + quad * 32);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          } else if (r < cta.n_valid) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              red_add_v4(dst + 32 * c + 4 * i, __uint_as_float(reg[4 * i]), __uint_as_float(reg[4 * i + 1]),
                         __uint_as_float(reg[4 * i + 2]), __uint_as_float(reg[4 * i + 3]));
          }
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 25) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (parts > 1) {
    // the CTAs of a split head group (a cluster) add their shares up in the order of their heads, each for a part of
    // the rows: one addition to the accumulator per element, and the same bits in every run
    cluster_sync();
    if (warp < 16) {
      const int rank = blockIdx.x % parts;
      bool all_ok = n_items > 0;   // an empty list leaves no share behind
      for (int p = 0; p < parts; ++p) all_ok = all_ok && ld_cluster_u32(smem_u32(&sm.abort_word), p) == 0;
      if (all_ok)
        for (int row = rank * 16 + warp; row < 256; row += parts * 16) {   // 0-127 dK, 128-255 dV; lane = 4 channels
          const int r = row & 127;
          if (r >= cta.n_valid || 4 * lane >= kD) continue;
          const uint32_t addr = smem_u32(share_of(sm, row) + (lane ^ (r & 7)) * 4);
          float4 sum = ld_cluster_f4(addr, 0);
          for (int p = 1; p < parts; ++p) {
            const float4 v = ld_cluster_f4(addr, p);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
          red_add_v4(ptrs.dkv[cta.dkv_dev] + ((size_t(cta.dkv_row + r) * 2 + (row >> 7)) * hkv + kv_head) * kHeadDim + 4 * lane,
                     sum.x, sum.y, sum.z, sum.w);
        }
    }
    cluster_sync();   // no CTA's shared memory goes away while another reads it
  }
  if (threadIdx.x == 0 && sm.abort_word) atomicExch(status, sm.abort_word);  // 1 = wait timeout, 3 = bad table
}

// The passes over the levels of dQ as launches of their own, plain ones (kSum: they are added to dQ; else they are
// cleared).  Bound by L2.
template <bool kSum>
__global__ void __launch_bounds__(256) dq_levels_kernel(const __grid_constant__ DqLevels lv, float* __restrict__ dq) {
  __shared__ RowLevels present;
  const int row0 = blockIdx.x * kLevelRows;
  grid_let_next();
  grid_wait();
  if (!kSum) {
    clear_levels(lv, row0, present);
    return;
  }
  find_levels(lv, row0, present);
  const int quads = lv.pitch / 4, per_row = lv.hq * quads;
  for (int c = threadIdx.x; c < kLevelRows * per_row; c += 256) {
    const int r = c / per_row, k = c % quads * 4;
    const uint64_t above = levels_above(present, r);
    if (above == 0 || k >= lv.channels) continue;
    const size_t head_row = size_t(row0 + r) * lv.hq + c % per_row / quads;
    float4* acc = reinterpret_cast<float4*>(dq + head_row * kHeadDim + k);
    float4 sum = *acc;
    add_levels(lv, above, head_row * lv.pitch + k, sum);
    *acc = sum;
  }
}

static constexpr int kSms = 148, kMaxParts = 8, kMaxLevels = 64;
// Launches of up to so many bytes of dQ tiles (one per visit) have levels, if these take no more than the other number.
// Levels cost what it takes to clear and to sum them, in the passes before and after the kernel or in launches of their
// own: four sequences of 300 to 2100 tokens, 8 / 2 heads, 110 MB, forward and backward, 107 us without, 130 and 135
// with them; 2048 tokens, 71 MB, 96, 101 and 108.  Above, what is added to no longer stays in L2: 2048 tokens, 32 / 8
// heads, 285 MB, 169 and 280 us, 4096 tokens, 8 / 2 heads, 277 MB, 152 and 235.  (A tile of its own for every visit,
// stored and then summed, took 150 us for the first.)
static constexpr long kMaxVisitBytes = 128l << 20, kMaxWorkspace = 512l << 20;
static std::atomic<uint64_t> g_bwd_smem_raised[4];
static long long* g_bwd_timeline_host = nullptr;  // non-null selects the instrumented build of the kernel

}  // namespace dcpk

void dcpk_fill_copy_ctx(dcpk::CopyCtx* ctx, void* const* src_ptrs, void* const* dst_ptrs, int stat_stride);

using namespace dcpk;

// Points the kernel's cycle-counter timeline at `buf` (>= 16 int64, device memory) or disables it (null).
extern "C" int dcpk_attn_bwd_set_timeline(void* buf) {
  long long* p = static_cast<long long*>(buf);
  g_bwd_timeline_host = p;
  return cudaMemcpyToSymbol(g_bwd_timeline, &p, sizeof(p)) == cudaSuccess ? 0 : -5;
}

// Bytes of the workspace of dcpk_attn_bwd for item lists of `n_levels` levels (see dq_level; 0: not known); 0: there is
// none.
extern "C" long dcpk_attn_bwd_workspace(int n_items_total, long q_rows, int hq, int channels, int n_levels) {
  if (n_levels < 2 || n_levels > kMaxLevels) return 0;
  const long pitch = level_pitch(channels) * long(sizeof(float));
  const long bytes = (n_levels - 1) * q_rows * hq * pitch;
  return long(n_items_total) * hq * kQTile * pitch <= kMaxVisitBytes && bytes <= kMaxWorkspace ? bytes : 0;
}

// Over how many CTAs a head group of `group` query heads is split, for `n_ctas` key tiles of `hkv` heads whose item
// lists have n_items_total entries in all and at most max_items (0: not known, the group stays whole).
//
// A CTA visits its items once per query head of the group, or the group is split over several CTAs (a cluster, at most
// the portable 8, which adds its parts of dK / dV up in a fixed order): shorter longest lists, and more CTAs to begin
// and end, which takes one as long as 8 visits (2.2 us each).  The launch takes as long as its longest list, or as all
// visits spread over the SMs, whichever is more; the split for which that is least is taken, the smallest of equals.
// Over 78 batches of 700 to 22000 tokens (causal, full, sink + window; 8 to 32 heads, groups of 4 and 8, 64 and 128
// channels) that is within 0.8 % of the best split on average, 12 % at worst; splitting while the longest list was
// above the SMs' average, but seldom into more than one wave, was 9 % off, 54 % at worst.  2048 tokens, 32 / 8 heads:
// 152 us before, 109 in two parts; eight sequences, 9105 tokens, 8 / 2 heads: 147 and 107 us.
// CTAs that all run at once add to a row of dQ in the order of their items, and as long as their lists are short and
// begin at different queries, as causal ones do, that is nearly the same in every run (ten sequences of 800 tokens or
// seven of 1200, 8 / 2 heads, 2000 tokens, 16 / 4 heads: the same bits in 100 of 100; from 17 items on, 2100 to 3900
// tokens, in 97 to 2).  Unless `any_wave` (dQ has levels, whose order does not matter) or some list is longer than
// that, they become more than one wave only where that takes 32 visits (about 70 us) off the longest list, which costs
// up to 10 % (1500 tokens, 32 / 8 heads, forward and backward, 126 -> 139 us).
extern "C" int dcpk_attn_bwd_parts(int n_ctas, int hkv, int group, int max_items, int n_items_total, int any_wave) {
  constexpr long kBegin = 8;
  constexpr int kRepeats = 16;
  auto visits = [&](int p) {   // times the SMs
    return std::max(kSms * (long(max_items) * (group / p) + kBegin),
                    long(n_items_total) * hkv * group + kBegin * n_ctas * hkv * p);
  };
  int parts = 1, in_one_wave = 0;   // the largest split whose CTAs all run at once, if there is one
  for (int p = 1; max_items > 0 && p <= group && p <= kMaxParts; ++p) {
    if (group % p != 0) continue;
    if (long(n_ctas) * hkv * p <= kSms) in_one_wave = p;
    else if (!any_wave && max_items <= kRepeats && in_one_wave > 0 && long(max_items) * (group / in_one_wave - group / p) < 32)
      continue;
    if (visits(p) < visits(parts)) parts = p;
  }
  return parts;
}

// Launches the backward kernel: one CTA per (entry of `ctas`, KV head).  channels: of the arenas' 128, those that may
// be other than zero (the first); the gradients of the others are left as they are.  n_items_total / n_mask_rows are
// the lengths of the item and mask tables; entries that point past them are reported (status 3), not read.  max_items:
// length of the longest item list (0: not known, the head groups stay whole).  workspace: as many bytes as
// dcpk_attn_bwd_workspace says; null: dQ has no levels.  level_passes: 1 they are cleared here (else dcpk_attn_bwd_prep
// did), + 2 and summed here (else dcpk_cut_cast_gradients does).
extern "C" int dcpk_attn_bwd(const void* q_arena, const void* do_arena, long q_rows, const void* kv_arena,
                             long kv_rows, int hq, int hkv, const void* ctas, int n_ctas, const void* items,
                             int n_items_total, int max_items, const void* masks, int n_mask_rows, const float* lse, const float* delta,
                             int stat_stride, float* const* dq_ptrs, float* const* dkv_ptrs, int n_dst, float scale, int channels,
                             int n_levels, void* workspace, int level_passes, const void* jobs, int n_jobs,
                             void* const* job_src_ptrs, void* const* job_dst_ptrs, int job_stat_stride, int* status, void* stream) {
  if (n_ctas <= 0) return n_jobs > 0 ? -6 : 0;   // copy jobs need a kernel to ride on
  if (n_dst > kMaxPeers || hq % hkv != 0 || channels < 1 || channels > kHeadDim) return -3;
  const bool levels = workspace != nullptr && dcpk_attn_bwd_workspace(n_items_total, q_rows, hq, channels, n_levels) > 0;
  CUtensorMap tm_q, tm_do, tm_kv, tm_dq, tm_dkv, tm_levels;
  if (encode_f32_tile_map(&tm_dq, dq_ptrs[0], uint64_t(q_rows), uint32_t(hq), kHeadDim, 32, 32)) return -1;
  tm_levels = tm_dq;
  if (levels && encode_f32_tile_map(&tm_levels, workspace, uint64_t(n_levels - 1) * q_rows, uint32_t(hq),
                                    uint32_t(level_pitch(channels)), 32, 32))
    return -1;
  if (encode_f32_tile_map(&tm_dkv, dkv_ptrs[0], uint64_t(kv_rows), uint32_t(2 * hkv), kHeadDim, 32, 32)) return -1;
  if (encode_arena_map(&tm_q, q_arena, uint64_t(q_rows), uint32_t(hq), kHeadDim, kQTile)) return -1;
  if (encode_arena_map(&tm_do, do_arena, uint64_t(q_rows), uint32_t(hq), kHeadDim, kQTile)) return -1;
  if (encode_arena_map(&tm_kv, kv_arena, uint64_t(kv_rows), uint32_t(2 * hkv), kHeadDim, 128)) return -1;
  BwdPtrs pp;
  for (int i = 0; i < kMaxPeers; ++i) {
    pp.dq[i] = i < n_dst ? dq_ptrs[i] : nullptr;
    pp.dkv[i] = i < n_dst ? dkv_ptrs[i] : nullptr;
  }
  CopyCtx ctx;
  dcpk_fill_copy_ctx(&ctx, n_jobs > 0 ? job_src_ptrs : nullptr, n_jobs > 0 ? job_dst_ptrs : nullptr, job_stat_stride);
  const int smem = int(sizeof(BwdSmem));
  static_assert(sizeof(BwdSmem) <= 227 * 1024, "shared memory of one CTA");
  const int v = g_bwd_timeline_host ? 3 : channels > 96 ? 0 : channels > 64 ? 1 : 2;
  auto kernel = v == 3 ? attn_bwd_kernel<true, 128> : v == 2 ? attn_bwd_kernel<false, 64>
              : v == 1 ? attn_bwd_kernel<false, 96> : attn_bwd_kernel<false, 128>;
  if (raise_smem_limit(kernel, smem, g_bwd_smem_raised[v]) != cudaSuccess) return -4;
  // about 16 fetch CTAs when there is something to fetch
  const int n_copy_rows = n_jobs > 0 ? (16 + hkv - 1) / hkv : 0;
  const bool any_order = levels || n_levels == 1;   // of the additions to dQ
  const int group = hq / hkv, parts = dcpk_attn_bwd_parts(n_ctas, hkv, group, max_items, n_items_total, any_order);
  const int heads_per_cta = group / parts;
  // Overlapped with the kernel before it only where all CTAs run at once: CTAs that begin together go through the
  // queries together and find one another's tiles in L2, those that begin as the SMs come free do not (forward and
  // backward of 121987 tokens, mixed masks, 41.3 ms plain, 44.3 overlapped; 6168 tokens 1008 and 1050 us; 4040 tokens
  // in one wave 134 and 131 us).  And only where dQ has levels, as the CTAs of an overlapped wave begin so far apart
  // that they add to dQ in another order each time.
  const dim3 grid(hkv * parts, n_ctas + n_copy_rows);
  const DcpkDqLevels of_call = {items, n_items_total, n_levels, int(q_rows), hq, channels, levels ? workspace : nullptr};
  const unsigned level_blocks = unsigned((q_rows + kLevelRows - 1) / kLevelRows);
  if (levels && (level_passes & 1) &&
      launch_overlapped(dq_levels_kernel<false>, level_blocks, 256, 0, static_cast<cudaStream_t>(stream), 1, false, make_levels(&of_call),
                        dq_ptrs[0]) != cudaSuccess)
    return -5;
  const cudaError_t rc = launch_overlapped(
      kernel, grid, kBwdThreads, smem, static_cast<cudaStream_t>(stream), unsigned(parts),
      any_order && long(grid.x) * grid.y <= kSms, tm_q, tm_do,
      tm_kv, tm_dq, tm_dkv, tm_levels, levels ? n_levels : 1, static_cast<const BwdCta*>(ctas), static_cast<const BwdItemDesc*>(items),
      static_cast<const int4*>(masks), lse, delta, pp, hq, hkv, heads_per_cta, stat_stride, n_dst, int(q_rows), int(kv_rows),
      n_mask_rows, n_items_total, scale, static_cast<const CopyJob*>(jobs), n_jobs, ctx, n_copy_rows, status);
  if (rc != cudaSuccess || cudaGetLastError() != cudaSuccess) return -5;
  if (levels && (level_passes & 2) &&
      launch_overlapped(dq_levels_kernel<true>, level_blocks, 256, 0, static_cast<cudaStream_t>(stream), 1, false, make_levels(&of_call),
                        dq_ptrs[0]) != cudaSuccess)
    return -5;
  return 0;
}
