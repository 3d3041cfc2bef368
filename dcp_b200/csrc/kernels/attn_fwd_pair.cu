// Blockwise range-masked attention forward for sm_100a: pairs of CTAs, 256 queries of one head per pair, persistent.
//
// A pair of CTAs (a cluster of two, cta_group::2) takes one 256-row tile after another; the even CTA has query rows
// 0-127 (tile A), the odd one 128-255 (tile B).  Warps of a CTA:
//   0-3, 4-7  softmax of every second KV tile (one thread per query row),
//   8         TMA producer: this CTA's Q rows and its halves of the K and V tiles,
//   9         UMMA issuer (even CTA only: a product covers both CTAs' rows),
//   10-11     fetch the next plan stage's remote operands (copy jobs: peer loads over NVLink into this
//             GPU's staging rows, see copy_jobs.cuh) while the tiles are computed,
//   12-15     epilogue: O out of TMEM, divided by the row sums, stored.
// All non-softmax warps donate registers (setmaxnreg).
//   S(j) = Q K(j)^T   M = 256, each CTA holds 64 of the 128 keys             -> TMEM
//   O   += P(j) V(j)  P as packed bf16 in the TMEM columns S(j) came from, each CTA holds 64 of the channels
// TMEM (512 columns): three score buffers [0,384), O [384,512).  Per KV tile j the issuer emits PV(j), QK(j+3), also
// across the end of a tile: the next tile's Q has a buffer of its own and its products wait only until the epilogue has
// taken O to registers.
//
// Why pairs: with one query tile per CTA there is room for three score buffers, so a softmax warp finds its next scores
// ready.  (Two query tiles per CTA leave one buffer each: scores, exponentials and both products of a tile are one
// serial chain of 3200 cycles per 2180 of tensor time.)  One query tile per CTA alone would read every K and V tile
// twice as often from L2; in a pair each CTA reads half of it, and the tensor core reads half as much of B from shared
// memory.
//
// Why no running maximum: out = O / l and lse = m + ln l are exact for any reference m, and bf16 has the exponent range
// of fp32, so m has to be near the row's largest score only within what fp32 holds.  A row keeps the maximum of the
// first tile it sees anything of; while some row of a warp has none, the two warps that share the rows hand the
// references on from KV tile to KV tile.  Afterwards no maximum is taken and nothing is handed on.  Where a row's sum
// exceeds 2^64 (a score 44 above the reference), or the sum or an element of the result is not finite (values of 2^64
// and more overflow O before the sum does; looked for where the sum exceeds 2^16, in what has been stored: a look in
// passing made the epilogue 350 cycles longer per tile), the pair goes through the tile again when it is done with all
// tiles, with the reference following the maximum to within 2^8 and O rescaled in TMEM where it moves.  That pass takes
// longer than the first, as references are handed on at every KV tile: 32 / 8 heads, all rows rising by 2^80 behind
// their first 128 keys, full 8192 x 16384 3.71 ms against 1.55 without the rise, causal 4096 x 4096 0.302 against 0.142
// (a kernel that kept the running maximum throughout took 1.86 and 0.161 ms for them).
//
// P of the first 64 keys is handed over while the softmax works on the other 64, so half of PV runs under it.  The next
// scores' barrier is asked before the last probabilities are stored: a look at shared memory queues behind the
// exponentials of the other warp, 200 cycles and more.  Arrivals on the other CTA's barriers carry no release at
// cluster scope (a fence that waits for everything the warp has stored; 1.6 times slower): what they announce is in
// TMEM.
//
// What bounds it: the issuing thread and the softmax warps that share its scheduler.  Where both are in time a KV tile
// takes 1250 cycles per CTA; the exponentials need 1024 of them and the products 1024.  Every look at a barrier costs
// the issuer 200 cycles, so it asks for its three at once, and K(j+3) and V(j), which one step consumes, share a
// barrier.
//
// Why the epilogue has warps of its own: the softmax warps leave sums and references in shared memory and go on with
// the next tile's scores, whose first product waits until O is in registers, about 2000 cycles; with the epilogue in
// the softmax warps the tensor core was idle for 4000 (16 heads, 16384 queries over 512 keys 139 -> 107 us, causal 4096
// x 4096 167 -> 159 us).  It stores rows straight from registers, a sector per lane and instruction: through shared
// memory O was in TMEM for 3500 cycles instead of 1900, as every look at shared memory queues behind the exponentials
// (8192 queries over 1500 keys 213 -> 201 us).  A copy per row by the copy engine takes 60 cycles to issue, 2000 for a
// half of 32 rows.
//
// Measured against two query tiles per CTA (32 / 8 heads, queries x keys; one box, L2 flushed between calls): full 8192
// x 16384 1.69 -> 1.55 ms (1415 TFLOP/s), causal 1.42 -> 1.26 ms, causal 4096 x 4096 0.169 -> 0.142, 2048 x 2048 equal,
// 8192 over 1500 keys 0.224 -> 0.177; 16 heads, 16384 over 512 keys 0.122 -> 0.095 ms; 8 heads, causal 1024 x 1024 27.5
// -> 19.5 us.  Tried and left: a launch with a pair per tile (4096 x 4096 4 % slower, 16384 tokens in sequences of 8192
// 6 %); the result written after the next tile's first exponentials (full 6 % slower); the maximum taken beside the
// exponentials (11 % slower).
//
// The partial (out, lse) of a tile is stored straight to its destination arena, which may be a
// peer GPU's memory (plain st.global over the NVLink mapping).
//
// Reference behaviour covered: the varlen forward with block tables and per-query KV ranges that
// dcp/runtime/flash_attention/executor.py:884-913 calls.
#include <cuda_fp16.h>
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "attn_common.cuh"
#include "copy_jobs.cuh"
#include "entries.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "smem_limit.h"
#include "tmap.cuh"

namespace dcpk {

static constexpr int kPairThreads = 512;  // 8 softmax warps, producer, UMMA issuer, 2 fetch warps, 4 epilogue warps
static constexpr int kPairs = 148 / 2;    // one CTA per SM
static constexpr int kSlots = 4;          // slot i holds this CTA's halves of K(i) and V(i-3): what one step of the issuer consumes
static constexpr int kSBufs = 3;
static constexpr int kQHalf = 128 * 64 * 2;      // [128 queries x 64 channels]
static constexpr int kKHalf = 64 * 64 * 2;       // [64 keys x 64 channels]
static constexpr int kKvBytes = 64 * 128 * 2;    // a CTA's half of a K or V tile
static constexpr int kRedoWords = 16;
static constexpr int kInfos = 4;
static constexpr float kGap = 8.f;            // exponent (base 2) by which a score may exceed a reference that can still move
static constexpr float kSafeSum = 65536.f;    // up to this row sum O is finite where values are below 2^112
static constexpr float kMaxSum = 1.8447e19f;  // 2^64: a row sum above it sends the tile through the second pass

// What the softmax and epilogue warps of a CTA need of a tile, put into shared memory by the TMA producer, which is
// some KV tiles ahead of them: from the tables it would take three dependent trips to memory between two tiles.  And
// what they leave for one another.
struct __align__(16) TileInfo {
  int4 mask[kTileM];        // ranges of this CTA's rows
  float m[kTileM];          // reference of a row
  float l[2][kTileM];       // its sums over the KV tiles of either warpgroup
  int4 first[2];            // first KV tiles
  uint8_t* out;             // where the first row goes
  int out_type, out_channels;   // how (see store_channels)
  float* lse;
  int n_rows, n_kv, kv_off, round;  // rows of this CTA; n_kv < 0: there are no more tiles
};

struct __align__(1024) PairSmem {
  uint8_t q[2][2 * kQHalf];
  uint8_t k[kSlots][kKvBytes];      // 64 of the 128 keys, all channels
  uint8_t v[kSlots][kKvBytes];      // all 128 keys, 64 of the channels
  TileInfo info[kInfos];
  uint32_t redo[kRedoWords];        // rounds that go through the second pass
  // of the even CTA (bytes and arrivals of both CTAs): q_full, kv_full, p_ready, o_empty; the others are signalled in
  // both
  uint64_t q_full[2], q_empty[2], kv_full[kSlots], kv_empty[kSlots], s_full[kSBufs], p_ready[kSBufs][2], o_empty, acc_full,
      m_ready[kInfos][4], l_ready[kInfos][4], info_full[kInfos], info_empty[kInfos];
  uint32_t tmem_base;
  int abort_word;
  int any_redo;
};

// One 128-key tile of the pair's KV walk, prepared by the host (build_fwd_tables with tile_m = 256).
struct KvSub {
  int row;       // first arena row of the 128 keys
  int pos0;      // position of the first key in the Q block's concatenated KV
  int n_valid;   // valid keys (1..128)
  int flags;     // bit 0 / 1: query tile A / B sees at least one key; bit 2 / 3: A / B sees every pair
};

template <typename F>
__device__ __forceinline__ void for_each_barrier(PairSmem& sm, F f) {   // f(barrier, arrivals)
  for (int i = 0; i < 2; ++i) { f(&sm.q_full[i], 1); f(&sm.q_empty[i], 1); }
  for (int i = 0; i < kSlots; ++i) { f(&sm.kv_full[i], 1); f(&sm.kv_empty[i], 1); }
  // of P and O: four warps of either CTA
  for (int i = 0; i < kSBufs; ++i) { f(&sm.s_full[i], 1); f(&sm.p_ready[i][0], 8); f(&sm.p_ready[i][1], 8); }
  f(&sm.o_empty, 8);
  f(&sm.acc_full, 1);
  for (int i = 0; i < 4 * kInfos; ++i) { f(&sm.m_ready[i >> 2][i & 3], 1); f(&sm.l_ready[i >> 2][i & 3], 2); }
  for (int i = 0; i < kInfos; ++i) { f(&sm.info_full[i], 1); f(&sm.info_empty[i], 12); }   // softmax and epilogue warps
}

// P = exp2(S * c - m) of 64 keys of a row, cut to bf16, to TMEM; `ps2` collects the row sum.  Packed fp32: one
// instruction scales two scores, one adds two probabilities.  Every probability carries the factor kTruncScale (folded
// into the exponent), so cutting it to bf16 is unbiased; the row sum carries the same factor, which cancels in O / l
// and is taken out of the LSE in the epilogue.
__device__ __forceinline__ void softmax_half(const uint32_t* s, uint64_t sl2_2, uint64_t negm_2, uint64_t* ps2, uint32_t p_addr) {
  uint32_t preg[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(s[2 * c]), __uint_as_float(s[2 * c + 1])), sl2_2, negm_2);
    float x0, x1;
    unpack_f32x2(x2, x0, x1);
    const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
    ps2[c & 3] = add_f32x2(ps2[c & 3], pack_f32x2(p0, p1));
    preg[c] = pack_bf16x2_trunc(p0, p1);
  }
  tmem_st32(p_addr, preg);
}

// 16 channels of a row, from `ch` on, in the caller's type (0 float, 1 half, 2 bf16) where the row has them, a multiple
// of 8: the bf16 result, which float holds as it is, and half rounded once more (beyond 65504 it is infinite there)
__device__ __forceinline__ void store_channels(uint8_t* row, int type, int channels, int ch, uint32_t* packed) {
  if (ch >= channels) return;
  const bool both = ch + 16 <= channels;
  uint8_t* p = row + ch * (type == 0 ? 4 : 2);
  const bool wide = (reinterpret_cast<uintptr_t>(p) & 31) == 0;
  if (type == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && !both) break;
      uint32_t f[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) { f[2 * i] = packed[4 * h + i] << 16; f[2 * i + 1] = packed[4 * h + i] & 0xffff0000u; }
      if (wide) {
        st_global_v8(p + 32 * h, f);
      } else {
        reinterpret_cast<uint4*>(p)[2 * h] = make_uint4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<uint4*>(p)[2 * h + 1] = make_uint4(f[4], f[5], f[6], f[7]);
      }
    }
    return;
  }
  if (type == 1)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half2 v = __floats2half2_rn(__uint_as_float(packed[i] << 16), __uint_as_float(packed[i] & 0xffff0000u));
      packed[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
  if (wide && both) {
    st_global_v8(p, packed);
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    if (both) reinterpret_cast<uint4*>(p)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
  }
}

// no element of a row that this thread has stored is infinite or not a number; its form as above
__device__ __forceinline__ bool finite_row(const uint8_t* row, int type, int channels) {
  // the exponent's bits and one more at their lowest: a carry into the sign's place where all are set
  const uint32_t exponent = type == 0 ? 0x7f800000u : type == 1 ? 0x7c007c00u : 0x7f807f80u;
  const uint32_t one = type == 0 ? 0x00800000u : type == 1 ? 0x04000400u : 0x00800080u;
  uint32_t carries = 0;
#pragma unroll 1
  for (const uint8_t* p = row; p < row + channels * (type == 0 ? 4 : 2); p += 16) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    carries |= ((v.x & exponent) + one) | ((v.y & exponent) + one) | ((v.z & exponent) + one) | ((v.w & exponent) + one);
  }
  return (carries & (type == 0 ? 0x80000000u : 0x80008000u)) == 0;
}

// kD: channels that are computed.  The arenas' rows have 128; heads of fewer are zero-padded there, and what S adds up
// over zeros is left out.  PV stays as it is, so that the output's padding is written.  8192 queries x 16384 keys, 32 /
// 8 heads, against all 128 channels: 64 channels 1.43 -> 1.33 ms (causal 1.08 -> 1.04: the exponentials bound it then),
// 96 channels 1.51 -> 1.47 ms. kForm: the results' type and width are arguments; rows of 128 in bf16 have an instance
// of their own, as a test per store cost the calls that have them 1 to 4 %.
template <int kD, bool kForm>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const AttnTile* __restrict__ tiles, int n_tiles,
                     const int4* __restrict__ kv_subs, const int4* __restrict__ masks, PeerPtrs ptrs, int hq, int hkv,
                     int lse_stride_a, int lse_stride_b, int n_dst_a, int n_dst, int out_type, int out_channels, int q_rows, int n_mask_rows,
                     int n_kv_subs, float scale, const CopyJob* __restrict__ jobs, int n_jobs,
                     const __grid_constant__ CopyCtx copy_ctx, int* __restrict__ status) {
  constexpr int kHalves = kD > 64 ? 2 : 1;   // of 64 channels of Q and K
  extern __shared__ uint8_t smem_raw[];
  PairSmem& sm = *reinterpret_cast<PairSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int X = blockIdx.x & 1;   // query tile of this CTA == its rank in the cluster
  if (threadIdx.x == 256) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    for_each_barrier(sm, [](uint64_t* bar, int count) { mbar_init(bar, count); });
    sm.abort_word = 0;
    sm.any_redo = 0;
    for (int i = 0; i < kRedoWords; ++i) sm.redo[i] = 0;
    mbar_fence_init();
  }
  if (warp == 9) tmem_alloc_pair(&sm.tmem_base, 512);
  tc_fence_before();
  cluster_sync();   // barriers and TMEM of both CTAs are there
  tc_fence_after();
  grid_let_next();
  grid_wait();
  const uint32_t tmem = sm.tmem_base;
  volatile int* abort_word = &sm.abort_word;
  const int4 none = make_int4(0, 0, 0, 0);

  // The pairs of CTAs take the tiles, which are ordered by length, in rounds and every second round backwards.
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  auto index_of = [&](int round) { return round * n_pairs + ((round & 1) ? n_pairs - 1 - pair : pair); };
  // the first tile from `round` on that has work for the pass and KV tiles, or none of them; false: there is none
  int first_empty = -1;   // first round with a tile that has none
  auto find_tile = [&](int pass, int& round, AttnTile& t, bool empty) -> bool {
    for (;; ++round) {
      const int i = index_of(round);
      if (i >= n_tiles) return false;
      if (pass > 0 && !((sm.redo[(round >> 5) & (kRedoWords - 1)] >> (round & 31)) & 1u)) continue;
      t = tiles[i];
      // table sanity: a tile that would store outside its destination arena, or read a head / row / table entry that
      // does not exist, is reported and skipped (by all warps of both CTAs)
      const int dst_rows = t.out_dev < n_dst_a ? lse_stride_a : lse_stride_b;
      const bool bad = t.out_dev < 0 || t.out_dev >= n_dst || t.out_row < 0 || t.n_rows < 0 ||
                       t.n_rows > 2 * kTileM || t.out_row + t.n_rows > dst_rows || t.head < 0 ||
                       t.head >= hq || t.q_row < 0 || t.q_row + t.n_rows > q_rows || t.n_kv < 0 ||
                       t.mask_row < 0 || t.mask_row + t.n_rows > n_mask_rows || t.kv_off < 0 ||
                       t.kv_off + t.n_kv > n_kv_subs;
      if (bad) atomicExch(status, kStatusBadArgs);
      if (bad) continue;
      if ((t.n_kv == 0) == empty) return true;
      if (!empty && first_empty < 0) first_empty = round;
    }
  };
  // End of a pass over the tiles, by all threads of both CTAs; true: a second pass follows.
  auto next_pass = [&](int pass) -> bool {
    // a CTA that gave up tells the other, which waits for it
    if (threadIdx.x == 0 && sm.abort_word) st_cluster_u32(smem_u32(&sm.abort_word), X ^ 1, 1u);
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    if (pass > 0 || !sm.any_redo) return false;
    if (threadIdx.x == 256) {
      for_each_barrier(sm, [](uint64_t* bar, int count) { mbar_inval(bar); mbar_init(bar, count); });
      mbar_fence_init();
    }
    cluster_sync();
    return true;
  };

  // register rebalancing between warpgroups (setmaxnreg inside each role's branch): the others give registers up, the
  // softmax warps take them (256 x 200 + 128 x 64 + 128 x 48 = 65536 = 512 x 128, what the block is
  // launched with)
  if (warp >= 12) {
    // ------------------------------------------------------------ epilogue: thread = query row
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const int quad = warp & 3, r = threadIdx.x & 127;
    const uint32_t o_addr = tmem + (uint32_t(quad * 32) << 16) + kSBufs * 128;
    const uint32_t o_bar = cluster_addr(smem_u32(&sm.o_empty), 0);
   for (int pass = 0;; ++pass) {
    // O is in registers: the products of the tile in slot `info`, which is there, may set it; false: that is the end
    auto hand_over = [&](int info) -> bool {
      const TileInfo& ti = sm.info[info];
      if (ti.n_kv < 0) return false;
      if (ti.n_kv > 0) {
        if (!((ti.first[0].w >> X) & 1)) {   // then no product sets O of this query tile, they only add to it
          uint32_t zero[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) zero[c] = 0;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) tmem_st32(o_addr + c * 32, zero);
          tmem_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(o_bar);
      }
      return true;
    };
    auto wait_info = [&](int info, int iph) { return __all_sync(0xffffffffu, mbar_wait(&sm.info_full[info], iph, abort_word)); };
    int acc_ph = 0;  // parity of the tiles with a product so far
    bool more = wait_info(0, 0) && hand_over(0);
    for (int info = 0, iph = 0; more;) {
      const TileInfo& ti = sm.info[info];
      const int n = ti.n_kv;
      const int next = info + 1 == kInfos ? 0 : info + 1, next_ph = next == 0 ? iph ^ 1 : iph;
      bool ok = mbar_wait(&sm.l_ready[info][quad], iph, abort_word);
      const bool next_there = __all_sync(0xffffffffu, mbar_test_wait(&sm.info_full[next], next_ph));   // asked while there is time
      const float l_sum = ti.l[0][r] + ti.l[1][r];
      const float inv_l = l_sum > 0.f ? 1.f / l_sum : 0.f;
      if (ok && r < ti.n_rows) ti.lse[r] = l_sum > 0.f ? ti.m[r] * scale + logf(l_sum) - kTruncLn : -INFINITY;
      if (n > 0) {
        ok = ok && mbar_wait(&sm.acc_full, acc_ph, abort_word);
        acc_ph ^= 1;
        tc_fence_after();
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      // a row from TMEM to where it goes, 16 channels (a whole sector) per store
      const bool mine = r < ti.n_rows;
      const int type = kForm ? ti.out_type : 2, channels = kForm ? ti.out_channels : kHeadDim;
      uint8_t* out = ti.out + size_t(r) * hq * channels * (type == 0 ? 4 : 2);
      const bool wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint32_t oreg[16], packed[8];
        if (n > 0) {  // warp-uniform: the TMEM load is a warp-collective instruction
          tmem_ld16(o_addr + c * 16, oreg);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) oreg[i] = 0;
        }
        if (c == 7) more = (next_there || wait_info(next, next_ph)) && hand_over(next);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          packed[i] = pack_bf16x2(__uint_as_float(oreg[2 * i]) * inv_l, __uint_as_float(oreg[2 * i + 1]) * inv_l);
        if (mine) {
          if (kForm) {
            store_channels(out, type, channels, c * 16, packed);
          } else if (wide) {
            st_global_v8(out + c * 32, packed);
          } else {
            reinterpret_cast<uint4*>(out)[2 * c] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            reinterpret_cast<uint4*>(out)[2 * c + 1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
          }
        }
      }
      if (pass == 0 && __any_sync(0xffffffffu, mine && !(l_sum <= kSafeSum))) {
        const bool again = mine && (!(l_sum < kMaxSum) || !finite_row(out, type, channels));
        if (__any_sync(0xffffffffu, again) && lane == 0) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            st_cluster_u32(smem_u32(&sm.any_redo), c, 1u);
            or_cluster_u32(smem_u32(&sm.redo[(ti.round >> 5) & (kRedoWords - 1)]), c, 1u << (ti.round & 31));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.info_empty[info]);
      info = next; iph = next_ph;
    }
    if (!next_pass(pass)) break;
   }
  } else if (warp >= 8) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
   if (warp == 8) {
    // ------------------------------------------------------------ TMA producer: this CTA's rows and halves
   for (int pass = 0;; ++pass) {
    if (lane == 0) {
      const uint32_t q_bar = cluster_addr(smem_u32(&sm.q_full[0]), 0), kv_bar = cluster_addr(smem_u32(&sm.kv_full[0]), 0);
      bool ok = true;
      int qi = 0, qph = 1, slot = 0, ph = 1, info = 0, iph = 1, used = 0;   // used: slots and, above them, Q buffers
      // V is loaded three KV tiles after K: where the last three are (oldest in the third)
      int row1 = 0, row2 = 0, row3 = 0, head1 = 0, head2 = 0, head3 = 0, behind = 0;
      auto load_slot = [&](bool with_k, bool with_v, int row, int kv_head) -> bool {
        if (!mbar_wait(&sm.kv_empty[slot], ph, abort_word)) return false;
        used |= 1 << slot;
        if (X == 0) mbar_expect_tx(&sm.kv_full[slot], 2 * (kHalves * kKHalf * with_k + kKvBytes * with_v));
        if (with_v) tma_load_3d_pair(sm.v[slot], &tm_v, kv_bar + 8 * slot, 64 * X, hkv + head3, row3);
        if (with_k) {
          tma_load_3d_pair(sm.k[slot], &tm_k, kv_bar + 8 * slot, 0, kv_head, row + 64 * X);
          if (kHalves > 1) tma_load_3d_pair(sm.k[slot] + kKHalf, &tm_k, kv_bar + 8 * slot, 64, kv_head, row + 64 * X);
        }
        if (++slot == kSlots) { slot = 0; ph ^= 1; }
        return true;
      };
      AttnTile tile;
      // Tiles without keys come last: the last three V of a tile are loaded with the K of the next ones, and announcing
      // a tile waits until the one kInfos before it is finished.
      bool empty = false;
      first_empty = -1;
      for (int round = 0; ok; ++round) {
        bool more = find_tile(pass, round, tile, empty);
        if (!more && !empty) {
          // the last three V: slots 3, 4 and 5 at the earliest
          if (behind > 0 && behind < 3) slot = 3;
          for (; ok && behind > 0; --behind) {
            if (behind < 3) { row3 = behind == 2 ? row2 : row1; head3 = behind == 2 ? head2 : head1; }
            ok = load_slot(false, true, 0, 0);
          }
          empty = true;
          round = first_empty;
          more = round >= 0 && find_tile(pass, round, tile, empty);
        }
        ok = ok && mbar_wait(&sm.info_empty[info], iph, abort_word);
        if (!ok) break;
        TileInfo& ti = sm.info[info];
        if (!more) {
          ti.n_kv = -1;
          mbar_arrive(&sm.info_full[info]);
          break;
        }
        const int4* subs = kv_subs + tile.kv_off;
        const int kv_head = tile.head / (hq / hkv), n = tile.n_kv;
        const int4 sub0 = n > 0 ? subs[0] : none;
        ti.first[0] = sub0;
        if (n > 1) ti.first[1] = subs[1];
        ti.n_kv = n;
        ti.kv_off = tile.kv_off;
        ti.round = round;
        ti.n_rows = tile.n_rows - X * kTileM;
        const bool own_form = kForm && tile.out_dev >= n_dst_a;   // partial results are rows of 128 in bf16
        ti.out_type = own_form ? out_type : 2;
        ti.out_channels = own_form ? out_channels : kHeadDim;
        ti.out = static_cast<uint8_t*>(ptrs.out[tile.out_dev]) +
                 (size_t(tile.out_row + X * kTileM) * hq + tile.head) * ti.out_channels * (ti.out_type == 0 ? 4 : 2);
        ti.lse = ptrs.lse[tile.out_dev] + size_t(tile.head) * (tile.out_dev < n_dst_a ? lse_stride_a : lse_stride_b) +
                 tile.out_row + X * kTileM;
        const int mask_bytes = 16 * min(max(tile.n_rows - X * kTileM, 0), kTileM);
        mbar_expect_tx(&sm.info_full[info], mask_bytes);
        if (mask_bytes > 0) bulk_load(ti.mask, masks + tile.mask_row + X * kTileM, mask_bytes, &sm.info_full[info]);
        if (++info == kInfos) { info = 0; iph ^= 1; }
        if (n == 0) continue;
        int ahead = sub0.x;
        ok = mbar_wait(&sm.q_empty[qi], qph, abort_word);
        if (!ok) break;
        used |= 1 << (kSlots + qi);
        if (X == 0) mbar_expect_tx(&sm.q_full[qi], 2 * kHalves * kQHalf);
        tma_load_3d_pair(sm.q[qi], &tm_q, q_bar + 8 * qi, 0, tile.head, tile.q_row + X * kTileM);
        if (kHalves > 1) tma_load_3d_pair(sm.q[qi] + kQHalf, &tm_q, q_bar + 8 * qi, 64, tile.head, tile.q_row + X * kTileM);
        if (++qi == 2) { qi = 0; qph ^= 1; }
        for (int j = 0; j < n && ok; ++j) {
          const int row = ahead;
          if (j + 1 < n) ahead = subs[j + 1].x;
          ok = load_slot(true, behind == 3, row, kv_head);
          behind = min(behind + 1, 3);
          row3 = row2; row2 = row1; row1 = row;
          head3 = head2; head2 = head1; head1 = kv_head;
        }
      }
      // arrivals from the even CTA's issuer have all come in before this CTA may retire
      for (int i = 0; ok && i < kSlots; ++i) {
        if ((used >> slot) & 1) ok = mbar_wait(&sm.kv_empty[slot], ph, abort_word);
        if (++slot == kSlots) { slot = 0; ph ^= 1; }
      }
      for (int i = 0; ok && i < 2; ++i) {
        if ((used >> (kSlots + qi)) & 1) ok = mbar_wait(&sm.q_empty[qi], qph, abort_word);
        if (++qi == 2) { qi = 0; qph ^= 1; }
      }
      // copies already in flight get a millisecond to land before the CTAs retire
      if (!ok)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    if (!next_pass(pass)) break;
   }
   } else if (warp == 9) {
    // ------------------------------------------------------------ UMMA issuer (even CTA), for both CTAs
   for (int pass = 0;; ++pass) {
    if (X == 0 && elect_one()) {   // one thread from here on
      constexpr uint32_t idesc_qk = make_idesc_bf16(256, 128, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_bf16(256, 128, 0, 1);
      // descriptors differ in the address field of the low word only
      const uint64_t some = make_sdesc_sw128(0, 16, 1024);
      const uint32_t hi = uint32_t(some >> 32);
      const uint32_t q_lo = uint32_t(some) + sdesc_addr(sm.q[0]), k_lo = uint32_t(some) + sdesc_addr(sm.k[0]),
                     v_lo = uint32_t(some) + sdesc_addr(sm.v[0]);
      auto desc = [&](uint32_t lo) { return (uint64_t(hi) << 32) | lo; };
      constexpr uint32_t kKvStep = kKvBytes >> 4, kQStep = 2 * kQHalf >> 4;   // in a descriptor's 16-byte units
      bool ok = true;
      // two walks over the KV tiles of all this pair's tiles: scores three ahead of products
      AttnTile t;
      int q_round = 0, q_left = 0, qi = 0, qph = 0;
      // the next KV tile's scores can be issued: its Q is there
      auto next_q = [&]() -> bool {
        if (q_left == 0) {
          q_left = -1;
          if (find_tile(pass, q_round, t, false)) {
            ++q_round;
            q_left = t.n_kv;
            ok = mbar_wait(&sm.q_full[qi], qph, abort_word);
          }
        }
        return ok && q_left > 0;
      };
      auto issue_qk = [&](int slot, int b) {
        const uint32_t q0 = q_lo + qi * kQStep, k0 = k_lo + slot * kKvStep, d = tmem + b * 128;
#pragma unroll
        for (int k = 0; k < kD / 16; ++k)
          umma_ss_pair(d, desc(q0 + (k >> 2) * (kQHalf >> 4) + (k & 3) * 2), desc(k0 + (k >> 2) * (kKHalf >> 4) + (k & 3) * 2),
                       idesc_qk, k > 0 ? 1u : 0u);
        umma_commit_pair(&sm.s_full[b]);
        if (--q_left == 0) {
          umma_commit_pair(&sm.q_empty[qi]);
          if (++qi == 2) { qi = 0; qph ^= 1; }
        }
      };
      for (int i = 0; i < kSBufs && next_q(); ++i) {
        ok = mbar_wait(&sm.kv_full[i], 0, abort_word);
        if (!ok) break;
        tc_fence_after();
        issue_qk(i, i);
        umma_commit_pair(&sm.kv_empty[i]);
      }
      int slot = kSBufs, ph = 0, b = 0, bph = 0, n_tiles_done = 0;
      for (int round = 0; ok && find_tile(pass, round, t, false); ++round) {
        const int n = t.n_kv;
        const int4* subs = kv_subs + t.kv_off;
        int flags = subs[0].w;
        for (int j = 0; j < n && ok; ++j) {
          // the three barriers are asked at once: an answer takes 200 cycles and more
          const bool kv_there = mbar_test_wait(&sm.kv_full[slot], ph), p0_there = mbar_test_wait(&sm.p_ready[b][0], bph),
                     p1_there = mbar_test_wait(&sm.p_ready[b][1], bph);
          const uint32_t hold_a = (flags & 1) - 1u, hold_b = ((flags >> 1) & 1) - 1u;   // all ones: the query tile sees none of the keys
          if (j + 1 < n) flags = subs[j + 1].w;
          if (!kv_there) ok = mbar_wait(&sm.kv_full[slot], ph, abort_word);
          if (ok && j == 0) ok = mbar_wait(&sm.o_empty, n_tiles_done & 1, abort_word);   // the last result is in registers
          const uint32_t v0 = v_lo + slot * kKvStep, a = tmem + b * 128;
#pragma unroll
          for (int h = 0; h < 2 && ok; ++h) {   // O += P V: the first 64 keys while the softmax warps still work on the others
            if (!(h ? p1_there : p0_there)) ok = mbar_wait(&sm.p_ready[b][h], bph, abort_word);
            if (!ok) break;
            tc_fence_after();
            if ((hold_a | hold_b) == 0) {
#pragma unroll
              for (int k = 4 * h; k < 4 * h + 4; ++k)
                umma_ts_pair(tmem + kSBufs * 128, a + k * 8, desc(v0 + k * 128), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
            } else {
#pragma unroll 1
              for (int k = 4 * h; k < 4 * h + 4; ++k)
                umma_ts_pair_hold(tmem + kSBufs * 128, a + k * 8, desc(v0 + k * 128), idesc_pv, (j > 0 || k > 0) ? 1u : 0u,
                                  hold_a, hold_b);
            }
          }
          if (!ok) break;
          if (j + 1 == n) umma_commit_pair(&sm.acc_full);
          // S(j+3) goes where P(j) was: behind the product that reads it
          if (next_q()) issue_qk(slot, b);
          umma_commit_pair(&sm.kv_empty[slot]);
          if (++slot == kSlots) { slot = 0; ph ^= 1; }
          if (++b == kSBufs) { b = 0; bph ^= 1; }
        }
        n_tiles_done += ok;
      }
      // TMEM and operands stay until all has retired
      if (!ok) { umma_commit_pair(&sm.acc_full); ++n_tiles_done; }
      for (int spin = 0; spin < 200000 && n_tiles_done > 0 && !mbar_try_wait(&sm.acc_full, (n_tiles_done - 1) & 1); ++spin) {}
    }
    __syncwarp();
    if (!next_pass(pass)) break;
   }
   } else {
    // ------------------------------------------------------------ operand fetch for the next stage
    run_copy_jobs(jobs, n_jobs, copy_ctx, blockIdx.x, gridDim.x, threadIdx.x - 320, 64);
    __syncwarp();
    if (next_pass(0)) next_pass(1);
   }
  } else {
    // ------------------------------------------------------------ softmax of every second KV tile
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    const int wg = warp >> 2, quad = warp & 3, r = threadIdx.x & 127;
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const uint32_t o_addr = tmem + lane_base + kSBufs * 128;
    const uint32_t p_bar = cluster_addr(smem_u32(&sm.p_ready[0][0]), 0);
    const float sl2 = scale * 1.4426950408889634f;
   for (int pass = 0;; ++pass) {
    bool ok = true, ready = false;
    int b = wg, bph = 0;       // buffer of this warpgroup's next KV tile, counted over all tiles
    int g0 = 0;                // KV tiles before this tile
    uint32_t published = 0;    // parities of the references handed on so far through either slot of `info`
    for (int info = 0, iph = 0;;) {
      // ---- next tile
      TileInfo& ti = sm.info[info];
      const uint32_t pub = published >> info;
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&sm.info_full[info], iph, abort_word));
      if (!ok || ti.n_kv < 0) break;
      const int n = ti.n_kv;
      const int4* subs = kv_subs + ti.kv_off;
      const int4 mk = r < ti.n_rows ? ti.mask[r] : none;
      const int first = wg ^ (g0 & 1);
      int4 ahead = ti.first[first];
      const bool sees = mk.y > mk.x || mk.w > mk.z;
      float m_ref = sees ? -INFINITY : 0.f, l_run = 0.f;   // the row's reference, as far as this warpgroup knows; its own sum
      bool exchange = pass > 0 || __any_sync(0xffffffffu, m_ref == -INFINITY);
      int n_pub = exchange ? n : 0;
      for (int j = first; j < n; j += 2) {
        const int4 sub = ahead;
        if (j + 2 < n) ahead = subs[j + 2];
        const uint32_t s_addr = tmem + lane_base + b * 128;
        const bool need = (sub.w >> X) & 1;
        if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(&sm.s_full[b], bph, abort_word));
        if (!ok) break;
        tc_fence_after();
        uint32_t sreg[128];
        if (need) {
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + c * 32, sreg + c * 32);
          tmem_wait_ld();
          if (!((sub.w >> (2 + X)) & 1)) {
            // the keys this row sees as one bit each: a range costs a handful of instructions per 32 keys and an
            // element one test, where comparing every key with four bounds costs six per element
            const int a0 = mk.x - sub.y, b0 = min(max(mk.y, mk.x) - sub.y, sub.z), a1 = mk.z - sub.y,
                      b1 = min(max(mk.w, mk.z) - sub.y, sub.z);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const uint32_t see = bits_between(a0 - 32 * w, b0 - 32 * w) | bits_between(a1 - 32 * w, b1 - 32 * w);
#pragma unroll
              for (int c = 0; c < 32; ++c)
                if (!((see >> c) & 1u)) sreg[32 * w + c] = 0xff800000u;   // -inf
            }
          }
        }
        if (exchange) {
          // what the warp that has the previous tile left behind
          float m_cur = m_ref;
          if (j > 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sm.m_ready[info][quad], (pub + j - 1) & 1, abort_word));
            if (!ok) break;
            m_cur = ti.m[r];
          }
          float m_new = m_cur;
          if (pass == 0 && __all_sync(0xffffffffu, m_cur != -INFINITY)) {
            exchange = false;   // settled by the other warpgroup
            n_pub = j;
          } else {
            if (need) {
              float mxp[8];   // eight chains: a single one would be 64 dependent steps
#pragma unroll
              for (int i = 0; i < 8; ++i) mxp[i] = -INFINITY;
#pragma unroll
              for (int c = 0; c < 64; ++c)
                mxp[c & 7] = fmax3(mxp[c & 7], __uint_as_float(sreg[2 * c]), __uint_as_float(sreg[2 * c + 1]));
              const float mx = fmaxf(fmaxf(fmaxf(mxp[0], mxp[1]), fmaxf(mxp[2], mxp[3])),
                                     fmaxf(fmaxf(mxp[4], mxp[5]), fmaxf(mxp[6], mxp[7])));
              m_new = (mx > m_cur + kGap / sl2) ? mx : m_cur;
            }
            ti.m[r] = m_new;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.m_ready[info][quad]);
            exchange = pass > 0 || __any_sync(0xffffffffu, m_new == -INFINITY);
            if (!exchange) n_pub = j + 1;
            if (j > 0 && __any_sync(0xffffffffu, m_new != m_cur)) {
              // no product may be adding to O; that of KV tile j - 3 has retired, as S(j) came after it, so the phase
              // is unambiguous
              const int i = g0 + j - 1 + kSBufs;   // its slot
              ok = __all_sync(0xffffffffu, mbar_wait(&sm.kv_empty[i % kSlots], (i / kSlots) & 1, abort_word));
              if (!ok) break;
              tc_fence_after();
              const float alpha = m_new != m_cur ? fast_exp2((m_cur - m_new) * sl2) : 1.f;   // exactly 1 where m stays
#pragma unroll 1
              for (int c = 0; c < 8; ++c) {
                uint32_t oreg[16];
                tmem_ld16(o_addr + c * 16, oreg);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) oreg[i] = __float_as_uint(__uint_as_float(oreg[i]) * alpha);
                tmem_st16(o_addr + c * 16, oreg);
              }
            }
          }
          if (m_ref != m_new) l_run *= fast_exp2((m_ref - m_new) * sl2);
          m_ref = m_new;
        }
        if (need) {
          const float m_sub = (m_ref == -INFINITY) ? 0.f : m_ref * sl2;
          const uint64_t sl2_2 = pack_f32x2(sl2, sl2), negm_2 = pack_f32x2(kTruncLog2 - m_sub, kTruncLog2 - m_sub);
          uint64_t ps2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            softmax_half(sreg + 64 * h, sl2_2, negm_2, ps2, s_addr + 32 * h);
            // the next scores: asked for here, where the answer is not waited for
            if (h == 1) ready = __all_sync(0xffffffffu, mbar_test_wait(&sm.s_full[b >= 1 ? b - 1 : 2], b >= 1 ? bph ^ 1 : bph));
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(p_bar + 16 * b + 8 * h);
          }
          float psp[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) unpack_f32x2(ps2[i], psp[2 * i], psp[2 * i + 1]);
          l_run += ((psp[0] + psp[1]) + (psp[2] + psp[3])) + ((psp[4] + psp[5]) + (psp[6] + psp[7]));
        } else {
          // Only the other query tile sees these keys: the product leaves O of this one alone (P times V would not,
          // where V is not finite).
          ready = false;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) { mbar_arrive_cluster(p_bar + 16 * b); mbar_arrive_cluster(p_bar + 16 * b + 8); }
        }
        b += 2;
        if (b >= kSBufs) { b -= kSBufs; bph ^= 1; }
      }
      // ---- the row's sum, for the reference it ends with
      float m_fin = m_ref;
      if (n > 0 && ok && exchange && ((g0 + n - 1) & 1) != wg) {
        ok = mbar_wait(&sm.m_ready[info][quad], (pub + n - 1) & 1, abort_word);
        m_fin = ti.m[r];
      }
      ti.l[wg][r] = l_run != 0.f ? l_run * fast_exp2((m_ref - m_fin) * sl2) : 0.f;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      published ^= uint32_t(n_pub & 1) << info;
      g0 += n;
      __syncwarp();
      if (lane == 0) { mbar_arrive(&sm.l_ready[info][quad]); mbar_arrive(&sm.info_empty[info]); }
      if (++info == kInfos) { info = 0; iph ^= 1; }
    }
    if (!next_pass(pass)) break;
   }
  }
  // nobody reads or signals the other CTA's shared memory any more
  if (warp == 9) tmem_dealloc_pair(tmem, 512);
  if (threadIdx.x == 0 && sm.abort_word) atomicExch(status, kStatusBarrierTimeout);
}

static std::atomic<uint64_t> g_pair_smem_raised[6];

}  // namespace dcpk

void dcpk_fill_copy_ctx(dcpk::CopyCtx* ctx, void* const* src_ptrs, void* const* dst_ptrs, int stat_stride);

using namespace dcpk;

// Same contract as dcpk_attn_fwd, for tile tables built with 256-row tiles (AttnTile.n_rows <= 256):
// `kv_entries` is the KvSub list (AttnTile.kv_off / n_kv index it), n_mask_rows / n_kv_entries are the
// lengths of the mask table and of that list (bounds checks).  Destinations from n_dst_a on are rows of `out_channels`
// (a multiple of 8, at most 128) of type `out_type` (0 fp32, 1 fp16, 2 bf16), those before it bf16 rows of 128; all
// 16-byte aligned.  A pass of its own for the caller's form took 6.5 us of 218 for 7680 tokens of 64 fp32 channels,
// forward and backward.
extern "C" int dcpk_attn_fwd_pair(const void* q_arena, long q_rows, const void* kv_arena, long kv_rows, int hq,
                                  int hkv, const void* tiles, int n_tiles, const void* kv_entries, int n_kv_entries,
                                  const void* masks, int n_mask_rows, void* const* out_ptrs, float* const* lse_ptrs,
                                  int n_dst, int lse_stride_a, int lse_stride_b, int n_dst_a, int out_type, int out_channels,
                                  float scale, int channels, const void* jobs, int n_jobs, void* const* job_src_ptrs,
                                  void* const* job_dst_ptrs, int job_stat_stride, int* status, void* stream) {
  if (n_tiles <= 0) return n_jobs > 0 ? -6 : 0;   // copy jobs need a kernel to ride on
  if (n_dst > kMaxPeers || hq % hkv != 0 || channels < 1 || channels > kHeadDim || out_type < 0 || out_type > 2 || out_channels < 8 ||
      out_channels > kHeadDim || out_channels % 8 != 0)
    return -3;
  CUtensorMap tm_q, tm_k, tm_v;
  if (encode_arena_map(&tm_q, q_arena, uint64_t(q_rows), uint32_t(hq), kHeadDim, 128)) return -1;
  if (encode_arena_map(&tm_k, kv_arena, uint64_t(kv_rows), uint32_t(2 * hkv), kHeadDim, 64)) return -1;
  if (encode_arena_map(&tm_v, kv_arena, uint64_t(kv_rows), uint32_t(2 * hkv), kHeadDim, 128)) return -1;
  PeerPtrs pp;
  for (int i = 0; i < kMaxPeers; ++i) {
    pp.out[i] = i < n_dst ? out_ptrs[i] : nullptr;
    pp.lse[i] = i < n_dst ? lse_ptrs[i] : nullptr;
  }
  CopyCtx ctx;
  dcpk_fill_copy_ctx(&ctx, n_jobs > 0 ? job_src_ptrs : nullptr, n_jobs > 0 ? job_dst_ptrs : nullptr, job_stat_stride);
  const int smem = int(sizeof(PairSmem)) + 1024;
  const bool form = out_type != 2 || out_channels != kHeadDim;
  const int v = (channels > 96 ? 0 : channels > 64 ? 1 : 2) + 3 * form;
  auto kernel = v == 5 ? attn_fwd_pair_kernel<64, true> : v == 4 ? attn_fwd_pair_kernel<96, true>
              : v == 3 ? attn_fwd_pair_kernel<128, true> : v == 2 ? attn_fwd_pair_kernel<64, false>
              : v == 1 ? attn_fwd_pair_kernel<96, false> : attn_fwd_pair_kernel<128, false>;
  if (raise_smem_limit(kernel, smem, g_pair_smem_raised[v]) != cudaSuccess) return -4;
  // short calls begin while the kernel before them ends (see kSmallPass in attn_edge.cu; a round is 5 us and more)
  const cudaError_t rc = launch_overlapped(
      kernel, 2 * std::min(n_tiles, kPairs), kPairThreads, smem, static_cast<cudaStream_t>(stream), 1, n_tiles <= 8 * kPairs,
      tm_q, tm_k, tm_v, static_cast<const AttnTile*>(tiles), n_tiles, static_cast<const int4*>(kv_entries),
      static_cast<const int4*>(masks), pp, hq, hkv, lse_stride_a, lse_stride_b, n_dst_a, n_dst, out_type, out_channels, int(q_rows),
      n_mask_rows, n_kv_entries, scale, static_cast<const CopyJob*>(jobs), n_jobs, ctx, status);
  return rc == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -5;
}
