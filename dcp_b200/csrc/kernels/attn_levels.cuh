// Levels of dQ: buffers that make its sums the same in every run.
//
// A row of dQ is added to by every key tile that it sees, as these come.  Two additions to zero give the same bits in
// either order, three do not: with a workspace each 256 keys (of the positions of an item's concatenated KV) have a
// buffer of their own, a level, and the levels are summed afterwards, in their order.  Level 0 is the accumulator
// itself, and the only one without a workspace.
#pragma once
#include <stdint.h>

#include "entries.h"

namespace dcpk {

// One item of the backward kernel = one query tile (up to 128 rows) that attends to a key tile; a CTA visits it once
// per query head it covers, so the table does not grow with the head count.
struct BwdItemDesc {
  int q_row;     // arena row of the query tile (same row addresses Q, dO, lse, delta)
  int n_rows;    // valid queries
  int kv_pos0;   // position of this CTA's first key inside the item's concatenated KV
  int mask_row;  // row in the range table
  int dq_dev;    // destination index of the dQ accumulator
  int dq_row;    // arena row in that accumulator
  int full;      // 1: every (query, key) pair of the tile is allowed
  int pad;
};

__device__ __forceinline__ int dq_level(int kv_pos0, int n_levels) {
  const int level = kv_pos0 >> 8;
  return level > 0 && level < n_levels ? level : 0;
}

inline int level_pitch(int channels) { return channels > 64 ? 128 : 64; }   // floats of a head's row in the workspace

// What kernels need to know of them; n_levels < 2: there are none.
struct DqLevels {
  const BwdItemDesc* items;
  float* buf;          // [n_levels - 1, q_rows, hq, pitch]
  int n_items, n_levels, q_rows, hq, channels, pitch;
};

inline DqLevels make_levels(const DcpkDqLevels* l) {
  if (!l || !l->workspace) return DqLevels{};
  return DqLevels{static_cast<const BwdItemDesc*>(l->items), static_cast<float*>(l->workspace), l->n_items, l->n_levels,
                  l->q_rows, l->hq, l->channels, level_pitch(l->channels)};
}

// A block works on so many rows at a time; which levels they have is in the items that cover them, so it looks through
// the whole table (a row at a time per warp, with a look each: 13 and 14 us for clearing and summing 42 MB, 10.5 and 13
// this way).
static constexpr int kLevelRows = 4;
struct RowLevels { uint32_t bits[kLevelRows][2]; };   // in shared memory

__device__ __forceinline__ void find_levels(const DqLevels& lv, int row0, RowLevels& rows) {   // by all threads of the block
  __syncthreads();
  if (threadIdx.x < 2 * kLevelRows) rows.bits[threadIdx.x >> 1][threadIdx.x & 1] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < lv.n_items; i += blockDim.x) {
    const BwdItemDesc d = lv.items[i];
    if (d.dq_dev != 0) continue;
    const int level = dq_level(d.kv_pos0, lv.n_levels);
    for (int row = max(d.dq_row, row0); row < min(min(d.dq_row + d.n_rows, lv.q_rows), row0 + kLevelRows); ++row)
      atomicOr(&rows.bits[row - row0][level >> 5], 1u << (level & 31));
  }
  __syncthreads();
}
__device__ __forceinline__ uint64_t levels_above(const RowLevels& rows, int r) {   // a bit per level but the first
  return (uint64_t(rows.bits[r][1]) << 32 | rows.bits[r][0]) & ~uint64_t(1);
}

// f(p): for each level of `left`, in their order, `p` the one of four channels that begin at `at` in the first buffer
template <typename F>
__device__ __forceinline__ void for_levels(const DqLevels& lv, uint64_t left, size_t at, F f) {
  const size_t size = size_t(lv.q_rows) * lv.hq * lv.pitch;
  for (; left != 0; left &= left - 1) f(reinterpret_cast<float4*>(lv.buf + (__ffsll(left) - 2) * size + at));
}

// clears the levels that the rows from `row0` on will be added to in
__device__ __forceinline__ void clear_levels(const DqLevels& lv, int row0, RowLevels& rows) {
  find_levels(lv, row0, rows);
  const int quads = lv.pitch / 4, per_row = lv.hq * quads;
  for (int c = threadIdx.x; c < kLevelRows * per_row; c += blockDim.x) {
    const int r = c / per_row, k = c % quads * 4;
    if (k >= lv.channels) continue;
    for_levels(lv, levels_above(rows, r), (size_t(row0 + r) * lv.hq + c % per_row / quads) * lv.pitch + k,
               [](float4* p) { *p = make_float4(0.f, 0.f, 0.f, 0.f); });
  }
}

// sum += the levels of `left` of four channels
__device__ __forceinline__ void add_levels(const DqLevels& lv, uint64_t left, size_t at, float4& sum) {
  const size_t size = size_t(lv.q_rows) * lv.hq * lv.pitch;
  while (left != 0) {
    float4 v[4];   // of four levels in flight
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (left != 0) v[u] = *reinterpret_cast<const float4*>(lv.buf + (__ffsll(left) - 2) * size + at);
      left &= left - 1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) { sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w; }
  }
}

}  // namespace dcpk
