// How the decode kernels over latent rows share a batch: the (row, key tile) units are numbered row by row and cut into equal runs, one per
// CTA, whatever the lengths.
#pragma once
#include <cuda_runtime.h>

#include "latent_attention.cuh"

namespace fa {
namespace hybrid {
namespace {

constexpr int KT = 64;         // keys per tile

__device__ __forceinline__ int row_tiles_of(const LatentAttentionArgs& a, long long row) {
  const int n = a.positions[row] + 1;
  return n > 0 ? (n + KT - 1) / KT : 1;
}

// Inclusive scan over the block of one int per thread; `buf` holds one int per warp.
__device__ __forceinline__ int block_scan(int v, int* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) buf[warp] = v;
  __syncthreads();
  int add = 0;
  for (int i = 0; i < warp; ++i) add += buf[i];
  __syncthreads();
  return v + add;
}

// My units [u0, u1), found[0]: the row of the first one, found[1]: that row's first unit.  False if there are none for this CTA.  All THREADS of the
// block call it; `buf` holds one int per warp, `found` two.  The grid's first CTA writes the prefix sums of the rows' tiles for the merge.
template <int THREADS>
__device__ __forceinline__ bool find_run(const LatentAttentionArgs& a, int* buf, int* found, int& u0, int& u1) {
  const int tid = threadIdx.x, cta = blockIdx.x;
  int total = 0, mine = 0, upto = 0;               // of my row in the last block of rows: its tiles, tiles up to and with it
  for (long long r0 = 0; r0 < a.rows; r0 += THREADS) {
    mine = r0 + tid < a.rows ? row_tiles_of(a, r0 + tid) : 0;
    upto = total + block_scan(mine, buf);
    if (cta == 0 && blockIdx.y == 0 && r0 + tid < a.rows) a.row_tiles[r0 + tid + 1] = upto;
    if (tid == THREADS - 1) found[0] = upto;
    __syncthreads();
    total = found[0];
    __syncthreads();
  }
  if (cta == 0 && blockIdx.y == 0 && tid == 0) a.row_tiles[0] = 0;
  const int per = (total + a.n_cta - 1) / a.n_cta;
  u0 = cta * per;
  u1 = min(u0 + per, total);
  if (u0 >= u1) return false;
  if (a.rows <= THREADS) {
    if (mine > 0 && upto - mine <= u0 && u0 < upto) { found[0] = tid; found[1] = upto - mine; }
    __syncthreads();
  } else {
    int base = 0;
    for (long long r0 = 0; r0 < a.rows; r0 += THREADS) {
      const int v = r0 + tid < a.rows ? row_tiles_of(a, r0 + tid) : 0;
      const int inc = base + block_scan(v, buf);
      if (v > 0 && inc - v <= u0 && u0 < inc) { found[0] = (int)(r0 + tid); found[1] = inc - v; }
      if (tid == THREADS - 1) buf[0] = inc;
      __syncthreads();
      base = buf[0];
      __syncthreads();
      if (base > u0) break;
    }
  }
  return true;
}

// A place in the run: tile `tile` of row `row`, which has `tiles` tiles and `n` keys.
struct Cursor {
  int row, tile, tiles, n;
};
__device__ __forceinline__ void start_row(const LatentAttentionArgs& a, Cursor& c, int row) {
  c.row = row;
  c.tile = 0;
  c.n = a.positions[row] + 1;
  c.tiles = c.n > 0 ? (c.n + KT - 1) / KT : 1;
}
__device__ __forceinline__ void advance(const LatentAttentionArgs& a, Cursor& c) {
  if (++c.tile == c.tiles && c.row + 1 < a.rows) start_row(a, c, c.row + 1);
}
// Pool page of block `blk` (16 keys) of the cursor's tile; keys past the end: the tile's first page (any finite rows will do, their weights are
// zero).  -1: no such page.
__device__ __forceinline__ int page_of(const LatentAttentionArgs& a, const Cursor& c, int blk) {
  const int seq = a.tok_seq[c.row];
  int b = c.tile * (KT / 16) + blk;
  if (b * 16 >= c.n) b = c.tile * (KT / 16);
  return seq >= 0 && seq < a.n_seq && c.n > 0 && b < a.max_blocks ? a.block_table[(long long)seq * a.max_blocks + b] : -1;
}

}  // namespace
}  // namespace hybrid
}  // namespace fa
