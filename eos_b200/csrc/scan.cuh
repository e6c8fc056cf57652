// Device-wide exclusive scans inside one launch, for the per-round and per-level compactions
// of the hierarchy builders.  A block takes its tile by a ticket, scans its own values in
// shared memory and gets the sum of all earlier tiles by looking back over their published
// sums (Merrill & Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back",
// 2016).  Tickets are taken in order by running blocks, so the tiles waited for always run.
#pragma once
#include "eos_internal.cuh"

namespace eos {

constexpr int kScanBlock = 256;
constexpr int kNoTile = 0x7fffffff;

// This block's next tile; kNoTile once a look-back of the call has given up (raised the timeout
// bit), so that no later launch reads what the tile that gave up left unwritten.  One thread.
__device__ __forceinline__ int take_tile(int* tickets, const int* err) {
  const int tile = atomicAdd(tickets, 1);
  return *(const volatile int*)err & kErrTimeout ? kNoTile : tile;
}

template <class T>
__device__ __forceinline__ T warp_inclusive_scan(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, v, off);
    if (lane >= off) v += u;
  }
  return v;
}

// Exclusive scan of one value per thread over the block (blockDim.x a multiple of 32, at
// most 1024); every thread gets its exclusive prefix and the block's total.
template <class T>
__device__ __forceinline__ T block_exclusive_scan(T v, T& total) {
  __shared__ T warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const T inc = warp_inclusive_scan(v);
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const T s = lane < n_warps ? warp_sums[lane] : T(0);
    warp_sums[lane] = warp_inclusive_scan(s);  // inclusive prefix of the warp sums
  }
  __syncthreads();
  total = warp_sums[n_warps - 1];
  const T ex = inc - v + (warp > 0 ? warp_sums[warp - 1] : T(0));
  __syncthreads();  // warp_sums is reused by the next call
  return ex;
}

// Published sum of a tile: flag in the top two bits (1 = the tile's own sum, 2 = the sum of
// all tiles up to it, 3 = it gave up, as does who meets it), the launch's epoch in the next twelve, the value in the low 50.  A
// word of an earlier launch carries another epoch, so the array is cleared once per build,
// not per launch.  Epochs repeat after 4,095 launches: a build of more (PLOC rounds of a
// degenerate scene) must write every word it reads in each of them, which it does because
// its tiles only get fewer.
constexpr unsigned long long kTileValue = (1ull << 50) - 1;
__device__ __forceinline__ unsigned long long tile_word(unsigned flag, unsigned epoch, unsigned long long value) {
  return ((unsigned long long)flag << 62) | ((unsigned long long)(epoch & 0xfffu) << 50) | value;
}

// Sum of the tiles before `tile`, whose own sum is `sum`; called by all lanes of one warp
// with the same arguments.  kTileValue + 1 when a tile did not publish within `polls` polls
// of its word (eos_ctx::build_polls); the caller then raises the timeout bit and leaves the
// launch without writing.
__device__ __forceinline__ unsigned long long tiles_before(volatile unsigned long long* words, int tile,
                                                           unsigned long long sum, unsigned epoch, int polls) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) words[tile] = tile_word(tile == 0 ? 2u : 1u, epoch, sum);
  unsigned long long before = 0;
  for (int at = tile - 1; at >= 0; at -= 32) {
    const int i = at - lane;
    unsigned long long w = tile_word(2u, epoch, 0);  // before the first tile
    unsigned missing = 1;
    for (int poll = 0; missing && poll < polls; ++poll) {
      if (i >= 0) w = words[i];
      const bool there = (w >> 62) != 0 && ((w >> 50) & 0xfffu) == (epoch & 0xfffu);
      missing = __ballot_sync(0xffffffffu, !there);
    }
    const unsigned whole = missing ? 0 : __ballot_sync(0xffffffffu, (w >> 62) == 2u);
    const int last = whole ? __ffs(whole) - 1 : 31;  // nearest tile that holds a full prefix
    if (missing || __any_sync(0xffffffffu, lane <= last && (w >> 62) == 3u)) {
      if (lane == 0) words[tile] = tile_word(3u, epoch, 0);
      return kTileValue + 1;
    }
    unsigned long long v = lane <= last ? (w & kTileValue) : 0;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    before += v;
    if (whole) break;
  }
  if (lane == 0 && tile > 0) words[tile] = tile_word(2u, epoch, before + sum);
  return before;
}

inline int scan_blocks(long long n) { return (int)((n + kScanBlock - 1) / kScanBlock); }

}  // namespace eos
