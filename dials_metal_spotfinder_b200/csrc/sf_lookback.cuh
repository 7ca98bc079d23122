// Prefix sums found within the launch that needs them: a kernel's blocks take
// tiles in turn, each publishes its tile's sum and adds up the sums of the
// tiles before it, a block's worth of them at a time, until it meets one that
// has published its whole prefix (Merrill and Garland, "Single-pass parallel
// prefix scan with decoupled look-back", 2016). Tiles are claimed in order
// from a counter, so every tile a block waits for is already being worked on
// by a resident block, and the waits end; each has a limit all the same,
// past which the block sets the status word and goes on with a prefix of 0
// (a position the caller's arrays hold), so that none waits for good.
// A whole block looks back, not a warp: with about a thousand tiles in
// flight, all of which have only their sums yet, 32 at a time would be 37
// round trips to L2 where 256 at a time is 5.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sf_label.hh"

namespace sf {

// A tile's word: how far it has got in the top two bits, its value (below
// 2^62) in the rest. Words are 0 before the launch.
constexpr uint64_t kTileSum = 1ull << 62, kTileDone = 2ull << 62, kTileValue = kTileSum - 1;
constexpr uint32_t kTileWaits = 1u << 20;

constexpr int kTileThreads = 256; // of every block that takes tiles

struct TileTurn {
  uint64_t tile;
  uint64_t part[kTileThreads / 32]; // per warp: its words' sum up to the first whole prefix
  bool done[kTileThreads / 32];     // whether it met one
  bool late;
};

// The block's next tile in *turn (shared memory); false when none is left.
// Every thread of the block calls it.
__device__ __forceinline__ bool next_tile(TileTurn *turn, uint32_t *counter, uint64_t tiles) {
  __syncthreads(); // the last turn's words are no longer read
  if (threadIdx.x == 0) {
    turn->tile = atomicAdd(counter, 1u);
    turn->late = false;
  }
  __syncthreads();
  return turn->tile < tiles;
}

// The sum over the tiles before this one, given this one's; every thread of
// the block calls it (with the same sum) and gets the prefix.
__device__ __forceinline__ uint64_t tile_prefix(TileTurn *turn, uint64_t *words, uint64_t sum,
                                                int32_t *status) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kWarps = kTileThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  volatile uint64_t *st = words;
  const uint64_t tile = turn->tile;
  if (tile > 0 && threadIdx.x == 0)
    st[tile] = kTileSum | sum;
  uint64_t prefix = 0;
  bool ended = tile == 0;
  for (int64_t at = static_cast<int64_t>(tile) - 1; !ended; at -= kTileThreads) {
    const int64_t i = at - static_cast<int64_t>(threadIdx.x);
    uint64_t v = kTileDone; // before the first tile
    if (i >= 0) {
      v = st[i];
      for (uint32_t tries = 0; v == 0; tries++) {
        if (tries == kTileWaits) {
          turn->late = true;
          v = kTileDone;
          break;
        }
        v = st[i];
      }
    }
    const uint32_t done = __ballot_sync(kAll, v >= kTileDone);
    // up to the nearest tile that has its prefix
    uint64_t part = lane <= (done ? __ffs(done) - 1 : 31) ? v & kTileValue : 0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
      part += __shfl_xor_sync(kAll, part, d);
    if (lane == 0) {
      turn->part[warp] = part;
      turn->done[warp] = done != 0;
    }
    __syncthreads();
    for (int w = 0; w < kWarps && !ended; w++) {
      prefix += turn->part[w];
      ended = turn->done[w];
    }
    __syncthreads(); // read by all before the next ones are written
  }
  const bool late = turn->late;
  if (late)
    prefix = 0;
  if (threadIdx.x == 0) {
    if (late)
      *status = kLabelWaitTimeout;
    st[tile] = kTileDone | ((prefix + sum) & kTileValue);
  }
  return prefix;
}

// ---- the exclusive scan of an array in place (scan.cu) ---------------------
// Its length is in device memory, so that a sequence of launches can be
// enqueued (or captured) without reading sizes back; sums stay below 2^62.
// `words` holds scan_words(the largest length) lookback words, cleared for
// this length by an earlier kernel (clear_scan_words); *counter starts at 0.
// The sum of all goes to *total, if given and the length is not 0.
constexpr int kScanThreads = kTileThreads;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

inline uint64_t scan_words(uint64_t max_len) { return max_len / kScanTile + 1; }
__device__ __forceinline__ void clear_scan_words(uint64_t *words, uint64_t len, uint64_t thread,
                                                 uint64_t threads) {
  for (uint64_t t = thread; t * kScanTile < len; t += threads)
    words[t] = 0;
}
// The scan itself, by the blocks of a launch (all of kScanThreads threads).
template <typename V>
__device__ __forceinline__ void scan_tiles(V *v, uint64_t n, V *total_out, uint32_t *counter,
                                           uint64_t *words, int32_t *status) {
  constexpr unsigned kAll = 0xffffffffu;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ TileTurn turn;
  __shared__ V sums[kScanThreads / 32];
  // read strided (coalesced), scanned per thread in array order: thread t
  // owns items base + t * kScanItems + i
  __shared__ V tile[kScanTile];
  while (next_tile(&turn, counter, tiles)) {
    const uint64_t base = turn.tile * kScanTile;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      const uint64_t at = base + i * kScanThreads + threadIdx.x;
      tile[i * kScanThreads + threadIdx.x] = at < n ? v[at] : V(0);
    }
    __syncthreads();
    V mine[kScanItems], run = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      mine[i] = tile[threadIdx.x * kScanItems + i];
      run += mine[i];
    }
    V incl = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const V t = __shfl_up_sync(kAll, incl, d);
      if (lane >= d)
        incl += t;
    }
    if (lane == 31)
      sums[warp] = incl;
    __syncthreads();
    V before = incl - run, total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; w++) {
      if (w < warp)
        before += sums[w];
      total += sums[w];
    }
    const V prefix = static_cast<V>(tile_prefix(&turn, words, total, status));
    if (total_out && turn.tile == tiles - 1 && threadIdx.x == 0)
      *total_out = prefix + total;
    before += prefix;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      tile[threadIdx.x * kScanItems + i] = before;
      before += mine[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      const uint64_t at = base + i * kScanThreads + threadIdx.x;
      if (at < n)
        v[at] = tile[i * kScanThreads + threadIdx.x];
    }
  }
}
template <typename V>
void launch_scan(V *v, const uint64_t *len, V *total, uint32_t *counter, uint64_t *words,
                 int32_t *status, unsigned grid, cudaStream_t s);

} // namespace sf
