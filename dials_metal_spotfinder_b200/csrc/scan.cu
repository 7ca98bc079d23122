// The exclusive prefix sum of a device array in place, in one launch (see
// sf_lookback.cuh): a block per SM, taking tiles of kScanTile elements in
// turn up to the device-side length.

#include "sf_host.hh"
#include "sf_lookback.cuh"

namespace sf {
namespace {

constexpr unsigned kFull = 0xffffffffu;

template <typename V>
__global__ void __launch_bounds__(kScanThreads)
    scan_in_place(V *v, const uint64_t *len, V *total_out, uint32_t *counter, uint64_t *words,
                  int32_t *status) {
  const uint64_t n = *len;
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
      const V t = __shfl_up_sync(kFull, incl, d);
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

} // namespace

template <typename V>
void launch_scan(V *v, const uint64_t *len, V *total, uint32_t *counter, uint64_t *words,
                 int32_t *status, unsigned grid, cudaStream_t s) {
  scan_in_place<V><<<grid, kScanThreads, 0, s>>>(v, len, total, counter, words, status);
}
template void launch_scan(uint32_t *, const uint64_t *, uint32_t *, uint32_t *, uint64_t *,
                          int32_t *, unsigned, cudaStream_t);
template void launch_scan(uint64_t *, const uint64_t *, uint64_t *, uint32_t *, uint64_t *,
                          int32_t *, unsigned, cudaStream_t);

} // namespace sf
