// The exclusive prefix sum of a device array in place, in one launch (see
// sf_lookback.cuh): a block per SM, taking tiles of kScanTile elements in
// turn up to the device-side length.

#include "sf_host.hh"
#include "sf_lookback.cuh"

namespace sf {
namespace {

template <typename V>
__global__ void __launch_bounds__(kScanThreads)
    scan_in_place(V *v, const uint64_t *len, V *total_out, uint32_t *counter, uint64_t *words,
                  int32_t *status) {
  scan_tiles(v, *len, total_out, counter, words, status);
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
