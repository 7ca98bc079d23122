// The bounded wait of the tile prefixes (csrc/sf_lookback.cuh): a block whose
// earlier tiles have all published gets their prefix; one that waits for tiles
// that nothing publishes gives up, with the status set, a prefix of 0 and its
// own tile published, and what the caller is told says so.
#include <cstdio>

#include "../../dials_metal_spotfinder_b200/csrc/sf_lookback.cuh"

namespace {

struct Result {
  unsigned long long prefix;
  int status;
};

__global__ void __launch_bounds__(sf::kTileThreads)
    take_prefix(uint64_t *words, uint64_t tile, uint64_t sum, Result *out) {
  __shared__ sf::TileTurn turn;
  __shared__ int status;
  if (threadIdx.x == 0) {
    turn.tile = tile;
    turn.late = false;
    status = sf::kLabelOk;
  }
  __syncthreads();
  const uint64_t prefix = sf::tile_prefix(&turn, words, sum, &status);
  __syncthreads();
  if (threadIdx.x == 0)
    *out = Result{prefix, status};
}

} // namespace

int main() {
  using namespace sf;
  constexpr int kTiles = 4;
  const uint64_t published[kTiles] = {kTileDone | 5, kTileSum | 7, kTileSum | 11, 0};
  uint64_t *words = nullptr;
  Result *out = nullptr;
  if (cudaMalloc(&words, sizeof(published)) != cudaSuccess ||
      cudaMallocHost(&out, sizeof(Result)) != cudaSuccess)
    return 2;
  for (int late = 0; late < 2; late++) {
    if (late)
      cudaMemset(words, 0, sizeof(published));
    else
      cudaMemcpy(words, published, sizeof(published), cudaMemcpyHostToDevice);
    take_prefix<<<1, kTileThreads>>>(words, kTiles - 1, 13, out);
    uint64_t own = 0;
    if (cudaMemcpy(&own, words + kTiles - 1, sizeof(own), cudaMemcpyDeviceToHost) != cudaSuccess)
      return 2;
    std::printf("prefix %llu status %d own %llu done %d\n", out->prefix, out->status,
                static_cast<unsigned long long>(own & kTileValue), own >= kTileDone);
  }
  std::printf("%s\n%s\n", label_error("grouping", kLabelWaitTimeout).c_str(),
              label_error("grouping", kLabelLiveOverflow).c_str());
  return 0;
}
