// Ordered compaction of the threshold's staged records into per-frame lists
// ascending by pixel index. This replaces the reference's host-side sort of
// the device emit (src/signal_order.cc:19-72 called from
// src/dext_cuda.cu:718-720): the tiles are already in index order, so an
// exclusive scan of their counts places every record directly.
//
// One launch, in which no block waits on another. The threshold has left
// each tile's count and, per group of kPlaceTiles tiles, their sum; a
// frame's tiles start at a multiple of kPlaceTiles, so every group belongs
// to one frame. The blocks of a group each
//   - add up the sums of the frame's groups before theirs (a 16M frame has
//     77, one read a thread): where the group's records start in the list;
//   - scan the group's counts, 32 tiles a warp at a time: where each 32
//     tiles' records start;
//   - copy their share of these, a warp per 32 tiles and a record per lane,
//     each lane finding its tile by a binary search over the lanes' prefix
//     counts.
// Bound: 32 bytes moved per record; small batches by latency, which is why a
// group is then shared by up to kPlaceSlices blocks. One launch took the place
// of three (a reduction, a scan, a copy of one block per group): 20 -> 7 us
// for one 2162 x 2068 uint16 frame, 89 -> 75 us for 16 of 4362 x 4148 (10.5 M
// records, 4.5 TB/s).

#include "sf_host.hh"

namespace sf {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = kPlaceThreads / 32;
constexpr int kGroups = kPlaceTiles / 32; // 32-tile pieces of a group
static_assert(kGroups == 32, "a piece per lane");

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, v, d);
    if (lane >= d)
      v += t;
  }
  return v;
}

__global__ void __launch_bounds__(kPlaceThreads) place_copy(PlaceLaunch L) {
  __shared__ int frame_s;
  __shared__ uint32_t before_s[kWarps], all_s[kWarps];
  __shared__ uint32_t piece_s[kGroups];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t group = blockIdx.x;
  const uint64_t tile0 = static_cast<uint64_t>(group) * kPlaceTiles;

  // the frame whose tiles these are: the last one starting at or before
  for (int f = threadIdx.x; f < L.nframes; f += kPlaceThreads)
    if (L.frames[f].tile_base <= tile0 &&
        (f + 1 == L.nframes || L.frames[f + 1].tile_base > tile0))
      frame_s = f;
  // each warp's pieces: their sums
  for (int p = warp; p < kGroups; p += kWarps) {
    const uint64_t tile = tile0 + p * 32 + lane;
    const uint32_t c = tile < L.ntiles ? L.tile_count[tile] : 0u;
    const uint32_t sum = __reduce_add_sync(kFull, c);
    if (lane == 0)
      piece_s[p] = sum;
  }
  __syncthreads();
  const int f = frame_s;
  const FrameDesc fd = L.frames[f];
  const uint32_t first = static_cast<uint32_t>(fd.tile_base / kPlaceTiles);
  const uint32_t groups = static_cast<uint32_t>(
      (static_cast<uint64_t>(fd.height) * fd.strips + kPlaceTiles - 1) / kPlaceTiles);
  const bool counts = group == first && blockIdx.y == 0; // writes the frame's count
  uint32_t before = 0, all = 0;
  for (uint32_t i = threadIdx.x; i < (counts ? groups : group - first); i += kPlaceThreads) {
    const uint32_t v = L.block_sums[first + i];
    all += v;
    if (i < group - first)
      before += v;
  }
  before = __reduce_add_sync(kFull, before);
  all = __reduce_add_sync(kFull, all);
  if (lane == 0) {
    before_s[warp] = before;
    all_s[warp] = all;
  }
  __syncthreads();
  before = 0;
  all = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    before += before_s[w];
    all += all_s[w];
  }
  if (counts && threadIdx.x == 0) {
    L.frame_count[f] = all;
    if (group == 0) {
      const int status = *L.run_status;
      *L.status = status;
      if (L.head) {
        L.head->count = all;
        L.head->status = status;
      }
    }
  }
  const uint32_t mine = piece_s[lane];
  const uint32_t piece_at = warp_incl_scan(mine, lane) - mine; // of piece `lane`

  const uint4 *pool = reinterpret_cast<const uint4 *>(L.pool);
  uint4 *out = reinterpret_cast<uint4 *>(L.out) + fd.out_base;
  for (int p = blockIdx.y * kWarps + warp; p < kGroups; p += gridDim.y * kWarps) {
    const uint32_t total = __shfl_sync(kFull, mine, p);
    if (total == 0)
      continue;
    const uint32_t at = before + __shfl_sync(kFull, piece_at, p);
    const uint64_t tile = tile0 + p * 32 + lane;
    const uint32_t c = tile < L.ntiles ? L.tile_count[tile] : 0u;
    const uint32_t incl = warp_incl_scan(c, lane);
    // a tile's records are pool[src + k] for its ranks k of this piece
    const uint32_t src = (c ? L.tile_start[tile] : 0u) - (incl - c);
    constexpr int kU = 4; // records a lane at a time, read before the first store
    for (uint32_t base = 0; base < total; base += 32 * kU) {
      uint4 v[kU];
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const uint32_t k = base + 32 * u + lane;
        // the tile of record k: the first whose inclusive count exceeds k
        uint32_t t = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
          const uint32_t n = __shfl_sync(kFull, incl, static_cast<int>(t + step - 1));
          if (n <= k)
            t += step;
        }
        const uint32_t s = __shfl_sync(kFull, src, static_cast<int>(t));
        if (k < total && at + k < fd.capacity)
          v[u] = pool[s + k];
      }
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const uint32_t k = base + 32 * u + lane;
        if (k < total && at + k < fd.capacity) {
          out[at + k] = v[u];
          if (L.head && at + k < HostHead::kRecords)
            reinterpret_cast<uint4 *>(L.head->list)[at + k] = v[u];
        }
      }
    }
  }
}

} // namespace

cudaError_t launch_place(const PlaceLaunch &L, cudaStream_t stream) {
  const uint32_t groups = static_cast<uint32_t>((L.ntiles + kPlaceTiles - 1) / kPlaceTiles);
  if (groups == 0)
    return cudaSuccess;
  // blocks enough for every SM, as far as a group can be shared
  uint32_t slices = 1;
  while (slices < kPlaceSlices && groups * slices < static_cast<uint32_t>(2 * L.sms))
    slices *= 2;
  place_copy<<<dim3(groups, slices), kPlaceThreads, 0, stream>>>(L);
  return cudaGetLastError();
}

} // namespace sf
