// ThresholdPlan: the device buffers and launch geometry for thresholding one
// batch shape (one or many frames, equal or uneven sizes), built once and
// reused frame after frame. Also the TMA descriptor over each frame arena.

#include <algorithm>
#include <cstring>
#include <mutex>

#include "sf_host.hh"

namespace sf {
namespace {

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                 const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion,
                                 CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  });
  if (fn == nullptr)
    throw DeviceError("cuTensorMapEncodeTiled is not available from the driver");
  return fn;
}

// A pitched host-to-device copy runs at 29 to 49 GB/s by its row length, a
// contiguous one at 50 to 55, after which laying the rows out costs one
// launch and a pass in device memory: from page-locked memory 303 us against
// 178 for a 2162 x 2068 uint16 frame, 139 against 100 for 1062 x 1028 uint32
// and 741 against 676 for 4362 x 4148 uint16, but 14 against 18 to 24 for
// 256 x 384. The two meet at about half a megabyte.
constexpr uint64_t kLinearUpload = 512 * 1024;

uint64_t round_up(uint64_t v, uint64_t m) { return (v + m - 1) / m * m; }

// Output rows per task, and what the launch then costs. A task costs its rows
// plus the 20 rows of halo it re-reads; how long a row takes depends on the
// warps that share the SM: as 5 + w for w of them, and no less than for 7, when
// a warp waits on itself (16-bit pixels, one frame of each of several sizes
// over many heights; 0.08 us a unit). So the height with the least
// (rows + 20) x (5 + w), an SM's w taken as the most that any has when the
// blocks are dealt out, in as many rounds as they need; no shorter than kMinSeg
// rows, below which the halo is most of the work and the gain is in the noise.
// The threshold of one frame: 2162 x 2068 uint16 59 -> 52 us (17 rows; 16, the
// least there was, put a tenth warp on some SMs), 1062 x 1028 44 -> 36 us
// (6 rows), 256 x 384 35 -> 27 us (4 rows).
//
// Strips of 4 columns a lane have 2.2 times the tasks of 8, but a row of theirs
// takes 8.2 + 0.4 w units, no less than 9.5: a small frame, whose warps have an
// SM's schedulers nearly to themselves, is done sooner. Between the two forms
// the costs are not quite alike: over 40 shapes of one to 64 frames, both
// forms timed at their best heights, strips of 4 were the slower only above 1.07
// times the cost of 8 (wide, narrow us: 256 x 384 uint16 25.9, 24.2; 700 x 900
// 32.5, 28.1 at 1.03 times; 1062 x 1028 34.9, 30.8 at 1.06; 64 frames of
// 128 x 128 38.7, 40.9 at 1.07; 32 of 256 x 384 47.0, 48.9 at 1.09; 1500 x 1500
// 40.7, 42.9 at 1.13; 2162 x 2068 49.3, 53.7 at 1.18), so they are taken up
// to there.
constexpr uint64_t kNarrowPercent = 107;
struct Heights {
  int rows;
  uint64_t cost; // tenths of a unit
};
constexpr int kMinSeg = 4;
Heights choose_seg_rows(int elem_bytes, int lane_cols,
                        const std::vector<ThresholdPlan::Shape> &shapes, uint64_t sms, int wpc,
                        int blocks_per_sm) {
  const bool narrow = elem_bytes == 2 && lane_cols == 4;
  auto row_cost = [&](uint64_t w) {
    return narrow ? std::max<uint64_t>(95, 82 + 4 * w) : std::max<uint64_t>(120, 50 + 10 * w);
  };
  const uint64_t out_cols = strip_out(elem_bytes, lane_cols);
  int max_h = 1;
  for (const auto &s : shapes)
    max_h = std::max(max_h, s.height);
  Heights best{max_h, ~0ull};
  for (int seg = std::min(kMinSeg, max_h); seg <= max_h; seg++) {
    uint64_t tasks = 0;
    for (const auto &s : shapes) {
      const uint64_t strips = (s.width + out_cols - 1) / out_cols;
      tasks += strips * ((s.height + seg - 1) / seg);
    }
    const uint64_t per_block = static_cast<uint64_t>(wpc);
    const uint64_t blocks = (tasks + per_block - 1) / per_block;
    const uint64_t per_sm = (blocks + sms - 1) / sms * per_block;
    const uint64_t fit = static_cast<uint64_t>(blocks_per_sm) * per_block;
    const uint64_t rest = per_sm % fit;
    const uint64_t row = per_sm / fit * row_cost(fit) + (rest ? row_cost(rest) : 0);
    const uint64_t cost = row * static_cast<uint64_t>(std::min(seg, max_h) + 2 * kHalo);
    if (cost < best.cost)
      best = Heights{seg, cost};
  }
  return best;
}

// The form and height of a batch's tasks.
TaskShape choose_task(int elem_bytes, const std::vector<ThresholdPlan::Shape> &shapes, int wpc,
                      int blocks_per_sm) {
  const uint64_t sms = static_cast<uint64_t>(device_sm_count());
  const int wide = elem_bytes == 2 ? 8 : 4;
  const Heights h = choose_seg_rows(elem_bytes, wide, shapes, sms, wpc, blocks_per_sm);
  if (elem_bytes == 2) {
    const Heights narrow = choose_seg_rows(elem_bytes, 4, shapes, sms, wpc, blocks_per_sm);
    if (100 * narrow.cost < kNarrowPercent * h.cost)
      return TaskShape{narrow.rows, 4};
  }
  return TaskShape{h.rows, wide};
}

} // namespace

TaskShape model_task(int elem_bytes, const std::vector<ThresholdPlan::Shape> &shapes, int wpc,
                     int blocks_per_sm) {
  int occ = elem_bytes == 2 ? threshold_occupancy<uint16_t>(wpc)
                            : threshold_occupancy<uint32_t>(wpc);
  if (occ < 1)
    throw DeviceError("the threshold kernel does not fit on this device");
  if (blocks_per_sm > 0)
    occ = std::min(occ, blocks_per_sm);
  return choose_task(elem_bytes, shapes, wpc, occ);
}

void encode_arena_map(CUtensorMap *map, void *base, int elem_bytes, uint64_t pitch_elems,
                      uint64_t rows, int lane_cols) {
  const cuuint64_t dims[2] = {pitch_elems, rows};
  const cuuint64_t strides[1] = {pitch_elems * static_cast<uint64_t>(elem_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(strip_cols(lane_cols)),
                             static_cast<cuuint32_t>(kBoxRows)};
  const cuuint32_t estride[2] = {1, 1};
  const CUtensorMapDataType dt =
      elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const CUresult r = encode_fn()(map, dt, 2, base, dims, strides, box, estride,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw DeviceError("cuTensorMapEncodeTiled failed with code " + std::to_string(r));
}

cudaStream_t create_stream(int rank) {
  int least = 0, greatest = 0;
  check(cudaDeviceGetStreamPriorityRange(&least, &greatest), "cudaDeviceGetStreamPriorityRange");
  cudaStream_t s = nullptr;
  check(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, std::max(greatest, least - rank)),
        "cudaStreamCreate");
  return s;
}

int device_sm_count() {
  int dev = 0, n = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  check(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev),
        "cudaDeviceGetAttribute");
  return n;
}

ThresholdPlan::ThresholdPlan(int elem_bytes, const std::vector<Shape> &shapes,
                             const PlanTuning &tuning, int slots)
    : elem_bytes_(elem_bytes), shapes_(shapes), tuning_(tuning) {
  if (elem_bytes != 2 && elem_bytes != 4)
    throw std::invalid_argument("pixels are 16 or 32 bits");
  if (shapes.empty())
    throw std::invalid_argument("a plan needs at least one frame");
  if (slots < 1)
    throw std::invalid_argument("a plan needs at least one slot");
  // eight two-warp blocks an SM
  if (tuning_.warps_per_block == 0)
    tuning_.warps_per_block = 2;
  const int wpc = tuning_.warps_per_block;
  if (wpc != 1 && wpc != 2 && wpc != 4)
    throw std::invalid_argument("warps_per_block must be 1, 2 or 4");

  for (const Shape &s : shapes) {
    if (s.height < 1 || s.width < 1)
      throw std::invalid_argument("frame with no pixels");
    if (static_cast<uint64_t>(s.height) * s.width > 0x7fffffffull)
      throw std::invalid_argument("frame larger than INT32_MAX pixels");
  }

  const int occ = elem_bytes == 2 ? threshold_occupancy<uint16_t>(wpc)
                                  : threshold_occupancy<uint32_t>(wpc);
  if (occ < 1)
    throw DeviceError("the threshold kernel does not fit on this device");
  const int per_sm = tuning_.blocks_per_sm > 0 ? std::min(tuning_.blocks_per_sm, occ) : occ;
  sms_ = device_sm_count();
  max_blocks_ = sms_ * per_sm;
  if (tuning_.seg_rows <= 0) {
    const TaskShape t = choose_task(elem_bytes, shapes, wpc, per_sm);
    tuning_.seg_rows = t.rows;
    tuning_.lane_cols = t.lane_cols;
  }
  lane_cols_ = tuning_.lane_cols == 4 || elem_bytes != 2 ? 4 : 8;

  const int out_cols = strip_out(elem_bytes, lane_cols_);
  int32_t max_strips = 0;
  for (const Shape &s : shapes)
    max_strips = std::max(max_strips, (s.width + out_cols - 1) / out_cols);
  // Every strip reads its columns from a multiple of its output columns; the
  // pitch is a multiple of 128 bytes so each arena row starts on a TMA-friendly
  // line.
  pitch_ = round_up(static_cast<uint64_t>(max_strips) * out_cols +
                        (strip_cols(lane_cols_) - out_cols),
                    128 / elem_bytes);

  uint64_t row = 0, tile = 0, out = 0;
  uint32_t task = 0;
  for (const Shape &s : shapes) {
    FrameDesc d;
    std::memset(&d, 0, sizeof(d));
    d.row0 = static_cast<int64_t>(row + kMarginRows);
    d.height = s.height;
    d.width = s.width;
    d.strips = (s.width + out_cols - 1) / out_cols;
    d.seg_rows = std::min(tuning_.seg_rows, s.height);
    d.segments = (s.height + d.seg_rows - 1) / d.seg_rows;
    d.task_begin = task;
    tile = round_up(tile, kPlaceTiles);
    d.tile_base = tile;
    d.out_base = out;
    // The reference's list capacity: the frame's own bytes, 16 to an entry
    // (src/dext_cuda.cu:611-616), so -2 comes back on exactly the same frames.
    const uint64_t cap = static_cast<uint64_t>(s.height) * s.width * elem_bytes / 16;
    d.capacity = static_cast<uint32_t>(cap);
    host_frames_.push_back(d);
    row += static_cast<uint64_t>(s.height) + 2 * kMarginRows;
    tile += static_cast<uint64_t>(s.height) * d.strips;
    out += cap;
    task += static_cast<uint32_t>(d.strips * d.segments);
  }
  arena_rows_ = row;
  ntiles_ = tile;
  ntasks_ = task;
  total_capacity_ = out;
  if (total_capacity_ >= 0xffffffffull)
    throw std::invalid_argument("batch too large for one plan");

  grid_blocks_ = static_cast<int>(std::min<uint64_t>((ntasks_ + wpc - 1) / wpc, max_blocks_));
  int32_t tallest = 0, longest = 0;
  for (const FrameDesc &d : host_frames_) {
    tallest = std::max(tallest, d.height);
    longest = std::max(longest, d.seg_rows);
  }
  share_rows_ = longest >= kMinSharedSeg && static_cast<uint32_t>(tallest) <= kMaxSharedRows &&
                ntasks_ <= kMaxSharedTasks;
  const uint64_t warps = static_cast<uint64_t>(grid_blocks_) * wpc;
  const uint64_t chunks =
      (total_capacity_ + (kChunkRecords - kMaxStaged) - 1) / (kChunkRecords - kMaxStaged) +
      warps + 1;
  const uint64_t pool_records = chunks * kChunkRecords;
  if (pool_records >= 0xffffffffull - kChunkRecords)
    throw std::invalid_argument("batch too large for one plan");
  pool_cap_ = static_cast<uint32_t>(pool_records);

  const uint64_t arena_bytes = pitch_ * arena_rows_ * elem_bytes;
  const uint64_t nblocks = (ntiles_ + kPlaceTiles - 1) / kPlaceTiles;
  const size_t nf = host_frames_.size();
  slots_.resize(slots);
  try {
    auto alloc = [&](void **p, uint64_t bytes, const char *what) {
      check(cudaMalloc(p, std::max<uint64_t>(bytes, 16)), what);
      device_bytes_ += bytes;
    };
    alloc(reinterpret_cast<void **>(&frames_), nf * sizeof(FrameDesc), "cudaMalloc frames");
    check(cudaMemcpy(frames_, host_frames_.data(), nf * sizeof(FrameDesc),
                     cudaMemcpyHostToDevice),
          "uploading frame descriptors");
    cleared_bytes_ = warps * 8 + (ntiles_ + nblocks + 3) * 4;
    unsigned char *cleared = nullptr;
    alloc(reinterpret_cast<void **>(&cleared), cleared_bytes_, "cudaMalloc tile counts");
    ranges_ = reinterpret_cast<unsigned long long *>(cleared);
    tile_count_ = reinterpret_cast<uint32_t *>(ranges_ + warps);
    block_sums_ = tile_count_ + ntiles_;
    pool_next_ = block_sums_ + nblocks;
    next_task_ = pool_next_ + 1;
    run_status_ = reinterpret_cast<int *>(next_task_ + 1);
    alloc(reinterpret_cast<void **>(&tile_start_), ntiles_ * 4, "cudaMalloc tile starts");
    alloc(reinterpret_cast<void **>(&pool_), pool_records * sizeof(SignalPixel),
          "cudaMalloc staging pool");
    for (Slot &sl : slots_) {
      alloc(&sl.arena, arena_bytes, "cudaMalloc arena");
      check(cudaMemset(sl.arena, 0xff, arena_bytes), "filling the arena");
      alloc(reinterpret_cast<void **>(&sl.out), total_capacity_ * sizeof(SignalPixel),
            "cudaMalloc output lists");
      alloc(reinterpret_cast<void **>(&sl.frame_count), (nf + 1) * 4,
            "cudaMalloc frame counts");
      sl.status = reinterpret_cast<int *>(sl.frame_count + nf);
      check(cudaMemset(sl.frame_count, 0, (nf + 1) * 4), "clearing frame counts");
      encode_arena_map(&sl.map, sl.arena, elem_bytes_, pitch_, arena_rows_, lane_cols_);
    }
    // The fills above ran on the legacy stream; the plan's users work on
    // non-blocking streams that do not wait for it.
    check(cudaStreamSynchronize(cudaStreamLegacy), "filling the arena");
  } catch (...) {
    release();
    throw;
  }
}

ThresholdPlan::~ThresholdPlan() { release(); }

void ThresholdPlan::release() {
  for (Slot &sl : slots_) {
    cudaFree(sl.arena);
    cudaFree(sl.out);
    cudaFree(sl.frame_count);
    sl = Slot();
  }
  cudaFree(frames_);
  cudaFree(ranges_); // and what follows it
  cudaFree(tile_start_);
  cudaFree(pool_);
  cudaFree(linear_);
  linear_ = nullptr;
  frames_ = nullptr;
  tile_count_ = tile_start_ = nullptr;
  pool_ = nullptr;
  pool_next_ = block_sums_ = nullptr;
  run_status_ = nullptr;
}

void *ThresholdPlan::frame_origin(int slot, int f) const {
  const uint64_t at = static_cast<uint64_t>(host_frames_[f].row0) * pitch_ + kMarginLeft;
  return static_cast<char *>(slots_[slot].arena) + at * elem_bytes_;
}

bool ThresholdPlan::linear_copy() {
  if (!linear_ && !linear_refused_) {
    uint64_t most = 0;
    for (const Shape &s : shapes_)
      most = std::max(most, static_cast<uint64_t>(s.height) * s.width * elem_bytes_);
    if (cudaMalloc(&linear_, most) != cudaSuccess) {
      cudaGetLastError(); // no room: the pitched copy needs none, of this plan's frames
      linear_ = nullptr;
      linear_refused_ = true;
      return false;
    }
    device_bytes_ += most;
  }
  return linear_ != nullptr;
}

void ThresholdPlan::upload(int slot, int f, const void *host, cudaStream_t stream) {
  const Shape &s = shapes_[f];
  const size_t row_bytes = static_cast<size_t>(s.width) * elem_bytes_;
  if (row_bytes * s.height >= kLinearUpload && linear_copy()) {
    check(cudaMemcpyAsync(linear_, host, row_bytes * s.height, cudaMemcpyDefault, stream),
          "copying a frame to the device");
    repitch(linear_, s.height, row_bytes, frame_origin(slot, f), pitch_ * elem_bytes_, stream);
    return;
  }
  check(cudaMemcpy2DAsync(frame_origin(slot, f), pitch_ * elem_bytes_, host, row_bytes,
                          row_bytes, s.height, cudaMemcpyDefault, stream),
        "copying a frame to the device");
}

void ThresholdPlan::upload_device(int slot, int f, const void *device, size_t pitch_bytes,
                                  cudaStream_t stream) {
  const Shape &s = shapes_[f];
  const size_t row_bytes = static_cast<size_t>(s.width) * elem_bytes_;
  check(cudaMemcpy2DAsync(frame_origin(slot, f), pitch_ * elem_bytes_, device, pitch_bytes,
                          row_bytes, s.height, cudaMemcpyDeviceToDevice, stream),
        "copying a frame into the arena");
}

void ThresholdPlan::enqueue(int slot, cudaStream_t stream, cudaEvent_t mid, HostHead *head) {
  Slot &sl = slots_.at(slot);
  check(cudaMemsetAsync(ranges_, 0, cleared_bytes_, stream), "clearing tile counts");
  ThresholdLaunch L;
  L.frames = frames_;
  L.nframes = static_cast<int32_t>(host_frames_.size());
  L.ntasks = ntasks_;
  L.next_task = next_task_;
  L.ranges = share_rows_ ? ranges_ : nullptr;
  L.tile_count = tile_count_;
  L.tile_start = tile_start_;
  L.block_sums = block_sums_;
  L.pool = pool_;
  L.pool_next = pool_next_;
  L.pool_cap = pool_cap_;
  L.status = run_status_;
  L.wait_limit = 1u << 22;
  L.warps_per_block = tuning_.warps_per_block;
  L.lane_cols = lane_cols_;
  L.max_blocks = max_blocks_;
  if (elem_bytes_ == 2)
    check(launch_threshold<uint16_t>(sl.map, L, stream), "launching the threshold");
  else
    check(launch_threshold<uint32_t>(sl.map, L, stream), "launching the threshold");
  if (mid)
    check(cudaEventRecord(mid, stream), "cudaEventRecord");

  PlaceLaunch P;
  P.frames = frames_;
  P.nframes = L.nframes;
  P.sms = sms_;
  P.ntiles = ntiles_;
  P.tile_count = tile_count_;
  P.tile_start = tile_start_;
  P.block_sums = block_sums_;
  P.pool = pool_;
  P.out = sl.out;
  P.frame_count = sl.frame_count;
  P.run_status = run_status_;
  P.status = sl.status;
  P.head = head;
  check(launch_place(P, stream), "launching the placement");
}

} // namespace sf
