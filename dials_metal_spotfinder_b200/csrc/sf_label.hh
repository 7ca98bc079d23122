// The device labeller: 3D (or 2D) six-connected grouping of signal pixels
// across frames, and the per-spot centroid / variance / intensity pass, with
// the reference's streaming semantics (src/dials_spots.cc:36-360): frames
// arrive in ascending order, a component is finished as soon as a frame is
// added that it has no pixel on, finished components come out ordered by
// their last frame and then their first pixel, and the open ones are carried
// on the device to the next batch.
#pragma once

#include <memory>
#include <vector>

#include "sf_host.hh"

namespace sf {

// src/dials_spots.hh:50-54 and :57-79, byte for byte.
struct Pixel {
  int32_t frame;
  uint32_t index;
  uint32_t value;
};
struct Spot {
  int32_t bbox[6];
  double position[3];
  double variance[3];
  double intensity;
  double intensity_variance;
  uint32_t n_signal;
  uint64_t first;
};
static_assert(sizeof(Pixel) == 12, "Pixel layout");
static_assert(sizeof(Spot) == 104, "Spot layout");

struct GroupOptions {
  uint64_t min_spot_size = 3;
  uint64_t max_spot_size = 1000;
  double max_separation = 2.0;
  bool two_d = false;
};

// Device-side scalars (one struct, so the host reads them back in one copy).
struct LabelScalars {
  // this batch
  int64_t batch_z0;       // frame number of the batch's first frame
  uint64_t n;             // live pixels (carried + new)
  uint64_t nw;            // 32-pixel words over n
  uint64_t nseg;          // frame segments (carried last frame + batch frames)
  uint64_t seg_len;       // bucket-count table length: nseg * ceil(closed / 32)
  uint64_t closed;        // finished components
  uint32_t open32;        // pixels carried on
  uint32_t runs_n;        // lab_link's work list
  uint32_t big_n;         // components past the middle spot-pass buffers
  // work counters: warps take the next entries as they finish their last,
  // so a few long union-find chains or large components do not hold a
  // whole grid-stride share
  uint32_t link_next, accept_next, big_next, mid_next;
  uint32_t mid_n;         // components past the small buffers, within the middle ones
  uint32_t close_next, count_next, open_next, pack_next; // tiles taken
  uint64_t members_pack;  // members (low 32) | components passing the size filters (high 32)
  uint64_t accepted_pack; // accepted spots | their pixels << 31
  uint64_t batch_spots, batch_pixels;
  // the carry between batches
  uint64_t carry_n;
  uint64_t carry_last_start; // first carried pixel on the carry's last frame
  int64_t carry_last_z;
  // running totals over the series (src/dials_spots.hh:99-106)
  uint64_t signal_pixels, groups, too_small, too_large, separated, accepted;
  uint64_t kept_total; // pixels of accepted spots so far (Spot::first base)
  int32_t status;      // nonzero: a capacity was exceeded
  int32_t pad1;
  uint64_t zero; // the offset of a batch's only list
};

enum : int32_t {
  kLabelOk = 0,
  kLabelLiveOverflow = 1,
  kLabelSpotOverflow = 2,
  kLabelWaitTimeout = 3, // a tile's wait for the tiles before it gave up
};
// What to tell the caller of `what` ("grouping") that ended with a status.
inline std::string label_error(const char *what, int32_t status) {
  return what + std::string(status == kLabelWaitTimeout ? ": a wait on the device gave up"
                                                        : " capacity exceeded") +
         " (status " + std::to_string(status) + ")";
}

// Page-locked host memory in which a small batch leaves its results, so that
// the host has them with its scalars, without copies of their own (two of them
// and a second wait were 30 us of each frame added). As far as they fit here:
// much more than a frame of a few thousand pixels finishes, and little to lock.
struct LabelHead {
  static constexpr uint64_t kSpots = 128, kPixels = 1536;
  Spot spots[kSpots];
  Pixel pixels[kPixels];
};

// What a component's root holds, in one 16-byte word at its position.
struct RootInfo {
  uint32_t size;
  int32_t lastz;   // its last frame
  uint32_t slot;   // its members' place; all ones while it is open
  uint32_t cursor; // members placed
};

class DeviceLabeller {
public:
  DeviceLabeller(int height, int width, const GroupOptions &options);
  ~DeviceLabeller();
  DeviceLabeller(const DeviceLabeller &) = delete;
  DeviceLabeller &operator=(const DeviceLabeller &) = delete;

  // Buffers for batches of up to `batch_pixels` new signal pixels over up to
  // `max_frames` frames, with up to `carry_pixels` carried between batches.
  // Grows (synchronising the device) only when asked for more; call before
  // any graph capture. With `room`, for a caller that learns the sizes frame
  // by frame, it grows by more than it was asked where that fits: the carry
  // grows by about a frame's pixels with each of the first frames, and
  // reallocating on every one of them was 67 of the 85 ms that four
  // 2162 x 2068 frames took.
  void reserve(uint64_t batch_pixels, int max_frames, uint64_t carry_pixels, bool room = false);

  // Enqueue one batch of `nframes` consecutive frames numbered from the
  // device-side batch_z0, which the batch then advances by nframes. Frame
  // f's list is lists[offs[f] ...] holding up to caps[f] records, with
  // counts[count_map[f]] entries (counts[f] when count_map is null), all in
  // device memory. With close_all every component is finished, as the
  // reference's finish() does; nframes may then be 0.
  void enqueue(int nframes, const SignalPixel *lists, const uint64_t *offs,
               const uint32_t *counts, const int32_t *count_map, const uint32_t *caps,
               bool close_all, cudaStream_t s);

  // The same for one frame, number z, of `count` records at `list`, where the
  // caller knows how many pixels the last batch left (`carried`); nothing but
  // the list is read from device memory.
  void enqueue_frame(int64_t z, const SignalPixel *list, uint32_t count, uint64_t carried,
                     cudaStream_t s);
  // ... and for finishing what is left.
  void enqueue_rest(uint64_t carried, cudaStream_t s);
  // Whether a batch of `nframes` frames with `pixels` pixels, carried and added,
  // takes the launches of one block. Those of the two calls above leave the
  // batch's spots and pixels in the head that head_to() gave, as far as they
  // fit there.
  bool one_block(uint64_t pixels, int nframes) const;

  // Sets batch_z0 for the next enqueue (an asynchronous copy from pinned
  // host memory; the labeller keeps the staging word until the next call).
  void set_next_frame(int64_t z, cudaStream_t s);

  // A batch captured in a CUDA graph was replayed: it swapped the live
  // buffers on the device, so the host's record of which holds the carry
  // swaps too.
  void note_replayed() { cur_ ^= 1; }
  int parity() const { return cur_; }

  LabelScalars *scalars() const { return sc_; }
  // Page-locked host memory that each batch leaves a copy of the scalars in
  // (there once its stream has passed); set before the first one.
  void report_to(LabelScalars *host) { report_ = host; }
  void head_to(LabelHead *host) { head_ = host; }
  Spot *batch_spots() const { return spots_out_; }
  Pixel *batch_pixels() const { return kept_out_; }
  uint64_t spot_capacity() const { return spot_cap_; }
  uint64_t batch_capacity() const { return batch_cap_; }
  int frame_capacity() const { return frame_cap_; }
  int height() const { return height_; }
  int width() const { return width_; }
  const GroupOptions &options() const { return opt_; }

private:
  struct Batch {
    int nframes = 0;
    const SignalPixel *lists = nullptr;
    const uint64_t *offs = nullptr;
    const uint32_t *counts = nullptr;
    const int32_t *count_map = nullptr;
    const uint32_t *caps = nullptr;
    uint32_t one_count = 0; // without counts: of the only frame
    int64_t one_z = 0;      // and its number
    bool close_all = false;
    uint64_t most = 0; // pixels, carried ones too, that it can hold
  };
  void enqueue_batch(const Batch &b, cudaStream_t s);
  void create_streams();
  void release();
  bool allocate(uint64_t batch_pixels, int frames, uint64_t carry_pixels, bool share);

  int height_, width_;
  GroupOptions opt_;

  unsigned char *arena_ = nullptr; // every buffer below but the scalars and the carry's table

  uint64_t batch_cap_ = 0, carry_cap_ = 0, live_cap_ = 0, spot_cap_ = 0;
  uint64_t batch_asked_ = 0, carry_asked_ = 0; // of the capacities: what reserve() was asked for
  int frame_cap_ = 0;
  int cur_ = 0; // which live buffer holds the carry

  struct Live {
    int32_t *frame = nullptr;
    uint32_t *index = nullptr;
    uint32_t *value = nullptr;
    uint32_t *parent = nullptr;
  } live_[2];
  uint32_t *root_ = nullptr;
  RootInfo *info_ = nullptr;
  uint32_t *bits_ = nullptr, *bcnt_ = nullptr; // root bitmap; bucket counts (lab_count)
  uint32_t *flist_ = nullptr;                   // the finished roots in position order
  uint32_t *comp_root_ = nullptr, *msize_ = nullptr, *members_ = nullptr;
  uint64_t *mpk_ = nullptr; // member offset (low 32) | size-filtered index (high 32)
  uint4 *runs_ = nullptr; // lab_link's work list
  uint32_t *run_starts_ = nullptr; // per 32 positions: the run starts (lab_gather)
  Spot *spot_tmp_ = nullptr;  // spots by size-filtered index, before acceptance
  Pixel *pix_tmp_ = nullptr;  // their pixels, by member offset
  uint64_t *pack_ = nullptr;
  uint64_t *close_st_ = nullptr, *count_st_ = nullptr, *open_st_ = nullptr,
           *pack_st_ = nullptr; // lookback words
  uint32_t *obits_ = nullptr, *ocnt_ = nullptr; // open pixels per 32 positions
  uint32_t *big_ = nullptr; // ranks of the components lab_accept's large launch takes
  uint32_t *mid_ = nullptr; // ... and its middle launch
  Spot *spots_out_ = nullptr;
  Pixel *kept_out_ = nullptr;
  uint64_t *seg_start_ = nullptr; // per batch segment: start, count (device)
  uint64_t *seg_count_ = nullptr;
  int64_t *seg_z_ = nullptr;
  uint32_t *tab_ = nullptr;       // block tables of the batch frames
  uint32_t *carry_tab_ = nullptr; // block table of the carry's last frame
  uint64_t nblk_ = 0;
  unsigned grid_ = 0;
  LabelScalars *sc_ = nullptr;
  LabelScalars *report_ = nullptr;
  LabelHead *head_ = nullptr;
  cudaStream_t aux_ = nullptr;  // the large components' spot pass
  cudaStream_t aux2_ = nullptr; // the middle-sized components' spot pass
  cudaEvent_t fork_ = nullptr, join_ = nullptr, join2_ = nullptr;
  int64_t *z_stage_ = nullptr; // pinned
};

} // namespace sf
