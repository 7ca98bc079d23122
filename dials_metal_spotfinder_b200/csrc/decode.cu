// The device side of the chunk codec: LZ4 blocks decoded one warp per block
// in shared memory, bitshuffle blocks un-transposed there, and the elements
// written straight into the destination frame at its row pitch (an engine
// arena). Raw frames take one contiguous copy and a re-pitching kernel. See
// codec.cu for the formats.

#include <algorithm>
#include <stdexcept>

#include "sf_capi.hh"
#include "sf_codec.hh"
#include "sf_host.hh"

namespace sf {
namespace {

constexpr int kDecodeWarps = 2; // per block of threads; the warps are independent
constexpr unsigned kFull = 0xffffffffu;
// Compressed bytes a warp stages in shared memory: every block of up to
// 8 KB that any coder made shorter. A longer one (nearly incompressible, so
// few sequences) is parsed from global memory instead.
constexpr uint32_t kStageCap = 8192;
constexpr uint16_t kSeqEnd = 0xffff, kSeqBad = 0xfffe;
// Sequences a lane parses at a time, and a warp's records at a time.
constexpr uint32_t kLaneSeqs = 4;
constexpr uint32_t kGroupSeqs = 32 * kLaneSeqs;
// 32-byte pieces of the output whose references a warp looks up at a time.
constexpr uint32_t kSegments = 4;

// What a warp owns of the shared memory. `next` (two bytes per compressed
// byte) lies over the output, which is written only once it is dead, and
// `extra` is what it needs beyond that; everything after the output is dead
// once the block is decoded and then holds `bounce` (see store_planes).
struct WarpLayout {
  uint32_t out, extra, stage, list, ends, starts, total;
};
__host__ __device__ constexpr uint32_t up16(uint32_t x) { return (x + 15) & ~15u; }
__host__ __device__ constexpr WarpLayout warp_layout(uint32_t out_bytes, uint32_t stage_bytes,
                                                     uint32_t elem) {
  WarpLayout w{};
  w.out = out_bytes;
  w.extra = up16(2 * stage_bytes) > out_bytes ? up16(2 * stage_bytes) - out_bytes : 0;
  w.stage = stage_bytes;
  // every fourth sequence start; a sequence spans at least three bytes
  w.list = up16((stage_bytes / (3 * kLaneSeqs) + 3) * 2);
  // a bit per compressed byte, and two words past the last
  w.ends = up16((stage_bytes / 32 + 3) * 4);
  // a bit per output byte, and a step's words past the last
  w.starts = up16((out_bytes / 32 + 1 + kSegments) * 4);
  const uint32_t rest =
      w.extra + w.stage + w.list + w.ends + w.starts + kGroupSeqs * static_cast<uint32_t>(sizeof(uint2));
  const uint32_t bounce = 1024 * elem;
  w.total = w.out + (rest > bounce ? rest : bounce);
  return w;
}

struct BlockDesc {
  uint64_t in;  // the LZ4 data, in the chunk
  uint64_t out; // its output, in the frame's bytes
  uint32_t len; // compressed length
  uint32_t n;   // decoded length
};

// A frame in device memory: rows of row_bytes at `pitch` bytes apart.
struct FrameDst {
  uint8_t *base;
  uint64_t pitch;
  uint64_t row_bytes;
  uint32_t word; // 4, 2 or 1: divides the base, the pitch, the rows and every block's offset
};

size_t round16(size_t x) { return (x + 15) & ~static_cast<size_t>(15); }

// One warp decodes one LZ4 block of `cs` bytes at `src` (shared or global
// memory) into `dst` (shared memory, n bytes). Lane 0 parses each sequence;
// the warp copies its literals and its match in parallel (a match of offset
// d repeats with period d, so byte i of it is byte i mod d of the d bytes
// before it: each lane steps its phase by 32 mod d, no division in the
// loop). Every length and offset is checked against both buffers before
// anything is written; returns false on a malformed block.
__device__ bool warp_lz4(const uint8_t *src, uint32_t cs, uint8_t *dst, uint32_t n, int lane) {
  uint32_t ip = 0, op = 0;
  while (true) {
    // c: offset | flag << 16 (0 a full sequence, 1 the last, 2 malformed);
    // a: literal count; b: literal start; m: match length
    uint32_t a = 0, b = 0, c = 0, m = 0;
    if (lane == 0) {
      int flag = 0;
      uint32_t lit = 0, off = 0, ml = 0;
      if (ip >= cs) {
        flag = 2;
      } else {
        const uint32_t token = src[ip++];
        uint64_t l = token >> 4;
        if (l == 15) {
          uint32_t v;
          do {
            if (ip >= cs) {
              flag = 2;
              break;
            }
            v = src[ip++];
            l += v;
          } while (v == 255);
        }
        if (!flag && (l > cs - ip || l > n - op))
          flag = 2;
        if (!flag) {
          lit = static_cast<uint32_t>(l);
          b = ip;
          ip += lit;
          if (ip == cs) {
            flag = 1;
          } else if (cs - ip < 2) {
            flag = 2;
          } else {
            off = src[ip] | (static_cast<uint32_t>(src[ip + 1]) << 8);
            ip += 2;
            uint64_t mm = (token & 15) + 4;
            if ((token & 15) == 15) {
              uint32_t v;
              do {
                if (ip >= cs) {
                  flag = 2;
                  break;
                }
                v = src[ip++];
                mm += v;
              } while (v == 255);
            }
            if (!flag && (off == 0 || off > op + lit || mm > n - op - lit))
              flag = 2;
            ml = static_cast<uint32_t>(mm);
          }
        }
      }
      a = lit;
      c = off | (static_cast<uint32_t>(flag) << 16);
      m = ml;
    }
    c = __shfl_sync(kFull, c, 0);
    const uint32_t flag = c >> 16, off = c & 0xffffu;
    if (flag == 2)
      return false;
    const uint32_t lit = __shfl_sync(kFull, a, 0);
    b = __shfl_sync(kFull, b, 0);
    for (uint32_t i = lane; i < lit; i += 32)
      dst[op + i] = src[b + i];
    op += lit;
    if (flag == 1)
      break;
    const uint32_t ml = __shfl_sync(kFull, m, 0);
    __syncwarp();
    if (off >= ml) {
      for (uint32_t i = lane; i < ml; i += 32)
        dst[op + i] = dst[op - off + i];
    } else {
      uint32_t q = lane % off;
      const uint32_t step = 32 % off;
      for (uint32_t i = lane; i < ml; i += 32) {
        dst[op + i] = dst[op - off + q];
        q += step;
        if (q >= off)
          q -= off;
      }
    }
    op += ml;
    __syncwarp();
  }
  __syncwarp();
  return op == n;
}

// A length continued past its four bits at byte q of the L compressed bytes:
// adds the run of 255s and the byte that ends it, and moves q past them.
// `ends` has a bit per byte that is not 255, set from L on; false where the
// length runs past the end. (Byte by byte, the warp would wait for its
// longest run at every step.)
__device__ __forceinline__ bool add_length(const uint8_t *in, uint32_t L, const uint32_t *ends,
                                           uint32_t *q, uint32_t *length) {
  if (*q >= L)
    return false;
  uint32_t word = *q >> 5;
  uint32_t w = ends[word] & (0xffffffffu << (*q & 31));
  while (w == 0) // ends with the word after the last byte's
    w = ends[++word];
  const uint32_t r = 32 * word + __ffs(w) - 1;
  if (r >= L)
    return false;
  *length += 255 * (r - *q) + in[r];
  *q = r + 1;
  return true;
}

// The LZ4 sequence at byte p < L, every read bounds-checked: its literals
// (count, start), its match (offset, length; 0 of the last sequence), and
// the byte after it -- L where no last sequence follows, kSeqEnd where its
// literals end the block, kSeqBad where it runs past the end.
struct Seq {
  uint32_t lit, start, off, len;
};
__device__ __forceinline__ uint32_t parse_seq(const uint8_t *in, uint32_t L,
                                              const uint32_t *ends, uint32_t p, Seq *s) {
  const uint32_t t = in[p];
  uint32_t q = p + 1;
  bool ok = true;
  *s = Seq{t >> 4, 0, 0, 0};
  if (s->lit == 15)
    ok = add_length(in, L, ends, &q, &s->lit);
  ok = ok && s->lit <= L - q;
  s->start = q;
  q += s->lit;
  const bool last = ok && q == L;
  ok = ok && (last || L - q >= 2);
  if (ok && !last) {
    s->off = in[q] | (static_cast<uint32_t>(in[q + 1]) << 8);
    s->len = (t & 15) + 4;
    q += 2;
    if (s->len == 19)
      ok = add_length(in, L, ends, &q, &s->len);
  }
  return !ok ? kSeqBad : last ? kSeqEnd : q;
}

// The same decode spread over the warp, for a block whose L compressed bytes
// sit in shared memory, `in_at` bytes after the output `dst`:
//  1. every lane parses a sequence at each of its byte positions p as if a
//     token started there: next[p] is where the next one would start;
//  2. two doublings in place (next[p] > p, and a warp's reads go before its
//     writes, so entries above p still hold the single step) make next[p]
//     the start four sequences on;
//  3. lane 0 follows next[] from byte 0, listing every fourth real start;
//  4. 128 sequences at a time, four a lane: parse, a warp scan of the output
//     lengths, the bounds checks, a record per sequence and a bit per output
//     byte that starts one;
//  5. the group's output, 32 bytes (one a lane) at a time. A byte's sequence
//     is its rank among the start bits; it is a literal, or the byte `off`
//     back: an earlier byte of the output, or of the same 32, in which case
//     the lanes follow each other's references, doubling (five rounds at
//     most), to the one that holds the value. All that but the reads of the
//     output itself is done for kSegments pieces together. A stretch inside
//     one match is copied at once, in 16-byte words when it repeats a short
//     period.
// Step 5 costs the same for 32 output bytes whatever the number of
// sequences in them; copying match by match, each by the whole warp, cost
// 45 instructions and a chain of shared-memory reads a sequence. The decode
// of one frame alone: 2162 x 2068 uint16 in plain LZ4 blocks (1200 sequences
// of 7 bytes a block) 575 -> 95 us, uint32 223 -> 155; uint16 in bslz4
// blocks (250 sequences, most of the output in a few) 77 -> 57; 4362 x 4148
// bslz4, whose 4418 blocks keep the SMs issuing either way, 135 -> 135.
// Bound: the latency of step 5's chain of shared-memory reads where a chunk
// has few blocks, instruction issue where it has many.
// Returns false on a malformed block, having written nothing past n.
__device__ bool warp_lz4_parallel(uint8_t *dst, uint32_t in_at, uint32_t L, uint16_t *next,
                                  uint16_t *list, uint32_t *ends, uint2 *rec, uint32_t *starts,
                                  uint32_t n, int lane) {
  const uint8_t *in = dst + in_at;
  for (uint32_t base = 0; base < L + 32; base += 32) {
    const uint32_t m = __ballot_sync(kFull, base + lane >= L || in[base + lane] != 255);
    if (lane == 0)
      ends[base >> 5] = m;
  }
  __syncwarp();
  for (uint32_t p = lane; p < L; p += 32) {
    Seq s;
    next[p] = static_cast<uint16_t>(parse_seq(in, L, ends, p, &s));
  }
  for (uint32_t k = lane; k < n / 32 + 1 + kSegments; k += 32)
    starts[k] = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 2; r++) {
    for (uint32_t base = 0; base < L; base += 128) {
      uint32_t a[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t p = base + 32 * u + lane;
        a[u] = p < L ? next[p] : kSeqBad;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (a[u] < L)
          a[u] = next[a[u]];
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t p = base + 32 * u + lane;
        if (p < L)
          next[p] = static_cast<uint16_t>(a[u]);
      }
    }
    __syncwarp();
  }
  uint32_t quads = 0;
  if (lane == 0) {
    uint32_t p = 0;
    while (p < L) { // neither mark is below L, and p rises
      list[quads++] = static_cast<uint16_t>(p);
      p = next[p];
    }
    if (p != kSeqEnd)
      quads = 0;
  }
  quads = __shfl_sync(kFull, quads, 0);
  if (quads == 0)
    return false;
  __syncwarp();

  const uint32_t le = 0xffffffffu >> (31 - lane);
  uint32_t obase = 0;
  for (uint32_t qb = 0; qb < quads; qb += 32) {
    Seq s[kLaneSeqs];
    uint32_t have = 0, total = 0;
    bool last = false;
    uint32_t p = qb + lane < quads ? list[qb + lane] : L;
#pragma unroll
    for (uint32_t k = 0; k < kLaneSeqs; k++) {
      s[k] = Seq{0, 0, 0, 0};
      if (p < L) { // step 3 saw the sequence end in the block
        p = parse_seq(in, L, ends, p, &s[k]);
        total += s[k].lit + s[k].len;
        have++;
        last = p >= L;
      }
      __syncwarp();
    }
    uint32_t incl = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, d);
      if (lane >= d)
        incl += y;
    }
    // lengths of up to 255 L a lane: the sums stay below 2^32
    uint32_t op = obase + incl - total;
    bool ok = op + total <= n;
#pragma unroll
    for (uint32_t k = 0; k < kLaneSeqs; k++)
      if (k < have) {
        const uint32_t m = op + s[k].lit;
        if (!(last && k + 1 == have))
          ok = ok && s[k].off != 0 && s[k].off <= m;
        rec[kLaneSeqs * lane + k] = make_uint2((op & 0xffffu) | (m << 16),
                                               ((s[k].start - op) & 0xffffu) | (s[k].off << 16));
        if (ok && s[k].lit + s[k].len)
          atomicOr(&starts[op >> 5], 1u << (op & 31));
        op = m + s[k].len;
      }
    if (__any_sync(kFull, !ok))
      return false;
    const uint32_t nseq = __reduce_add_sync(kFull, have);
    const uint32_t end = obase + __shfl_sync(kFull, incl, 31); // of the group's output
    __syncwarp();

    uint32_t lo = obase; // bytes below are written
    uint32_t before = 0; // sequences of the group that start before this segment
    uint32_t S = lo & ~31u;
    while (S < end) {
      uint32_t w[kSegments];
#pragma unroll
      for (uint32_t u = 0; u < kSegments; u++)
        w[u] = starts[(S >> 5) + u]; // none at or past `end`
      if (S < lo)
        w[0] &= 0xffffffffu << (lo - S);
      if (w[0] == 0 && S >= lo) {
        // inside one sequence: a long enough stretch of its match?
        const uint2 r = rec[before - 1];
        const uint32_t stop = before < nseq ? rec[before].x & 0xffffu : end;
        const uint32_t m = r.x >> 16, d = r.y >> 16, len = stop - S;
        if (S >= m && len >= 64) {
          bool copied = true;
          if (d <= 16 && (d & (d - 1)) == 0) {
            // period 1, 2, 4, 8 or 16: every 16-byte word from S is the same
            uint32_t q[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
              q[k] = 0;
#pragma unroll
              for (uint32_t t = 0; t < 4; t++)
                q[k] |= static_cast<uint32_t>(dst[S - d + ((4 * k + t) & (d - 1))]) << (8 * t);
            }
            const uint32_t nv = len / 16;
            uint4 *v = reinterpret_cast<uint4 *>(dst + S);
            for (uint32_t i = lane; i < nv; i += 32)
              v[i] = make_uint4(q[0], q[1], q[2], q[3]);
            if (static_cast<uint32_t>(lane) < (len & 15u))
              dst[S + 16 * nv + lane] = dst[S - d + (lane & (d - 1))];
            __syncwarp();
          } else {
            // a whole number of periods back is as good as one, and the more
            // is written the further back it can be: as many whole rows of 32
            // as lie between, up to four at once
            uint32_t D = d;
            for (uint32_t c = S; copied && c < stop;) {
              while (2 * D <= c - (m - d) && D < 128)
                D *= 2;
              const uint32_t rows = min(D / 32, 4u);
              copied = rows > 0; // else: too little written yet
              uint32_t v[4];
#pragma unroll
              for (uint32_t u = 0; u < 4; u++)
                if (u < rows && c + 32 * u + lane < stop)
                  v[u] = dst[c + 32 * u + lane - D];
#pragma unroll
              for (uint32_t u = 0; u < 4; u++)
                if (u < rows && c + 32 * u + lane < stop)
                  dst[c + 32 * u + lane] = static_cast<uint8_t>(v[u]);
              __syncwarp();
              c += 32 * rows;
            }
          }
          if (copied) {
            lo = stop;
            S = lo & ~31u;
            continue;
          }
        }
      }
      // at: where the byte's value is read, for the lanes that read one;
      // from: the lane of the piece that does
      uint32_t at[kSegments], from[kSegments];
      bool within[kSegments], inside = false;
#pragma unroll
      for (uint32_t u = 0; u < kSegments; u++) {
        const uint32_t P = S + 32 * u, i = P + lane;
        const uint32_t rank = before + __popc(w[u] & le);
        before += __popc(w[u]);
        const uint2 r = rec[rank ? rank - 1 : 0u];
        const bool active = i >= lo && i < end;
        const bool literal = i < (r.x >> 16);
        const uint32_t back = i - (r.y >> 16); // off <= i
        within[u] = active && !literal && back >= P;
        inside = inside || within[u];
        from[u] = within[u] ? back - P : static_cast<uint32_t>(lane);
        // a byte below lo is already there; one at or past the end is unused
        at[u] = i < lo ? i : 0u;
        if (active && !within[u])
          at[u] = literal ? in_at + i + static_cast<uint32_t>(static_cast<int16_t>(r.y & 0xffffu))
                          : back;
      }
      while (__any_sync(kFull, inside)) {
        inside = false;
#pragma unroll
        for (uint32_t u = 0; u < kSegments; u++) {
          const uint32_t q = __shfl_sync(kFull, from[u], static_cast<int>(from[u]));
          inside = inside || q != from[u];
          from[u] = q;
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < kSegments; u++) {
        const uint32_t i = S + 32 * u + lane;
        const uint32_t v = __shfl_sync(kFull, static_cast<uint32_t>(dst[at[u]]),
                                       static_cast<int>(from[u]));
        if (i >= lo && i < end)
          dst[i] = static_cast<uint8_t>(v);
        __syncwarp();
      }
      S += 32 * kSegments;
    }
    obase = end;
  }
  return obase == n;
}

// The row holding byte `col` counted from the start of `row`; `col` becomes
// the byte's place in it.
__device__ __forceinline__ uint8_t *frame_row(const FrameDst &D, uint8_t *row, uint64_t &col) {
  const uint64_t down = ((col | D.row_bytes) >> 32)
                            ? col / D.row_bytes
                            : static_cast<uint32_t>(col) / static_cast<uint32_t>(D.row_bytes);
  col -= down * D.row_bytes;
  return row + down * D.pitch;
}

// Where linear byte `o` of the frame lives.
__device__ __forceinline__ uint8_t *frame_at(const FrameDst &D, uint64_t o, uint64_t &col) {
  col = o;
  return frame_row(D, D.base, col);
}

// Writes `nb` (<= 32) bytes held in w[0..7] to frame bytes [o, o + nb): the
// widest stores the destination's alignment allows when they sit in one row,
// byte by byte across a row end.
__device__ __forceinline__ void put(const FrameDst &D, uint64_t o, uint32_t nb,
                                   const uint32_t (&w)[8]) {
  uint64_t col;
  uint8_t *row = frame_at(D, o, col);
  uint8_t *p = row + col;
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  if (col + nb <= D.row_bytes) {
    if ((nb & 15) == 0 && (at & 15) == 0) {
#pragma unroll
      for (int k = 0; k < 2; k++)
        if (16u * k < nb)
          reinterpret_cast<uint4 *>(p)[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2],
                                                       w[4 * k + 3]);
      return;
    }
    if ((nb & 7) == 0 && (at & 7) == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (8u * k < nb)
          reinterpret_cast<uint2 *>(p)[k] = make_uint2(w[2 * k], w[2 * k + 1]);
      return;
    }
    if ((nb & 3) == 0 && (at & 3) == 0) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (4u * k < nb)
          reinterpret_cast<uint32_t *>(p)[k] = w[k];
      return;
    }
  }
#pragma unroll
  for (uint32_t q = 0; q < 32; q++) {
    if (q < nb) {
      if (col == D.row_bytes) {
        row += D.pitch;
        col = 0;
      }
      row[col++] = static_cast<uint8_t>(w[q >> 2] >> (8 * (q & 3)));
    }
  }
}

// transpose8x8 on a word's two halves: its first two steps stay within each.
__device__ __forceinline__ void transpose_halves(uint32_t &lo, uint32_t &hi) {
  uint32_t t = (lo ^ (lo >> 7)) & 0x00AA00AAu;
  lo ^= t ^ (t << 7);
  t = (hi ^ (hi >> 7)) & 0x00AA00AAu;
  hi ^= t ^ (t << 7);
  t = (lo ^ (lo >> 14)) & 0x0000CCCCu;
  lo ^= t ^ (t << 14);
  t = (hi ^ (hi >> 14)) & 0x0000CCCCu;
  hi ^= t ^ (t << 14);
  t = (lo ^ (hi << 4)) & 0xF0F0F0F0u;
  lo ^= t;
  hi ^= t >> 4;
}

// Eight elements of E bytes from their bytes: byte i of lo[j], hi[j] (i < 4,
// i >= 4) is byte j of element i.
template <int E>
__device__ __forceinline__ void weave(const uint32_t (&lo)[E], const uint32_t (&hi)[E],
                                      uint32_t *w) {
  if constexpr (E == 1) {
    w[0] = lo[0];
    w[1] = hi[0];
  } else if constexpr (E == 2) {
    w[0] = __byte_perm(lo[0], lo[1], 0x5140);
    w[1] = __byte_perm(lo[0], lo[1], 0x7362);
    w[2] = __byte_perm(hi[0], hi[1], 0x5140);
    w[3] = __byte_perm(hi[0], hi[1], 0x7362);
  } else {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t a0 = h ? hi[0] : lo[0], a1 = h ? hi[1] : lo[1];
      const uint32_t a2 = h ? hi[2] : lo[2], a3 = h ? hi[3] : lo[3];
      const uint32_t p = __byte_perm(a0, a1, 0x5140), q = __byte_perm(a2, a3, 0x5140);
      const uint32_t r = __byte_perm(a0, a1, 0x7362), t = __byte_perm(a2, a3, 0x7362);
      w[4 * h + 0] = __byte_perm(p, q, 0x5410);
      w[4 * h + 1] = __byte_perm(p, q, 0x7632);
      w[4 * h + 2] = __byte_perm(r, t, 0x5410);
      w[4 * h + 3] = __byte_perm(r, t, 0x7632);
    }
  }
}

// Eight elements of E bytes, group g of a bit-transposed block of `plane`
// bytes per bit plane, back in element order: element i's byte j is byte i
// of the 8 x 8 transpose of bytes (8j + k) * plane + g, k = 0..7.
template <int E>
__device__ __forceinline__ void untranspose(const uint8_t *buf, uint32_t plane, uint32_t g,
                                            uint32_t (&w)[8]) {
  uint32_t lo[E], hi[E];
#pragma unroll
  for (int j = 0; j < E; j++) {
    uint64_t x = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
      x |= static_cast<uint64_t>(buf[(8 * j + k) * plane + g]) << (8 * k);
    lo[j] = static_cast<uint32_t>(x);
    hi[j] = static_cast<uint32_t>(x >> 32);
    transpose_halves(lo[j], hi[j]);
  }
  weave<E>(lo, hi, w);
}

// The 16-byte unit of the bounce buffer that holds unit u: spread so that
// lanes writing four units each, or reading consecutive words, meet in no
// bank.
__device__ __forceinline__ uint32_t spread(uint32_t u) { return u ^ ((u >> 3) & 7u); }

// `bytes` bytes at `src` (shared memory) to frame bytes [o, o + bytes), a
// word of D.word bytes a lane, so that the warp's stores are consecutive.
template <bool SPREAD, typename V>
__device__ __forceinline__ void put_words(const FrameDst &D, uint64_t o, const uint8_t *src,
                                          uint32_t bytes, int lane) {
  constexpr uint32_t kRow = 32 * sizeof(V); // bytes the warp writes at a time
  uint64_t col0;
  uint8_t *row = frame_at(D, o, col0);
  auto word = [&](uint32_t b) {
    return *reinterpret_cast<const V *>(src + (SPREAD ? spread(b >> 4) * 16 + (b & 15u) : b));
  };
  if (D.row_bytes < kRow) {
    for (uint32_t b = lane * sizeof(V); b < bytes; b += kRow) {
      uint64_t col = col0 + b;
      uint8_t *to = frame_row(D, row, col);
      *reinterpret_cast<V *>(to + col) = word(b);
    }
    return;
  }
  // the lane's word crosses at most one row's end from each of its words to
  // the next
  const uint64_t skip = D.pitch - D.row_bytes;
  uint64_t col = col0 + lane * sizeof(V);
  uint8_t *to = row + col;
  constexpr int kU = 4; // words in flight
  for (uint32_t b0 = lane * sizeof(V); b0 < bytes; b0 += kU * kRow) {
    V v[kU];
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (b0 + u * kRow < bytes)
        v[u] = word(b0 + u * kRow);
#pragma unroll
    for (int u = 0; u < kU; u++) {
      if (col >= D.row_bytes) {
        col -= D.row_bytes;
        to += skip;
      }
      if (b0 + u * kRow < bytes)
        *reinterpret_cast<V *>(to) = v[u];
      col += kRow;
      to += kRow;
    }
  }
}
template <bool SPREAD>
__device__ __forceinline__ void put_all(const FrameDst &D, uint64_t o, const uint8_t *src,
                                        uint32_t bytes, int lane) {
  if (D.word == 4)
    put_words<SPREAD, uint32_t>(D, o, src, bytes, lane);
  else if (D.word == 2)
    put_words<SPREAD, uint16_t>(D, o, src, bytes, lane);
  else
    put_words<SPREAD, uint8_t>(D, o, src, bytes, lane);
}

// A decoded bitshuffle block of n bytes at `buf`, back in element order, to
// the frame: a lane takes a 32-bit word of every bit plane, which holds four
// groups of eight elements, separates the groups by byte transposes, undoes
// their bit transposes, and leaves their bytes in `bounce`, from which the
// warp writes rows of consecutive words. (A lane storing its own 16 bytes
// in the four-byte words the arena's alignment allows touched every sector
// four times.)
template <int E>
__device__ __forceinline__ void store_planes(const uint8_t *buf, uint32_t n, uint8_t *bounce,
                                             const FrameDst &D, uint64_t o, int lane) {
  const uint32_t plane = n / (8 * E);
  if constexpr (E == 2 || E == 4) {
    if ((plane & 3u) == 0) {
      const uint32_t words = plane / 4;
      for (uint32_t base = 0; base < words; base += 32) {
        const uint32_t wd = base + lane;
        if (wd < words) {
          uint32_t y[4][2 * E];
#pragma unroll
          for (int j = 0; j < 2 * E; j++) {
            uint32_t x[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
              x[k] = *reinterpret_cast<const uint32_t *>(buf + (4 * j + k) * plane + 4 * wd);
            const uint32_t t0 = __byte_perm(x[0], x[1], 0x5140);
            const uint32_t t1 = __byte_perm(x[2], x[3], 0x5140);
            const uint32_t t2 = __byte_perm(x[0], x[1], 0x7362);
            const uint32_t t3 = __byte_perm(x[2], x[3], 0x7362);
            y[0][j] = __byte_perm(t0, t1, 0x5410);
            y[1][j] = __byte_perm(t0, t1, 0x7632);
            y[2][j] = __byte_perm(t2, t3, 0x5410);
            y[3][j] = __byte_perm(t2, t3, 0x7632);
          }
#pragma unroll
          for (int g = 0; g < 4; g++) {
            uint32_t lo[E], hi[E], w[2 * E];
#pragma unroll
            for (int j = 0; j < E; j++) {
              lo[j] = y[g][2 * j];
              hi[j] = y[g][2 * j + 1];
              transpose_halves(lo[j], hi[j]);
            }
            weave<E>(lo, hi, w);
#pragma unroll
            for (int h = 0; h < E / 2; h++)
              reinterpret_cast<uint4 *>(bounce)[spread((4 * lane + g) * (E / 2) + h)] =
                  make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
          }
        }
        __syncwarp();
        put_all<true>(D, o + 32ull * E * base, bounce, min(32u, words - base) * 32 * E, lane);
        __syncwarp();
      }
      return;
    }
  }
  for (uint32_t g = lane; g < plane; g += 32) {
    uint32_t w[8];
    untranspose<E>(buf, plane, g, w);
    put(D, o + 8ull * E * g, 8 * E, w);
  }
}

// Blocks of a chunk, one warp each, grid-strided. Each warp owns a piece of
// the shared memory (warp_layout) for the decoded block, its compressed
// bytes and the decode's tables. E > 0: bitshuffle blocks of E-byte
// elements, un-transposed on the way out; E == 0: plain LZ4. Warp 0 of block
// 0 also copies the chunk's raw tail (elements after the last block).
template <int E>
__global__ void __launch_bounds__(kDecodeWarps * 32, 1)
    decode_blocks(const uint8_t *__restrict__ chunk, const BlockDesc *__restrict__ blocks,
                  uint32_t nblocks, uint32_t out_bytes, uint32_t stage_bytes, FrameDst D,
                  uint64_t raw_in, uint32_t raw_bytes, uint64_t raw_out, int *err) {
  extern __shared__ __align__(16) uint8_t decode_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const WarpLayout W = warp_layout(out_bytes, stage_bytes, E);
  uint8_t *obuf = decode_smem + static_cast<size_t>(warp) * W.total;
  uint8_t *ibuf = obuf + W.out + W.extra;
  uint16_t *list = reinterpret_cast<uint16_t *>(ibuf + W.stage);
  uint32_t *ends = reinterpret_cast<uint32_t *>(ibuf + W.stage + W.list);
  uint2 *rec = reinterpret_cast<uint2 *>(ibuf + W.stage + W.list + W.ends);
  uint32_t *starts = reinterpret_cast<uint32_t *>(rec + kGroupSeqs);
  if (blockIdx.x == 0 && warp == 0) {
    for (uint32_t i = lane; i < raw_bytes; i += 32) {
      uint64_t col;
      uint8_t *row = frame_at(D, raw_out + i, col);
      row[col] = chunk[raw_in + i];
    }
  }
  const uint32_t nwarps = gridDim.x * kDecodeWarps;
  for (uint32_t b = blockIdx.x * kDecodeWarps + warp; b < nblocks; b += nwarps) {
    const BlockDesc d = blocks[b];
    const uint32_t skew = static_cast<uint32_t>(d.in & 15);
    bool ok;
    if (skew + d.len <= stage_bytes) {
      const uint4 *g = reinterpret_cast<const uint4 *>(chunk + (d.in - skew));
      uint4 *sm = reinterpret_cast<uint4 *>(ibuf);
      const uint32_t nvec = (skew + d.len + 15) / 16;
      for (uint32_t i = lane; i < nvec; i += 32)
        sm[i] = __ldg(g + i);
      __syncwarp();
      ok = warp_lz4_parallel(obuf, W.out + W.extra + skew, d.len,
                             reinterpret_cast<uint16_t *>(obuf), list, ends, rec, starts, d.n,
                             lane);
    } else {
      ok = warp_lz4(chunk + d.in, d.len, obuf, d.n, lane);
    }
    __syncwarp();
    if (!ok) {
      if (lane == 0)
        atomicExch(err, 1);
      __syncwarp();
      continue;
    }
    if constexpr (E > 0)
      store_planes<E>(obuf, d.n, obuf + W.out, D, d.out, lane);
    else
      put_all<false>(D, d.out, obuf, d.n, lane);
    __syncwarp();
  }
}

// Plain LZ4 blocks too large for shared memory, one warp each, decoded in
// place into the frame's linear bytes at `out` (then re-pitched).
__global__ void __launch_bounds__(kDecodeWarps * 32, 1)
    decode_linear(const uint8_t *__restrict__ chunk, const BlockDesc *__restrict__ blocks,
                  uint32_t nblocks, uint8_t *out, int *err) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nwarps = gridDim.x * kDecodeWarps;
  for (uint32_t b = blockIdx.x * kDecodeWarps + warp; b < nblocks; b += nwarps) {
    const BlockDesc d = blocks[b];
    if (!warp_lz4(chunk + d.in, d.len, out + d.out, d.n, lane) && lane == 0)
      atomicExch(err, 1);
    __syncwarp();
  }
}

// Rows of row_bytes, contiguous at `src`, to `dst` at `pitch`; one warp a
// row, V-byte words (V divides row_bytes and pitch, and both bases are
// V-aligned).
template <typename V>
__global__ void __launch_bounds__(256)
    repitch_rows(const V *__restrict__ src, uint64_t row_words, uint8_t *dst, uint64_t pitch,
                 uint64_t rows) {
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * 8;
  const int lane = threadIdx.x & 31;
  for (uint64_t r = blockIdx.x * 8ull + (threadIdx.x >> 5); r < rows; r += warps) {
    const V *s = src + r * row_words;
    V *d = reinterpret_cast<V *>(dst + r * pitch);
    for (uint64_t i = lane; i < row_words; i += 32)
      d[i] = __ldg(s + i);
  }
}

template <typename T> void grow(T **p, size_t &cap, size_t bytes, const char *what) {
  if (bytes <= cap)
    return;
  cudaFree(*p);
  *p = nullptr;
  cap = 0;
  check(cudaMalloc(reinterpret_cast<void **>(p), bytes), what);
  cap = bytes;
}

template <int E> void configure_decoder() {
  check(cudaFuncSetAttribute(decode_blocks<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kDecodeWarps *
                                              warp_layout(static_cast<uint32_t>(kMaxBlockBytes),
                                                          kStageCap + 16, E)
                                                  .total)),
        "cudaFuncSetAttribute");
}

} // namespace

void repitch(const uint8_t *src, size_t height, size_t row_bytes, void *dst, size_t pitch,
             cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>(
      std::min<size_t>((height + 7) / 8, static_cast<size_t>(device_sm_count()) * 8));
  uint8_t *d = static_cast<uint8_t *>(dst);
  const uintptr_t at = reinterpret_cast<uintptr_t>(dst);
  auto fits = [&](size_t v) { return row_bytes % v == 0 && pitch % v == 0 && at % v == 0; };
  if (fits(16))
    repitch_rows<uint4><<<grid, 256, 0, s>>>(reinterpret_cast<const uint4 *>(src),
                                             row_bytes / 16, d, pitch, height);
  else if (fits(8))
    repitch_rows<uint2><<<grid, 256, 0, s>>>(reinterpret_cast<const uint2 *>(src),
                                             row_bytes / 8, d, pitch, height);
  else if (fits(4))
    repitch_rows<uint32_t><<<grid, 256, 0, s>>>(reinterpret_cast<const uint32_t *>(src),
                                                row_bytes / 4, d, pitch, height);
  else if (fits(2))
    repitch_rows<uint16_t><<<grid, 256, 0, s>>>(reinterpret_cast<const uint16_t *>(src),
                                                row_bytes / 2, d, pitch, height);
  else
    repitch_rows<uint8_t><<<grid, 256, 0, s>>>(src, row_bytes, d, pitch, height);
  check(cudaGetLastError(), "launching the frame copy");
}

DeviceChunkDecoder::~DeviceChunkDecoder() {
  // the owner has drained the stream the decodes ran on; cudaFree waits
  // for the rest
  if (h2d_)
    cudaStreamSynchronize(h2d_);
  for (Set &S : sets_) {
    cudaFree(S.d_in);
    if (S.copied)
      cudaEventDestroy(S.copied);
    if (S.freed)
      cudaEventDestroy(S.freed);
  }
  for (Table &T : tables_) {
    cudaFree(T.d);
    if (T.h)
      cudaFreeHost(T.h);
    if (T.copied)
      cudaEventDestroy(T.copied);
    if (T.freed)
      cudaEventDestroy(T.freed);
  }
  if (h2d_)
    cudaStreamDestroy(h2d_);
  cudaFree(d_linear_);
  cudaFree(d_err_);
}

void DeviceChunkDecoder::prepare() {
  if (h2d_)
    return;
  error_flag();
  static bool configured = false; // per process; setting it twice is harmless
  if (!configured) {
    configure_decoder<0>();
    configure_decoder<1>();
    configure_decoder<2>();
    configure_decoder<4>();
    configured = true;
  }
  for (Set &S : sets_) {
    check(cudaEventCreateWithFlags(&S.copied, cudaEventDisableTiming), "cudaEventCreate");
    check(cudaEventCreateWithFlags(&S.freed, cudaEventDisableTiming), "cudaEventCreate");
  }
  for (Table &T : tables_) {
    check(cudaEventCreateWithFlags(&T.copied, cudaEventDisableTiming), "cudaEventCreate");
    check(cudaEventCreateWithFlags(&T.freed, cudaEventDisableTiming), "cudaEventCreate");
  }
  check(cudaStreamCreateWithFlags(&h2d_, cudaStreamNonBlocking), "cudaStreamCreate");
}

DeviceChunkDecoder::Set &DeviceChunkDecoder::next_set(size_t in_bytes) {
  prepare();
  Set &S = sets_[next_];
  next_ = (next_ + 1) % kSets;
  if (in_bytes > S.in_cap) {
    if (S.used)
      check(cudaEventSynchronize(S.freed), "waiting for a staging set");
    grow(&S.d_in, S.in_cap, in_bytes, "cudaMalloc chunk staging");
  }
  // the copy may overwrite the set once the decode that read it is done
  check(cudaStreamWaitEvent(h2d_, S.freed, 0), "ordering a staging set");
  S.used = true;
  return S;
}

DeviceChunkDecoder::Table &DeviceChunkDecoder::next_table(size_t entries) {
  prepare();
  Table &T = tables_[next_table_];
  next_table_ = (next_table_ + 1) % kTables;
  if (T.used)
    // the host rewrites the page-locked copy below
    check(cudaEventSynchronize(T.copied), "waiting for a block table");
  if (entries > T.cap) {
    if (T.used)
      check(cudaEventSynchronize(T.freed), "waiting for a block table");
    if (T.h)
      cudaFreeHost(T.h);
    T.h = nullptr;
    cudaFree(T.d);
    T.d = nullptr;
    T.cap = 0;
    check(cudaMallocHost(&T.h, entries * sizeof(BlockDesc)), "cudaMallocHost block table");
    check(cudaMalloc(&T.d, entries * sizeof(BlockDesc)), "cudaMalloc block table");
    T.cap = entries;
  }
  check(cudaStreamWaitEvent(h2d_, T.freed, 0), "ordering a block table");
  T.used = true;
  return T;
}

void DeviceChunkDecoder::reserve(size_t chunk_bytes, size_t blocks) {
  for (int k = 0; k < kSets; k++)
    next_set(round16(chunk_bytes) + 16);
  for (int k = 0; k < kTables; k++)
    next_table(std::max<size_t>(blocks, 1));
}

void DeviceChunkDecoder::enqueue_raw(const void *src, size_t height, size_t row_bytes, void *dst,
                                     size_t dst_pitch, cudaStream_t s) {
  const size_t bytes = height * row_bytes;
  if (bytes == 0)
    return;
  Set &S = next_set(round16(bytes));
  check(cudaMemcpyAsync(S.d_in, src, bytes, cudaMemcpyDefault, h2d_), "copying a frame");
  check(cudaEventRecord(S.copied, h2d_), "cudaEventRecord");
  check(cudaStreamWaitEvent(s, S.copied, 0), "ordering after the copy");
  repitch(S.d_in, height, row_bytes, dst, dst_pitch, s);
  check(cudaEventRecord(S.freed, s), "cudaEventRecord");
}

int DeviceChunkDecoder::start_copy(const uint8_t *chunk, size_t nbytes) {
  Set &S = next_set(round16(nbytes) + 16);
  check(cudaMemcpyAsync(S.d_in, chunk, nbytes, cudaMemcpyDefault, h2d_), "copying a chunk");
  return static_cast<int>(&S - sets_);
}

void DeviceChunkDecoder::abandon() noexcept {
  if (h2d_)
    cudaStreamSynchronize(h2d_);
}

void DeviceChunkDecoder::enqueue(const uint8_t *chunk, size_t nbytes, const ChunkLayout &L,
                                 size_t height, size_t width, void *dst, size_t dst_pitch,
                                 cudaStream_t s, int started) {
  const size_t row_bytes = width * L.elem;
  if (L.algorithm == SF_CHUNK_RAW) {
    enqueue_raw(chunk, height, row_bytes, dst, dst_pitch, s);
    return;
  }
  const bool bs = L.algorithm == SF_CHUNK_BSLZ4;
  if (bs && L.elem != 1 && L.elem != 2 && L.elem != 4)
    throw std::invalid_argument("the device decodes 1, 2 or 4-byte bitshuffle elements");
  const size_t nb = L.block_in.size();
  if (nb == 0 && L.raw_bytes == 0)
    return;
  Set &S = sets_[started == kNotStarted ? start_copy(chunk, nbytes) : started];
  Table &T = next_table(std::max<size_t>(nb, 1));
  BlockDesc *t = static_cast<BlockDesc *>(T.h);
  uint32_t max_len = 0;
  for (size_t b = 0; b < nb; b++) {
    t[b] = BlockDesc{L.block_in[b], L.block_out[b], L.block_len[b], L.block_n[b]};
    max_len = std::max(max_len, L.block_len[b]);
  }
  if (nb)
    check(cudaMemcpyAsync(T.d, T.h, nb * sizeof(BlockDesc), cudaMemcpyHostToDevice, h2d_),
          "copying a block table");
  // the chunk's copy was enqueued before the table's
  check(cudaEventRecord(T.copied, h2d_), "cudaEventRecord");
  check(cudaStreamWaitEvent(s, T.copied, 0), "ordering after the copies");

  const uint64_t frame_bytes = static_cast<uint64_t>(height) * row_bytes;
  const auto *tbl = static_cast<const BlockDesc *>(T.d);
  const uint32_t n32 = static_cast<uint32_t>(nb);
  if (L.block_bytes > kMaxBlockBytes) {
    // plain LZ4 with blocks beyond shared memory (bitshuffle blocks never
    // are): decoded into a linear frame, then laid out at the pitch
    grow(&d_linear_, linear_cap_, round16(frame_bytes), "cudaMalloc frame staging");
    const unsigned grid = static_cast<unsigned>(std::max<size_t>(
        1, std::min<size_t>((nb + kDecodeWarps - 1) / kDecodeWarps,
                            static_cast<size_t>(device_sm_count()) * 16)));
    decode_linear<<<grid, kDecodeWarps * 32, 0, s>>>(S.d_in, tbl, n32, d_linear_, d_err_);
    check(cudaGetLastError(), "launching the chunk decoder");
    repitch(d_linear_, height, row_bytes, dst, dst_pitch, s);
    check(cudaEventRecord(S.freed, s), "cudaEventRecord");
    check(cudaEventRecord(T.freed, s), "cudaEventRecord");
    return;
  }
  const uint32_t out_bytes = static_cast<uint32_t>(round16(std::max<uint64_t>(L.block_bytes, 16)));
  const uint32_t stage_bytes = static_cast<uint32_t>(round16(std::min(max_len, kStageCap) + 15));
  const int e = bs ? static_cast<int>(L.elem) : 0;
  const size_t smem = static_cast<size_t>(kDecodeWarps) *
                      warp_layout(out_bytes, stage_bytes, static_cast<uint32_t>(e)).total;
  const unsigned grid = static_cast<unsigned>(std::max<size_t>(
      1, std::min<size_t>((nb + kDecodeWarps - 1) / kDecodeWarps,
                          static_cast<size_t>(device_sm_count()) * 16)));
  const uint64_t ways = reinterpret_cast<uintptr_t>(dst) | dst_pitch | row_bytes | L.block_bytes;
  const FrameDst D{static_cast<uint8_t *>(dst), dst_pitch, row_bytes,
                   ways % 4 == 0 ? 4u : ways % 2 == 0 ? 2u : 1u};
  const uint64_t raw_out = frame_bytes - L.raw_bytes;
  const uint32_t raw32 = static_cast<uint32_t>(L.raw_bytes);
  if (e == 0)
    decode_blocks<0><<<grid, kDecodeWarps * 32, smem, s>>>(S.d_in, tbl, n32, out_bytes,
                                                           stage_bytes, D, L.raw_in, raw32,
                                                           raw_out, d_err_);
  else if (e == 1)
    decode_blocks<1><<<grid, kDecodeWarps * 32, smem, s>>>(S.d_in, tbl, n32, out_bytes,
                                                           stage_bytes, D, L.raw_in, raw32,
                                                           raw_out, d_err_);
  else if (e == 2)
    decode_blocks<2><<<grid, kDecodeWarps * 32, smem, s>>>(S.d_in, tbl, n32, out_bytes,
                                                           stage_bytes, D, L.raw_in, raw32,
                                                           raw_out, d_err_);
  else
    decode_blocks<4><<<grid, kDecodeWarps * 32, smem, s>>>(S.d_in, tbl, n32, out_bytes,
                                                           stage_bytes, D, L.raw_in, raw32,
                                                           raw_out, d_err_);
  check(cudaGetLastError(), "launching the chunk decoder");
  check(cudaEventRecord(S.freed, s), "cudaEventRecord");
  check(cudaEventRecord(T.freed, s), "cudaEventRecord");
}

int *DeviceChunkDecoder::error_flag() {
  if (!d_err_) {
    check(cudaMalloc(&d_err_, sizeof(int)), "cudaMalloc");
    check(cudaMemset(d_err_, 0, sizeof(int)), "clearing the decode flag");
    check(cudaStreamSynchronize(cudaStreamLegacy), "clearing the decode flag");
  }
  return d_err_;
}

bool DeviceChunkDecoder::take_error() {
  if (!d_err_)
    return false;
  int v = 0;
  check(cudaMemcpy(&v, d_err_, sizeof(int), cudaMemcpyDeviceToHost), "reading the decode flag");
  if (v)
    check(cudaMemset(d_err_, 0, sizeof(int)), "clearing the decode flag");
  return v != 0;
}

} // namespace sf

extern "C" int sf_chunk_decode_device(int algorithm, const void *chunk, size_t nbytes,
                                      size_t height, size_t width, int elem_bytes,
                                      void *device_image, size_t pitch_bytes) {
  return sf::guarded([&] {
    if (!chunk || !device_image || height == 0 || width == 0 ||
        (elem_bytes != 2 && elem_bytes != 4) || pitch_bytes < width * elem_bytes)
      return -1;
    // per host thread: a stream and a decoder, reused by later calls
    struct Local {
      cudaStream_t s = nullptr;
      sf::DeviceChunkDecoder dec;
      ~Local() {
        if (s) {
          cudaStreamSynchronize(s);
          cudaStreamDestroy(s);
        }
      }
    };
    static thread_local Local loc;
    if (!loc.s)
      sf::check(cudaStreamCreateWithFlags(&loc.s, cudaStreamNonBlocking), "cudaStreamCreate");
    const auto *bytes = static_cast<const uint8_t *>(chunk);
    const size_t eb = static_cast<size_t>(elem_bytes);
    const int started = sf::may_copy_first(algorithm, nbytes, height * width, eb)
                            ? loc.dec.start_copy(bytes, nbytes)
                            : sf::DeviceChunkDecoder::kNotStarted;
    try {
      const sf::ChunkLayout L = sf::parse_chunk(algorithm, bytes, nbytes, height * width, eb);
      loc.dec.enqueue(bytes, nbytes, L, height, width, device_image, pitch_bytes, loc.s, started);
    } catch (...) {
      loc.dec.abandon();
      throw;
    }
    sf::check(cudaStreamSynchronize(loc.s), "cudaStreamSynchronize");
    if (loc.dec.take_error())
      throw sf::DeviceError("a malformed LZ4 block");
    return 0;
  });
}
