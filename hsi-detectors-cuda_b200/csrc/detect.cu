// detect.cu - threshold + non-maximum suppression + ordered compaction.
//
// Two launches for a whole batch of score maps (three when a map is very
// tall), no atomics, so every list comes out in raster order and is identical
// run to run:
//   1. flags:  one warp per 2048-pixel row segment writes every pixel's
//              pass/fail as ballot words (a bitmask in the workspace) and the
//              segment's count.  The map streams through once; a
//              candidate (a score past the threshold) looks at its
//              (2r+1)^2 window, straight from global memory, where the
//              block's eight warps -- neighbouring rows -- have brought it
//              into L1, and a chunk of 128 pixels with more than a few
//              candidates at the windows of all of them together.  A
//              neighbour suppresses when it comes first in the window's order
//              (better score, or the same score at a lower linear index);
//              out-of-frame neighbours are skipped and NaN never wins or
//              ties, exactly like the CPU loop.
//   2. emit:   a block takes eight segments of one map, adds up the counts of
//              the segments before them, and each warp writes its segment's
//              detections at offset + in-segment rank, dropping (but having
//              counted) those past capacity.  The map's last block advances
//              *count.  Maps of more than kDirectSegs segments, where those
//              sums would cost more than a launch, get their offsets from a
//              scan launch in between.
// Semantics are the reference CPU path's (src/sam_cpu.cpp:86-138), polarity
// included; the reference GPU kernel (src/detect.cu:43-87) ignores polarity
// and emits in atomic arrival order, both of which this replaces.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "launch_state.h"

namespace hsi_b200 {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;        // row segments per block of flags and emit
constexpr int kSeg = 2048;                   // pixels per row segment
constexpr int kWordsPerSeg = kSeg / 32;      // 64
constexpr int kMaxJobs = 64;
constexpr int kChunk = 128;                  // pixels a warp takes at a time, four per lane
constexpr int kGroupR = 2;                   // largest radius of the lanes' own windows on 16-byte groups
constexpr int kHeldR = 4;                    // largest radius with an instance of its own
constexpr int kDenseR = 8;                   // largest radius of a whole chunk's windows
// A block of emit reads the counts of all earlier segments of its map: 2 KB on
// average for 1024 rows.  At 16384 segments (a 16384-row map) the 2048 blocks
// read 64 MB of L2 together, about what a scan launch costs; the sums grow
// with the square of the height.
constexpr int kDirectSegs = 16384;

struct Job {
  const float* score;
  const int32_t* target;
  int height, width;
  float threshold;
  int radius;
  int higher;
  int vec;           // rows start on 16 bytes
  int capacity;
  hsi_detection* out;
  uint32_t* count;
  int seg0;          // first segment of this map in the batch
  int segs_per_row;  // ceil(width / kSeg)
  int unit0;         // first block of eight segments of this map in the batch
};

// N: job slots; a single map travels in a small parameter block.
template <int N>
struct Batch {
  Job jobs[N];
  int njobs;
  int units;          // blocks of flags and of emit
  uint32_t* counts;   // [total_segs]
  uint32_t* offsets;  // [total_segs]; without a scan only a map's first entry: its *count at the start
  uint32_t* masks;    // [total_segs * 64]
};

template <int N>
__device__ __forceinline__ int find_job(const Batch<N>& b, int unit) {
  if constexpr (N == 1) return 0;
  int lo = 0, hi = b.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (b.jobs[mid].unit0 <= unit) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <bool HIGHER>
__device__ __forceinline__ bool over_threshold(float s, float threshold) {
  return HIGHER ? s >= threshold : s <= threshold;  // NaN fails both
}

// Whether neighbour o suppresses the candidate s: a better score, or the same
// score when the neighbour comes `earlier` in linear index.  NaN never does.
template <bool HIGHER>
__device__ __forceinline__ bool suppresses(float o, float s, bool earlier) {
  if (HIGHER) return earlier ? o >= s : o > s;
  return earlier ? o <= s : o < s;
}

// One candidate by a whole warp, a lane per neighbour and round, rows nearest
// the candidate first (smooth maps decide in the first round): any radius.
// A few per cent of the pixels are candidates, so a 128-pixel chunk has two or
// three; they cost about 20 instructions each here, where the whole chunk's
// windows (below) cost some hundreds however few of its pixels are candidates.
// So up to kFew candidates of a chunk go one by one.  Eight 1024 x 1024 maps
// with 5 % of uniform random scores past the threshold (6.4 a chunk), kFew 3, 6
// and 10: radius 1 42, 50 and 59 us, 2 58, 55 and 60, 4 74, 80 and 85, 8 99, 109
// and 123, 12 156, 149 and 147.
// 64 such maps with 1 and 30 % past the threshold, radius 2: 206 and 409 us for
// both launches; the ring-buffer tiles before (one barrier per row, then a scan
// launch) took 444 and 478.  One 64 x 96 map: 5.4 us against 69, where a tile
// walked its 64 rows in one block.
constexpr int kFew = 4;
constexpr int kRounds = 3;       // rounds whose neighbours a lane keeps: all of them up to radius kHeldR
constexpr unsigned kFlatR = 16;  // largest radius whose further rounds run across the window's rows
// Window rows in the order 0, 1, -1, 2, -2, ..: the side is 2 r + 1 with r up to
// the map's larger side, which may take the whole of 32 bits, and a row is up to
// 2^31 pixels, so its neighbours' offsets take 64.
struct WarpWindow {
  unsigned side;               // 2 r + 1
  int dx[kRounds], dy[kRounds];  // this lane's neighbours; (0, 0), the candidate itself, past the window
};
__device__ __forceinline__ int window_row(unsigned i) {
  return (i & 1u) ? static_cast<int>(i / 2u) + 1 : -static_cast<int>(i / 2u);
}
__device__ __forceinline__ void warp_neighbour(unsigned k, unsigned side, int& dx, int& dy) {
  dx = dy = 0;
  if (k >= static_cast<uint64_t>(side) * side) return;
  const unsigned i = k / side;
  dy = window_row(i);
  dx = static_cast<int>(k - i * side) - static_cast<int>(side / 2u);
}
__device__ __forceinline__ WarpWindow warp_window(const Job& J) {
  WarpWindow w;
  w.side = 2u * static_cast<unsigned>(J.radius) + 1u;
#pragma unroll
  for (int k = 0; k < kRounds; ++k) warp_neighbour(32 * k + (threadIdx.x & 31), w.side, w.dx[k], w.dy[k]);
  return w;
}
// Whether the neighbour at (x + dx, y + dy), if the map has it, suppresses the candidate s at (x, y).
template <bool HIGHER>
__device__ __forceinline__ bool neighbour_suppresses(const Job& J, int x, int y, int dx, int dy, float s) {
  const int nx = x + dx, ny = y + dy;
  const bool in = static_cast<unsigned>(nx) < static_cast<unsigned>(J.width) &&
                  static_cast<unsigned>(ny) < static_cast<unsigned>(J.height);
  const float o = in ? __ldg(J.score + static_cast<int64_t>(ny) * J.width + nx) : __int_as_float(0x7fc00000);
  return suppresses<HIGHER>(o, s, dy < 0 || (dy == 0 && dx < 0));
}
template <int R, bool HIGHER>
__device__ __forceinline__ bool warp_suppressed(const Job& J, const WarpWindow& w, int x, int y, float s) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kHeld = R <= 2 ? 1 : R == 3 ? 2 : kRounds;
#pragma unroll
  for (int k = 0; k < kHeld; ++k)
    if (__any_sync(kAll, neighbour_suppresses<HIGHER>(J, x, y, w.dx[k], w.dy[k], s))) return true;
  if constexpr (R <= kHeldR) return false;
  const int lane = threadIdx.x & 31, r = static_cast<int>(w.side / 2u);
  if (w.side <= 2 * kFlatR + 1 && 2 * (min(y + r, J.height - 1) - max(y - r, 0)) >= r) {
#pragma unroll 1
    for (unsigned k = 32 * kHeld; k < w.side * w.side; k += 32) {
      int dx, dy;
      warp_neighbour(k + lane, w.side, dx, dy);
      if (__any_sync(kAll, neighbour_suppresses<HIGHER>(J, x, y, dx, dy, s))) return true;
    }
    return false;
  }
  // rows of more than a warp's lanes, or most of them outside the map: row by row
  const float* p = J.score + static_cast<int64_t>(y) * J.width + x;
  const int lo = max(x - r, 0), hi = r < J.width - 1 - x ? x + r : J.width - 1;
#pragma unroll 1
  for (unsigned i = 32 * kHeld / w.side; i < w.side; ++i) {
    const int dy = window_row(i);
    if (static_cast<unsigned>(y) + static_cast<unsigned>(dy) >= static_cast<unsigned>(J.height)) continue;
    const float* row = p + static_cast<int64_t>(dy) * J.width - x;
    for (int n0 = lo; n0 <= hi; n0 += 32) {
      const int nx = n0 + lane;
      const bool in = nx <= hi;
      const float o = __ldg(in ? row + nx : p);
      if (__any_sync(kAll, suppresses<HIGHER>(o, s, in && (dy < 0 || (dy == 0 && nx < x))))) return true;
    }
  }
  return false;
}

// ---- the windows of a whole chunk --------------------------------------------
//
// Slot j of lane l is column 32 j + l of the chunk; slot 4 holds the columns
// beside it, lanes 16..31 those on its left (slot -1) and lanes 0..15 those on
// its right.
struct Columns {
  float v[5];
};

template <bool HIGHER>
__device__ __forceinline__ float first_of(float a, float b) { return HIGHER ? fmaxf(a, b) : fminf(a, b); }  // NaN never
template <bool HIGHER>
__device__ __forceinline__ Columns first_of(const Columns& a, const Columns& b) {
  Columns c;
#pragma unroll
  for (int j = 0; j < 5; ++j) c.v[j] = first_of<HIGHER>(a.v[j], b.v[j]);
  return c;
}
// The columns d to the right (d <= 8): every slot.
__device__ __forceinline__ Columns right_of(const Columns& a, int d) {
  const int lane = threadIdx.x & 31;
  const bool wraps = lane < d;  // the taker, d lanes lower around the warp, wants the next slot's
  Columns c;
#pragma unroll
  for (int j = 0; j < 5; ++j)
    c.v[j] = __shfl_sync(0xffffffffu, wraps ? a.v[j == 4 ? 0 : j + 1] : a.v[j], (lane + d) & 31);
  return c;
}
// The columns d to the left (d <= 8): slots 0..3.
__device__ __forceinline__ Columns left_of(const Columns& a, int d) {
  const int lane = threadIdx.x & 31;
  const bool wraps = lane >= 32 - d;
  Columns c;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    c.v[j] = __shfl_sync(0xffffffffu, wraps ? a.v[j == 0 ? 4 : j - 1] : a.v[j], (lane - d) & 31);
  c.v[4] = c.v[3];
  return c;
}

// The chunks of a segment with more than kFew candidates (bit i of `chunks`: the
// columns from xs + 128 i on) at the job's radius, 1 and up: their mask words;
// returns how many pixels pass.  A neighbour suppresses by its score and by
// whether it comes before or after the candidate, so the candidate passes when
// the first score of the rows above and of its row's columns on the left is not
// as good as its own, and that of the rows below and of the columns on the
// right is not better.  Each column's first scores above and below are found
// once, by one coalesced load a row and 32 columns; the window's width is
// covered by doubling, with shuffles.  The eight neighbours come first: they
// leave few pixels of a smooth map, which go one by one, and a ninth of a
// random one.  So do the pixels that pass at kDenseR where the radius is larger.
// 2 r + 1 loads of five slots and some 250 instructions for the 128 pixels.  Eight
// random 1024 x 1024 maps, 30 % past the threshold: radius 3 68 us, 4 77, 5 85, 8
// 103; 1023 x 1021 the same.  A window per pixel (49 and 81 neighbours) took 89
// and 122 us on 16-byte groups, 180 and 310 on rows that do not start on 16
// bytes, and the ring-buffer tiles before 111, 127, 262 and 368.
// One copy behind all instances of flag_segment, which outgrow the instruction
// cache otherwise; a call from inside their loops spilled their registers.
template <bool HIGHER>
__device__ __forceinline__ uint32_t dense_chunks(const Job& J, int y, int xs, unsigned chunks, uint32_t* mask) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const float nan = __int_as_float(0x7fc00000);
  const int width = J.width, height = J.height, r = min(J.radius, kDenseR);
  const float threshold = J.threshold;
  uint32_t total = 0;
#pragma unroll 1
  for (; chunks != 0u; chunks &= chunks - 1u) {
    const int xc = xs + kChunk * (__ffs(chunks) - 1);
    const int left = width - xc - lane;  // columns from this lane's first on
    const bool beside = lane >= 16 ? (xc > 0 && lane >= 32 - r) : (lane < r && left > 128);
    const int xb = lane >= 16 ? lane - 32 : 128 + lane;
    const float* centre = J.score + static_cast<int64_t>(y) * width + xc;
    const auto load = [&](int dy) {
      const float* p = centre + static_cast<int64_t>(dy) * width;
      Columns c;
#pragma unroll
      for (int j = 0; j < 4; ++j) c.v[j] = left > 32 * j ? __ldg(p + lane + 32 * j) : nan;
      c.v[4] = beside ? __ldg(p + xb) : nan;
      return c;
    };
    const Columns none{{nan, nan, nan, nan, nan}};
    Columns here = load(0), above = y >= 1 ? load(-1) : none, below = height - y > 1 ? load(1) : none;
    const Columns s = here;
    uint32_t word[4];  // bit l of word j: column xc + 32 j + l
    const auto pass = [&](const Columns& before, const Columns& after) {
      int n = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        word[j] = __ballot_sync(kAll, over_threshold<HIGHER>(s.v[j], threshold) &&
                                          !suppresses<HIGHER>(before.v[j], s.v[j], true) &&
                                          !suppresses<HIGHER>(after.v[j], s.v[j], false));
        n += __popc(word[j]);
      }
      return n;
    };
    const Columns l = first_of<HIGHER>(above, here), rr = first_of<HIGHER>(here, below);
    int n = pass(first_of<HIGHER>(first_of<HIGHER>(left_of(l, 1), above), right_of(above, 1)),
                 first_of<HIGHER>(first_of<HIGHER>(right_of(rr, 1), below), left_of(below, 1)));
    bool decided = J.radius == 1;
    if (!decided && n > kFew) {
#pragma unroll 2
      for (int d = 2; d <= r; ++d) {
        const Columns a = y >= d ? load(-d) : none, b = height - y > d ? load(d) : none;
        above = first_of<HIGHER>(above, a);
        below = first_of<HIGHER>(below, b);
      }
      // the first of q columns from each one on, q the largest power of two <= r;
      // 2 q then covers more than half of the window of 2 r + 1
      int q = 1;
#pragma unroll 1
      for (; 2 * q <= r; q *= 2) {
        above = first_of<HIGHER>(above, right_of(above, q));
        below = first_of<HIGHER>(below, right_of(below, q));
        here = first_of<HIGHER>(here, right_of(here, q));
      }
      above = first_of<HIGHER>(above, right_of(above, q));
      below = first_of<HIGHER>(below, right_of(below, q));
      const int rest = 2 * q - r - 1;  // the 2 q columns that end the window start here, on the left of the pixel
      n = pass(first_of<HIGHER>(first_of<HIGHER>(left_of(above, r), left_of(above, rest)),
                                first_of<HIGHER>(left_of(here, r), left_of(here, q))),
               first_of<HIGHER>(first_of<HIGHER>(left_of(below, r), left_of(below, rest)),
                                first_of<HIGHER>(right_of(here, 1), right_of(here, r - q + 1))));
      decided = J.radius <= kDenseR;
    }
    uint32_t m = lane < 2 ? (lane == 0 ? word[0] : word[1]) : (lane == 2 ? word[2] : word[3]);
    if (!decided && n > 0) {
      const WarpWindow ww = warp_window(J);
      uint32_t todo = lane < 4 ? m : 0u;
      for (unsigned lanes = __ballot_sync(kAll, todo != 0u); lanes != 0u; lanes = __ballot_sync(kAll, todo != 0u)) {
        const int j = __ffs(lanes) - 1;
        const int bit = __ffs(__shfl_sync(kAll, todo, j)) - 1;
        const int c = 32 * j + bit;
        const bool out = warp_suppressed<kHeldR + 1, HIGHER>(J, ww, xc + c, y, __ldg(centre + c));
        if (lane == j) {
          todo &= todo - 1u;
          if (out) m &= ~(1u << bit);
        }
      }
    }
    if (lane < 4 && width - xc > 32 * lane) {
      mask[(xc - xs) / 32 + lane] = m;
      total += __popc(m);
    }
  }
  return __reduce_add_sync(kAll, total);
}

// The windows of the four pixels x .. x + 3 of a lane at a fixed radius, on
// 16-byte groups: rows dy0 .. dy1 of the window, all of their loads in flight
// together.  Clears the pixels of `keep` that a neighbour suppresses.  The
// width is a multiple of 4, so a group lies wholly inside or outside the map.
template <int R, int DY0, int DY1, bool HIGHER>
__device__ __forceinline__ void window_rows(const Job& J, int x, int y, const float (&s)[4], unsigned& keep) {
  const float nan = __int_as_float(0x7fc00000);
  float4 g[DY1 - DY0 + 1][3];
#pragma unroll
  for (int dy = DY0; dy <= DY1; ++dy) {
    const int ny = y + dy;
    const bool row = ny >= 0 && ny < J.height;
    const float4* p = reinterpret_cast<const float4*>(J.score + static_cast<int64_t>(row ? ny : y) * J.width + x);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const bool in = row && (k != 0 || x >= 4) && (k != 2 || x + 4 < J.width);
      g[dy - DY0][k] = in ? __ldg(p + k - 1) : make_float4(nan, nan, nan, nan);
    }
  }
#pragma unroll
  for (int dy = DY0; dy <= DY1; ++dy) {
    const float4(&q)[3] = g[dy - DY0];
    const float v[12] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w, q[2].x, q[2].y, q[2].z, q[2].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      bool hit = false;
#pragma unroll
      for (int dx = -R; dx <= R; ++dx) {
        if (dy == 0 && dx == 0) continue;
        hit |= suppresses<HIGHER>(v[4 + j + dx], s[j], dy < 0 || (dy == 0 && dx < 0));
      }
      if (hit) keep &= ~(1u << j);
    }
  }
}

// Three rows at a time: 36 registers of loads in flight.
template <int R, bool HIGHER, int DY = -R>
__device__ __forceinline__ void window(const Job& J, int x, int y, const float (&s)[4], unsigned& keep) {
  static_assert(R >= 1 && R <= kGroupR, "one group each side");
  if (keep == 0) return;
  constexpr int kLast = DY + 2 < R ? DY + 2 : R;
  window_rows<R, DY, kLast, HIGHER>(J, x, y, s, keep);
  if constexpr (kLast < R) window<R, HIGHER, kLast + 1>(J, x, y, s, keep);
}

// Bits 0..7 of x moved to bits 0, 4, .., 28.
__device__ __forceinline__ uint32_t spread4(uint32_t x) {
  x = (x | (x << 12)) & 0x000F000Fu;
  x = (x | (x << 6)) & 0x03030303u;
  x = (x | (x << 3)) & 0x11111111u;
  return x;
}

// The four pixels of a lane in one chunk.  VEC (rows on 16 bytes, width a
// multiple of 4): columns 4l .. 4l + 3; otherwise l, l + 32, l + 64, l + 96.
template <bool VEC>
__device__ __forceinline__ int column_of(int lane, int j) { return VEC ? 4 * lane + j : 32 * j + lane; }

template <bool VEC>
__device__ __forceinline__ float4 load_chunk(const float* __restrict__ row, int x0, int end) {
  const int lane = threadIdx.x & 31;
  const float nan = __int_as_float(0x7fc00000);
  float4 c = make_float4(nan, nan, nan, nan);
  if constexpr (VEC) {
    if (x0 + 4 * lane < end) c = __ldg(reinterpret_cast<const float4*>(row + x0 + 4 * lane));
  } else {
    const float* p = row + x0 + lane;
    if (x0 + lane < end) c.x = __ldg(p);
    if (x0 + lane + 32 < end) c.y = __ldg(p + 32);
    if (x0 + lane + 64 < end) c.z = __ldg(p + 64);
    if (x0 + lane + 96 < end) c.w = __ldg(p + 96);
  }
  return c;
}

struct SegmentFlags {
  uint32_t count;  // pixels that pass
  unsigned dense;  // bit i: the chunk of columns from 128 i on is left to dense_chunks
};

// One segment: mask words and count.  R = kHeldR + 1 stands for any radius
// above kHeldR.  The body of a chunk exists once per instance (the candidates
// of all four pixel slots share one loop, three chunks are loaded ahead by
// rotation instead of unrolling): unrolled sixteen-fold the instances
// outgrew the instruction cache and ran at half this speed.
template <int R, bool HIGHER, bool VEC>
__device__ __forceinline__ SegmentFlags flag_segment(const Job& J, int y, int xs, uint32_t* mask) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int end = min(J.width, xs + kSeg);
  const float* row = J.score + static_cast<int64_t>(y) * J.width;
  uint32_t total = 0;
  unsigned dense = 0;
  WarpWindow ww{};
  if constexpr (R > 0) ww = warp_window(J);
  float4 c = load_chunk<VEC>(row, xs, end), c1 = load_chunk<VEC>(row, xs + kChunk, end);
  float4 c2 = load_chunk<VEC>(row, xs + 2 * kChunk, end);
#pragma unroll 1
  for (int xc = xs; xc < end; xc += kChunk) {
    const float4 c3 = load_chunk<VEC>(row, xc + 3 * kChunk, end);
    const float s[4] = {c.x, c.y, c.z, c.w};
    unsigned keep = 0;  // bit j: pixel j of this lane passes
#pragma unroll
    for (int j = 0; j < 4; ++j) keep |= over_threshold<HIGHER>(s[j], J.threshold) ? 1u << j : 0u;
    unsigned n = 0;
    if constexpr (R > 0) n = __reduce_add_sync(kAll, __popc(keep));
    if (n > kFew && !(VEC && R <= kGroupR)) {
      dense |= 1u << ((xc - xs) / kChunk);
    } else {
      if constexpr (VEC && R > 0 && R <= kGroupR) {
        if (n > kFew) {
          window<R, HIGHER>(J, xc + 4 * lane, y, s, keep);
          __syncwarp();
          n = 0;  // decided
        }
      }
      if (n > 0) {
        unsigned todo = keep;
        for (unsigned lanes = __ballot_sync(kAll, todo != 0u); lanes != 0u; lanes = __ballot_sync(kAll, todo != 0u)) {
          const int l = __ffs(lanes) - 1;
          const int j = __ffs(__shfl_sync(kAll, todo, l)) - 1;
          const float mine = j < 2 ? (j == 0 ? s[0] : s[1]) : (j == 2 ? s[2] : s[3]);
          const float sl = __shfl_sync(kAll, mine, l);
          const bool out = warp_suppressed<R, HIGHER>(J, ww, xc + column_of<VEC>(l, j), y, sl);
          if (lane == l) {
            todo &= todo - 1u;
            if (out) keep &= ~(1u << j);
          }
        }
      }
      uint32_t word[4];  // bit l of word j: column_of(l, j)
#pragma unroll
      for (int j = 0; j < 4; ++j) total += __popc(word[j] = __ballot_sync(kAll, (keep >> j) & 1u));
      if (lane < 4 && xc + 32 * lane < end) {
        uint32_t m = 0u;
        if constexpr (VEC) {  // columns 32 lane + 4i + j come from bit 8 lane + i of word[j]
#pragma unroll
          for (int j = 0; j < 4; ++j) m |= spread4((word[j] >> (8 * lane)) & 0xffu) << j;
        } else {
          m = lane < 2 ? (lane == 0 ? word[0] : word[1]) : (lane == 2 ? word[2] : word[3]);
        }
        mask[(xc - xs) / 32 + lane] = m;
      }
    }
    c = c1;
    c1 = c2;
    c2 = c3;
  }
  return {total, dense};
}

template <int R, bool HIGHER>
__device__ __forceinline__ SegmentFlags flag_radius(const Job& J, int y, int xs, uint32_t* mask) {
  return J.vec ? flag_segment<R, HIGHER, true>(J, y, xs, mask) : flag_segment<R, HIGHER, false>(J, y, xs, mask);
}

template <bool HIGHER>
__device__ __forceinline__ SegmentFlags flag_dispatch(const Job& J, int y, int xs, uint32_t* mask) {
  switch (J.radius > 0 ? J.radius : 0) {
    case 0: return flag_radius<0, HIGHER>(J, y, xs, mask);
    case 1: return flag_radius<1, HIGHER>(J, y, xs, mask);
    case 2: return flag_radius<2, HIGHER>(J, y, xs, mask);
    case 3: return flag_radius<3, HIGHER>(J, y, xs, mask);
    case 4: return flag_radius<4, HIGHER>(J, y, xs, mask);
    default: return flag_radius<kHeldR + 1, HIGHER>(J, y, xs, mask);
  }
}

template <int N>
__global__ void __launch_bounds__(kThreads, 4) flags_kernel(const __grid_constant__ Batch<N> b) {
  const Job& J = b.jobs[find_job(b, blockIdx.x)];
  const int local = (blockIdx.x - J.unit0) * kWarps + (threadIdx.x >> 5);
  if (local >= J.height * J.segs_per_row) return;
  const int y = local / J.segs_per_row, xs = (local % J.segs_per_row) * kSeg;
  const int seg = J.seg0 + local;
  uint32_t* mask = b.masks + static_cast<int64_t>(seg) * kWordsPerSeg;
  const SegmentFlags f = J.higher ? flag_dispatch<true>(J, y, xs, mask) : flag_dispatch<false>(J, y, xs, mask);
  uint32_t n = f.count;
  if (f.dense != 0u)
    n += J.higher ? dense_chunks<true>(J, y, xs, f.dense, mask) : dense_chunks<false>(J, y, xs, f.dense, mask);
  if ((threadIdx.x & 31) == 0) {
    b.counts[seg] = n;
    if (local == 0) b.offsets[seg] = *J.count;  // before emit's last block advances it
  }
}

// Mask words of segment `local` of job J that cover pixels of the map (words
// past the row's end are never written).
__device__ __forceinline__ int seg_words(const Job& J, int local) {
  const int xs = (local % J.segs_per_row) * kSeg;
  const int len = min(kSeg, J.width - xs);
  return (len + 31) / 32;
}

// One block per map: the segments' offsets, from *count; *count += total.
template <int N>
__global__ void __launch_bounds__(1024) scan_kernel(const __grid_constant__ Batch<N> b) {
  __shared__ uint32_t s_warp[32];
  const Job& J = b.jobs[blockIdx.x];
  const int segs = J.height * J.segs_per_row;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t carry = *J.count;
  for (int chunk = 0; chunk < segs; chunk += 1024) {
    const int i = chunk + threadIdx.x;
    const uint32_t v = i < segs ? b.counts[J.seg0 + i] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    __syncthreads();  // the previous chunk's sums have been read
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += o;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    if (i < segs) b.offsets[J.seg0 + i] = carry + (warp > 0 ? s_warp[warp - 1] : 0u) + incl - v;
    carry += s_warp[31];
  }
  __syncthreads();  // every thread has read *count
  if (threadIdx.x == 0) *J.count = carry;
}

// One warp per segment, eight consecutive segments of a map per block.  Lane l
// holds mask words l and l + 32, their exclusive prefix of popcounts comes
// from two shuffle scans, and the warp then visits the non-empty words in
// order with lane = bit, so that the detections of one word go to consecutive
// slots in one coalesced store.
template <int N, bool SCANNED>
__global__ void __launch_bounds__(kThreads) emit_kernel(const __grid_constant__ Batch<N> b) {
  __shared__ uint32_t s_sum[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Job& J = b.jobs[find_job(b, blockIdx.x)];
  const int segs = J.height * J.segs_per_row;
  const int first = (blockIdx.x - J.unit0) * kWarps;  // this block's segments
  const int local = first + warp;
  const int seg = J.seg0 + local;
  const uint32_t* counts = b.counts + J.seg0;
  const uint32_t count = local < segs ? counts[local] : 0u;
  uint32_t base;
  if constexpr (SCANNED) {
    if (count == 0u) return;  // nothing passed in this segment (the same for the whole warp)
    base = b.offsets[seg];
  } else {
    const bool last = first + kWarps >= segs;
    if (!__syncthreads_or(count != 0u) && !last) return;
    uint32_t before = 0;
#pragma unroll 4
    for (int i = threadIdx.x; i < first; i += kThreads) before += counts[i];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_sum[warp] = before;
    __syncthreads();
    base = b.offsets[J.seg0];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) base += s_sum[w];
    uint32_t mine = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = first + w < segs ? counts[first + w] : 0u;
      if (w < warp) mine += c;
      all += c;
    }
    if (last && threadIdx.x == 0) *J.count = base + all;
    base += mine;
    if (count == 0u) return;
  }
  const uint32_t lt = (1u << lane) - 1u;
  const int nw = seg_words(J, local);
  const uint32_t* m = b.masks + static_cast<int64_t>(seg) * kWordsPerSeg;
  const uint32_t w0 = lane < nw ? m[lane] : 0u;
  const uint32_t w1 = lane + 32 < nw ? m[lane + 32] : 0u;
  const uint32_t c0 = __popc(w0), c1 = __popc(w1);
  uint32_t i0 = c0, i1 = c1;  // inclusive scans over the lanes
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o0 = __shfl_up_sync(0xffffffffu, i0, d);
    const uint32_t o1 = __shfl_up_sync(0xffffffffu, i1, d);
    if (lane >= d) {
      i0 += o0;
      i1 += o1;
    }
  }
  const uint32_t first_half = __shfl_sync(0xffffffffu, i0, 31);
  const uint32_t e0 = i0 - c0, e1 = first_half + i1 - c1;  // exclusive prefixes of words lane, lane + 32
  const int y = local / J.segs_per_row;
  const int x0 = (local % J.segs_per_row) * kSeg;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const uint32_t mine = half ? w1 : w0, pre = half ? e1 : e0;
    uint32_t nonempty = __ballot_sync(0xffffffffu, mine != 0u);
    while (nonempty) {
      const int wi = __ffs(nonempty) - 1;
      nonempty &= nonempty - 1u;
      const uint32_t word = __shfl_sync(0xffffffffu, mine, wi);
      const uint32_t wpre = __shfl_sync(0xffffffffu, pre, wi);
      if ((word >> lane) & 1u) {
        const uint32_t slot = base + wpre + __popc(word & lt);
        if (slot < static_cast<uint32_t>(J.capacity)) {
          const int x = x0 + (32 * half + wi) * 32 + lane;
          const int64_t p = static_cast<int64_t>(y) * J.width + x;
          hsi_detection d;
          d.x = x;
          d.y = y;
          d.target = J.target ? J.target[p] : 0;
          d.score = J.score[p];
          J.out[slot] = d;
        }
      }
    }
  }
}

// Row segments of a map; 64-bit, so sizes far past the limits below stay exact.
int64_t segs_of(int height, int width) {
  return static_cast<int64_t>(height) * ((static_cast<int64_t>(width) + kSeg - 1) / kSeg);
}

// Largest segment count of one batch (the kernels index segments in int).
constexpr int64_t kMaxBatchSegs = 0x3fffffff;

size_t ws_bytes_for_segs(int64_t segs) { return static_cast<size_t>(segs) * sizeof(uint32_t) * (2 + kWordsPerSeg) + 256; }

template <int N>
int launch_batch(const hsi_detect_job* jobs, int n, void* ws, size_t ws_bytes, cudaStream_t s) {
  Batch<N> b;
  int64_t segs = 0, units = 0;
  bool direct = true;
  for (int i = 0; i < n; ++i) {
    const hsi_detect_job& j = jobs[i];
    if (!j.score || !j.count || j.height <= 0 || j.width <= 0 || j.capacity < 0) return HSI_E_INVALID;
    if (j.capacity > 0 && !j.out) return HSI_E_INVALID;
    if (j.polarity != HSI_LOWER_IS_BETTER && j.polarity != HSI_HIGHER_IS_BETTER) return HSI_E_INVALID;
    Job& J = b.jobs[i];
    J.score = j.score;
    J.target = j.target;
    J.height = j.height;
    J.width = j.width;
    J.threshold = j.threshold;
    // a window past the map's far edges sees no more of it
    J.radius = std::min(j.nms_radius, std::max(j.height, j.width));
    J.higher = j.polarity == HSI_HIGHER_IS_BETTER;
    J.vec = j.width % 4 == 0 && (reinterpret_cast<uintptr_t>(j.score) & 15u) == 0;
    J.capacity = j.capacity;
    J.out = j.out;
    J.count = j.count;
    J.seg0 = static_cast<int>(segs);
    J.segs_per_row = (j.width + kSeg - 1) / kSeg;
    J.unit0 = static_cast<int>(units);
    const int64_t map_segs = segs_of(j.height, j.width);
    segs += map_segs;
    units += (map_segs + kWarps - 1) / kWarps;
    if (segs > kMaxBatchSegs) return HSI_E_CAPACITY;
    direct = direct && map_segs <= kDirectSegs;
  }
  if (!ws || ws_bytes < ws_bytes_for_segs(segs)) return HSI_E_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(ws) & 15u) != 0) return HSI_E_INVALID;
  b.njobs = n;
  b.units = static_cast<int>(units);
  uint32_t* p = static_cast<uint32_t*>(ws);
  b.counts = p;
  b.offsets = p + segs;
  b.masks = p + 2 * segs;
  flags_kernel<N><<<b.units, kThreads, 0, s>>>(b);
  if (direct) {
    emit_kernel<N, false><<<b.units, kThreads, 0, s>>>(b);
  } else {
    scan_kernel<N><<<n, 1024, 0, s>>>(b);
    emit_kernel<N, true><<<b.units, kThreads, 0, s>>>(b);
  }
  return static_cast<int>(cudaGetLastError());
}

int run_batch(const hsi_detect_job* jobs, int n, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (!jobs || n <= 0 || n > kMaxJobs) return HSI_E_INVALID;
  return n == 1 ? launch_batch<1>(jobs, n, ws, ws_bytes, s) : launch_batch<kMaxJobs>(jobs, n, ws, ws_bytes, s);
}

}  // namespace
}  // namespace hsi_b200

using namespace hsi_b200;

extern "C" HSI_API size_t hsi_detect_workspace_bytes(int height, int width) {
  if (height <= 0 || width <= 0) return 0;
  const int64_t segs = segs_of(height, width);
  return segs > kMaxBatchSegs ? 0 : ws_bytes_for_segs(segs);
}

extern "C" HSI_API size_t hsi_detect_batch_workspace_bytes(const hsi_detect_job* jobs, int num_jobs) {
  if (!jobs || num_jobs <= 0) return 0;
  int64_t segs = 0;
  for (int i = 0; i < num_jobs; ++i) {
    if (jobs[i].height <= 0 || jobs[i].width <= 0) return 0;
    segs += segs_of(jobs[i].height, jobs[i].width);
    if (segs > kMaxBatchSegs) return 0;
  }
  return ws_bytes_for_segs(segs);
}

extern "C" HSI_API int hsi_detect(const float* d_score, const int32_t* d_target, int height, int width,
                                  float threshold, int nms_radius, int polarity, int capacity,
                                  hsi_detection* d_out, uint32_t* d_count, void* d_workspace,
                                  size_t workspace_bytes, hsi_stream_t stream) {
  hsi_detect_job j;
  j.score = d_score;
  j.target = d_target;
  j.height = height;
  j.width = width;
  j.threshold = threshold;
  j.nms_radius = nms_radius;
  j.polarity = polarity;
  j.capacity = capacity;
  j.out = d_out;
  j.count = d_count;
  return run_batch(&j, 1, d_workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" HSI_API int hsi_detect_batch(const hsi_detect_job* jobs, int num_jobs, void* d_workspace,
                                        size_t workspace_bytes, hsi_stream_t stream) {
  return run_batch(jobs, num_jobs, d_workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}

// ---- allocation-free detection ------------------------------------------------
//
// For callers that cannot allocate device memory at all -- for example a
// plug-in that a host application hands only its input and output buffers,
// while the application owns every byte of device memory and lets nothing
// else call cudaMalloc -- hsi_detect_noalloc runs the same launches as
// hsi_detect with its scratch in the file-scope array below instead of a
// caller workspace.  The array is part of the library's device image, so
// every GPU that loads the library holds it (2.06 MiB) until the process
// exits, and every call on one device shares it.
namespace hsi_b200 {
namespace {

constexpr int kNoAllocSegs = HSI_DETECT_NOALLOC_MAX_SEGMENTS;
constexpr size_t kNoAllocBytes = static_cast<size_t>(kNoAllocSegs) * sizeof(uint32_t) * (2 + kWordsPerSeg) + 256;

// Segment counts, the map's offset and ballot masks of one call.  Every word a
// call reads is written earlier by that same call (flags writes the counts, the
// map's offset and every mask word that covers pixels of the map, and emit reads
// no other; maps of this size have no scan launch), so nothing here needs to
// start at zero and stale contents from a previous call are never read.
static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocBytes / sizeof(uint32_t)];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
struct NoAllocAddr {
  unsigned long long context;  // the context the address belongs to (0 = none yet)
  void* addr;                  // device address of the array in that context
};
NoAllocAddr g_noalloc_addr[kNoAllocMaxDevices];

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// Process-unique id of the current context.  A device reset (or any other
// re-creation of the context) reloads the module, so the array may move; the
// id changes with it, where a context handle could be reused.
int current_context_id(unsigned long long* id) {
  static const CtxGetCurrentFn get_current = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess
               ? reinterpret_cast<CtxGetCurrentFn>(p)
               : nullptr;
  }();
  static const CtxGetIdFn get_id = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess
               ? reinterpret_cast<CtxGetIdFn>(p)
               : nullptr;
  }();
  if (!get_current || !get_id) return HSI_E_NO_DEVICE;
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return HSI_E_NO_DEVICE;
  return get_id(ctx, id) == CUDA_SUCCESS ? HSI_OK : HSI_E_NO_DEVICE;
}

// Once per device (and again whenever that device's context is re-created),
// with the device current: look up the array's device address (in host code
// its name is only a host-side stand-in).
int noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kNoAllocMaxDevices) return HSI_E_NO_DEVICE;
  unsigned long long ctx = 0;
  if (current_context_id(&ctx) != HSI_OK) {
    // no context is current before the runtime's first call on this thread:
    // the symbol lookup makes the device's primary context current
    void* addr = nullptr;
    e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    const int st = current_context_id(&ctx);
    if (st != HSI_OK) return st;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  NoAllocAddr& a = g_noalloc_addr[dev];
  if (a.addr == nullptr || a.context != ctx) {
    void* addr = nullptr;
    e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    if ((reinterpret_cast<uintptr_t>(addr) & 255u) != 0) return HSI_E_INVALID;
    a.addr = addr;
    a.context = ctx;
  }
  *out = a.addr;
  return HSI_OK;
}

}  // namespace
}  // namespace hsi_b200

extern "C" HSI_API int hsi_detect_noalloc(const float* d_score, const int32_t* d_target, int height, int width,
                                          float threshold, int nms_radius, int polarity, int capacity,
                                          hsi_detection* d_out, uint32_t* d_count, hsi_stream_t stream) {
  if (height <= 0 || width <= 0) return HSI_E_INVALID;
  const int64_t segs = static_cast<int64_t>(height) * ((static_cast<int64_t>(width) + kSeg - 1) / kSeg);
  if (segs > kNoAllocSegs) return HSI_E_CAPACITY;
  void* scratch = nullptr;
  const int st = noalloc_scratch(&scratch);
  if (st != HSI_OK) return st;
  hsi_detect_job j;
  j.score = d_score;
  j.target = d_target;
  j.height = height;
  j.width = width;
  j.threshold = threshold;
  j.nms_radius = nms_radius;
  j.polarity = polarity;
  j.capacity = capacity;
  j.out = d_out;
  j.count = d_count;
  return run_batch(&j, 1, scratch, kNoAllocBytes, reinterpret_cast<cudaStream_t>(stream));
}
