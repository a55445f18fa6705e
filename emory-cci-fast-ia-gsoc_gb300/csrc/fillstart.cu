// Grayscale hole filling: a start near the end.
//
// The fill is the erosion reconstruction of (image on the border, max inside).  Started from that
// marker, a front crosses the whole image tile by tile, and on a noisy image the time is that chain
// of dependent tile visits (16384^2 u8: 14.4 ms, 3% of the copy bandwidth).  But any start between the
// marker and the result gives the same result, and on an image with few grey levels most of the result
// is known early: away from the border a pixel fills to the larger of its own value and the level at
// which the image conducts from the border to it.  So:
//   (1) the lowest level at which a 64 x 64 crop is crossed from left to right is found for 12 x 12 crops
//       (conducting levels), and from them, by the cheapest way over neighbouring crops, the level at
//       which each crop is reached from the left or the right border (reaching levels);
//   (2) levels around the median reaching level are tried in rising order: the pixels at or below the
//       level are labelled (union-find: no chain) and the components that touch the border are marked.
//       No further level is tried once these hold half of the pixels at or below it on a grid over the
//       image's inner half;
//   (3) the start is the lowest level tried at which a pixel is marked (it is joined to a border
//       pixel through pixels at or below the level, so its result is at most the level), and the
//       marker elsewhere.
// The reconstruction then only works near the border and in closed pockets.
//
// A level above the right one would leave the whole chain to do, and a level below it marks nothing, so
// images without a level of their own have to be told from the others before anything is labelled.
// The start is the plain marker when
//   - the crops have no level (most pixels differ from all others), or the reaching levels are spread
//     over many values (a slope, a vignette, a noise of many levels);
//   - a band of rows across the image's middle, labelled first, is not reached from its ends (a wall
//     that no crop saw).
//
// What is tried is decided on the device, so every launch is made for every image.  The kernels of a level
// that is not tried read one word and return: 52 us a level at 16384^2, 18 at 4096^2 (205 with a labelling
// tile to a warp and a word read by every warp).  Whole fill of u8 images, 4-connected, at 16384^2, 4096^2 and
// 1500 x 1400, in ms from the plain front, and with this start:
//   31 noise levels around dark objects     14.9  3.04 0.66    4.9  0.68 0.36
//   dark noise, bright border of a pixel     3.2  0.55 0.23    2.0  0.28 0.14
//   dark noise in a bright noisy surround    4.2  0.64 0.28    2.9  0.55 0.30
//   flat dark ground, bright objects         3.3  0.57 0.24    2.0  0.30 0.16
//   noise that rises along the image        11.0  1.46 0.68   10.1  1.33 0.63   (no level: plain marker)
//   closed wall 200 px in                    3.3  0.59 0.39    2.7  0.63 0.36   (found by the band)
// The plain marker itself is written four pixels at a time, which pays for the estimate (the front took
// these times with a pixel at a time); the wall at 4096^2 is the one kind found where that is not enough.
#include "fillstart.cuh"

#include <limits.h>
#include <stdint.h>

#include <algorithm>
#include <limits>
#include <type_traits>

#include "../../include/nsgb.h"
#include "common.cuh"
#include "launch.cuh"

namespace nsgb {

namespace {

constexpr int kCropThreads = 512, kCropWarps = kCropThreads / 32;
constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kCropGrid = 12, kCrops = kCropGrid * kCropGrid, kCrop = 64;
constexpr int kTries = 3;
constexpr int kCheckGrid = 64;   // check points per side
constexpr int kCheckCtas = kCheckGrid * kCheckGrid / kThreads;
static_assert(kCheckGrid * kCheckGrid % kThreads == 0, "whole CTAs");
constexpr int kBandRows = 1024;  // rows of the band, at most an eighth of the image's
constexpr int kUnitRows = 4;     // rows of 128 columns: what a warp writes of the start, or a multiple
// Smaller sides keep the plain marker: 1024^2 u8 noise takes 0.61 ms from it and 0.59 from an estimated
// start, 1300^2 u16 0.93 and 0.61, 768^2 u8 0.41 and 0.50 (measured with an estimate of 0.1 ms; this one
// takes 0.035).
constexpr int kMinSide = 1280;
constexpr int64_t kSmallPx = 1 << 23;
constexpr int kTilesPerRound = 1 << 16;  // labelling tiles for each round of a CTA: eight full loads of the device

// What is labelled: the image at level 0 .. kTries - 1, or the band at the highest of them.
constexpr int kBand = kTries;

// All zero before the first launch.
struct FillCtl {
  int go[kTries + 1];       // label it
  int level[kTries + 1];
  int n, expected;          // levels, and which of them is expected to conduct
  int low[kTries + 1];      // check points at or below the level
  int joined[kTries + 1];   // ... of them joined to the border
  int checked[kTries + 1];  // CTAs that have counted theirs
  int crops_done;
  int crop[kCrops];         // conducting levels
};
static_assert(sizeof(FillCtl) <= kFillCtlBytes, "control words");

// One load per CTA: a load per warp of a launch that has nothing to do, all of one word, took 10 us.
__device__ __forceinline__ bool active(const FillCtl* c, int k) {
  return __syncthreads_or(threadIdx.x == 0 && __ldcg(&c->go[k]) != 0);
}

template <typename T>
struct alignas(4 * sizeof(T)) Quad {
  T v[4];
};

template <typename T>
__device__ __forceinline__ const T* row_of(const Img& m, int y) {
  return (const T*)((const char*)m.plane + (int64_t)y * m.pitch);
}
template <typename T>
__device__ __forceinline__ int value(const Img& m, int y, int x) {
  return (int)__ldg(row_of<T>(m, y) + x);
}

template <typename T>
struct AtMost {
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  int level;
  __device__ uint32_t operator()(const Img& m, int y, int x) const { return value<T>(m, y, x) <= level ? 1u : 0u; }
};

__device__ __forceinline__ uint64_t shfl64(uint64_t v, int lane) {
  const uint32_t lo = __shfl_sync(NSGB_FULL, (uint32_t)v, lane), hi = __shfl_sync(NSGB_FULL, (uint32_t)(v >> 32), lane);
  return ((uint64_t)hi << 32) | lo;
}

// The runs of `open` that hold a bit of `seed` (seed within open): a carry runs through a run upwards,
// and through its mirror image downwards.
__device__ __forceinline__ uint64_t runs_of(uint64_t seed, uint64_t open, uint64_t mirror) {
  seed |= ((open + seed) ^ open) & open;
  const uint64_t back = __brevll(seed);
  return __brevll(back | (((mirror + back) ^ mirror) & mirror));
}

// Is the crop crossed from left to right by pixels at or below t?  One warp, lane = rows l and l + 32.
// best: the crop's largest value at or below t (INT_MIN if there is none).
template <int CONN>
__device__ __forceinline__ bool crossed(const int* v, int t, int& best) {
  const int lane = threadIdx.x & 31;
  uint64_t open[2], rev[2], at[2];
  int top = INT_MIN;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int* row = v + (lane + 32 * h) * (kCrop + 1);
    uint32_t w[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll 8
      for (int x = 0; x < 32; ++x) {
        const int p = row[32 * k + x];
        if (p <= t) {
          w[k] |= 1u << x;
          top = max(top, p);
        }
      }
    }
    open[h] = ((uint64_t)w[1] << 32) | w[0];
    rev[h] = __brevll(open[h]);
    at[h] = runs_of(open[h] & 1ull, open[h], rev[h]);
  }
  best = __reduce_max_sync(NSGB_FULL, top);
  for (int it = 0; it < kCrop * kCrop; it += 2) {
    if (__any_sync(NSGB_FULL, ((at[0] | at[1]) >> (kCrop - 1)) != 0ull)) return true;
    const uint64_t before0 = at[0], before1 = at[1];
#pragma unroll
    for (int step = 0; step < 2; ++step) {
      const int up = (lane + 31) & 31, down = (lane + 1) & 31;
      const uint64_t u0 = shfl64(at[0], up), u1 = shfl64(at[1], up);
      const uint64_t d0 = shfl64(at[0], down), d1 = shfl64(at[1], down);
      uint64_t n0 = lane == 0 ? d0 : lane == 31 ? u0 | d1 : u0 | d0;  // row 32 is lane 0's second
      uint64_t n1 = lane == 0 ? u0 | d1 : lane == 31 ? u1 : u1 | d1;  // row 31 is lane 31's first
      if (CONN == 8) {
        n0 |= (n0 << 1) | (n0 >> 1);
        n1 |= (n1 << 1) | (n1 >> 1);
      }
      at[0] = runs_of(at[0] | (n0 & open[0]), open[0], rev[0]);
      at[1] = runs_of(at[1] | (n1 & open[1]), open[1], rev[1]);
    }
    if (!__any_sync(NSGB_FULL, at[0] != before0 || at[1] != before1)) return false;
  }
  return false;
}

// The conducting level of crop k, by the whole CTA: sixteen levels at a time, first those of the middle of
// the crop's values (in noise that settles it), then evenly between the highest that is not crossed and the
// lowest that is.  kNone: most of its pixels differ, or four rounds do not settle it.
constexpr int kNone = INT_MAX;
template <typename T, int CONN>
__device__ __forceinline__ int crop_level(const Img& m, int k, int* v) {
  constexpr int kSample = 128;
  __shared__ int s_min, s_max, s_lo, s_hi, s_below, s_sorted[kSample];
  const int t = threadIdx.x, warp = t >> 5;
  const int y0 = (int)(((int64_t)(m.H - kCrop) * (k / kCropGrid)) / (kCropGrid - 1));
  const int x0 = (int)(((int64_t)(m.W - kCrop) * (k % kCropGrid)) / (kCropGrid - 1));
  if (t == 0) s_min = INT_MAX, s_max = INT_MIN;
  __syncthreads();
  int lo = INT_MAX, hi = INT_MIN;
#pragma unroll
  for (int q = 0; q < kCrop * kCrop / kCropThreads; ++q) {
    const int y = q * (kCropThreads / kCrop) + t / kCrop, x = t % kCrop;
    const int p = value<T>(m, y0 + y, x0 + x);
    v[y * (kCrop + 1) + x] = p;
    lo = min(lo, p);
    hi = max(hi, p);
  }
  lo = __reduce_min_sync(NSGB_FULL, lo);
  hi = __reduce_max_sync(NSGB_FULL, hi);
  if ((t & 31) == 0) {
    atomicMin(&s_min, lo);
    atomicMax(&s_max, hi);
  }
  __syncthreads();
  if (sizeof(T) > 1) {
    bool first = t < 256;
    const int own = v[(t & 255) / 4 * (kCrop + 1) + 16 * (t & 3)];
    for (int j = 0; j < (t & 255) && first; ++j) first = v[j / 4 * (kCrop + 1) + 16 * (j & 3)] != own;
    if (__syncthreads_count(first) > 128) return kNone;
  }
  if (t < kSample) {
    const auto at = [&](int j) { return v[(j / 2) * (kCrop + 1) + 32 * (j & 1) + (7 * j) % 32]; };
    const int own = at(t);
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < kSample; ++j) {
      const int o = at(j);
      rank += o < own || (o == own && j < t);
    }
    s_sorted[rank] = own;
  }
  long long fails = (long long)s_min - 1;
  int crosses = s_max;
  for (int round = 0; round < 4; ++round) {
    // any of the crop's values between the two?
    if (t == 0) s_below = 0, s_lo = INT_MIN, s_hi = crosses;
    __syncthreads();
    bool between = false;
#pragma unroll
    for (int q = 0; q < kCrop * kCrop / kCropThreads; ++q) {
      const int p = v[(q * (kCropThreads / kCrop) + t / kCrop) * (kCrop + 1) + t % kCrop];
      between = between || (p > fails && p < crosses);
    }
    if (!__syncthreads_or(between)) return crosses;
    const long long level = round == 0 ? s_sorted[kSample / 4 + warp * (kSample / 2 / kCropWarps)]
                                       : fails + (((long long)crosses - fails) * (warp + 1)) / (kCropWarps + 1);
    if (level > fails) {  // whole warps
      int best;
      const bool ok = crossed<CONN>(v, (int)level, best);
      if ((t & 31) == 0) {
        if (ok) {
          atomicMin(&s_hi, best);
        } else {
          s_below = 1;
          atomicMax(&s_lo, (int)level);
        }
      }
    }
    __syncthreads();
    crosses = s_hi;
    if (s_below) fails = s_lo;
    __syncthreads();
  }
  return kNone;
}

// The levels to try, `tries` at most, from the crops' conducting levels; one CTA, s: 8 * kCrops words.
// Reaching levels are taken over a crop's eight neighbours and over its four: a level that conducts
// over any distance is crossed in more than half of the crops, between what it takes for most crops to be
// reached over eight neighbours (41%, site percolation) and over four (59%).
__device__ __forceinline__ void choose_levels(int tries, bool probe, FillCtl* c, int* s) {
  int* const own = s;                    // conducting levels
  int* const sorted = s + kCrops;        // ... in order
  int* const distinct = s + 2 * kCrops;  // the different ones
  int* const begin = s + 3 * kCrops;     // ... and the first crop in order of each
  __shared__ unsigned s_new[kCropWarps];
  __shared__ int s_lower, s_middle, s_upper, s_expected;
  const int k = threadIdx.x;
  const bool crop = k < kCrops;
  // threads 0 .. 143: eight neighbours, 256 .. 399: four
  const int nb = k >> 8, i = k & 255;
  const bool on = i < kCrops;
  int* const reach = s + (4 + 2 * nb) * kCrops;  // reaching levels
  int* const order = reach + kCrops;             // ... in order
  const int cy = i / kCropGrid, cx = i - cy * kCropGrid;
  int mine = 0, far = 0;
  if (on) {
    mine = __ldcg(&c->crop[i]);
    if (nb == 0) own[i] = mine;
    reach[i] = far = cx == 0 || cx == kCropGrid - 1 ? mine : INT_MAX;
  }
  if (__syncthreads_count(crop && mine == kNone) > kCrops / 4) return;
  for (int it = 0; it < kCrops; ++it) {
    int r = INT_MAX;
    if (on) {
#pragma unroll
      for (int d = 0; d < 9; ++d) {
        const int y = cy + d / 3 - 1, x = cx + d % 3 - 1;
        if (nb == 1 && (d & 1) == 0 && d != 4) continue;
        if ((unsigned)y < (unsigned)kCropGrid && (unsigned)x < (unsigned)kCropGrid) r = min(r, reach[y * kCropGrid + x]);
      }
      r = max(r, mine);
    }
    const bool lower = on && r < far;
    if (!__syncthreads_or(lower)) break;
    if (lower) reach[i] = far = r;
    __syncthreads();
  }
  if (on) {
    int a = 0, b = 0;
#pragma unroll 8
    for (int j = 0; j < kCrops; ++j) {
      const int o = own[j], r = reach[j];
      a += o < mine || (o == mine && j < i);
      b += r < far || (r == far && j < i);
    }
    if (nb == 0) sorted[a] = mine;
    order[b] = far;
  }
  __syncthreads();
  // rank of every conducting level among the different ones
  const bool fresh = crop && (k == 0 || sorted[k] != sorted[k - 1]);
  const unsigned word = __ballot_sync(NSGB_FULL, fresh);
  if ((k & 31) == 0) s_new[k >> 5] = word;
  __syncthreads();
  int rank = __popc(s_new[k >> 5] & (0xFFFFFFFFu >> (31 - (k & 31)))) - 1, ranks = 0;
  for (int w = 0; w < kCropWarps; ++w) {
    ranks += __popc(s_new[w]);
    if (w < (k >> 5)) rank += __popc(s_new[w]);
  }
  const int* const order8 = s + 5 * kCrops;
  const int* const order4 = s + 7 * kCrops;
  if (fresh) {
    const int v = sorted[k];
    distinct[rank] = v;
    begin[rank] = k;
    if (v == order8[kCrops / 4]) s_lower = rank;
    if (v == order8[kCrops / 2]) s_middle = rank;
    if (v == order8[3 * kCrops / 4]) s_upper = rank;
    if (v == order4[kCrops / 2]) s_expected = rank;
  }
  __syncthreads();
  // One level has to reach most crops: with 31 noise levels the quartiles of the reaching levels lie one
  // level apart at most, with 256 two to four.
  if (k != 0 || order4[kCrops / 2] == kNone || s_upper - s_middle > 1 || s_upper - s_lower > 2 ||
      s_expected - s_middle > 1)
    return;
  // The level below the one that conducts is tried first although it does not reach the middle: what it
  // marks starts lower, and without it the front near the border is the whole chain again (4096^2 i32,
  // 8-connected, a level that reaches none of the inner half: 3.5 ms without, 1.3 with it).  The level
  // above the expected one is for an estimate that falls just short; one that few crops hold is a wall's.
  int n = 0;
  for (int r = s_expected - s_lower < tries ? s_lower : s_expected; r < ranks && r <= s_expected + 1 && n < tries; ++r) {
    const int held = (r + 1 < ranks ? begin[r + 1] : kCrops) - begin[r];
    if (distinct[r] == kNone || (r > s_expected && held < kCrops / 8)) continue;
    if (r == s_expected) c->expected = n;
    c->level[n++] = distinct[r];
  }
  if (n == 0) return;
  c->n = n;
  c->level[kBand] = c->level[n - 1];
  c->go[probe ? kBand : 0] = 1;
}

// The crops' conducting levels, one CTA each; the last CTA to finish chooses the levels.
template <typename T, int CONN>
__global__ void __launch_bounds__(kCropThreads) crop_kernel(const __grid_constant__ Img m, int tries, bool probe,
                                                            ccl::Forest f, FillCtl* c) {
  __shared__ int s[kCrop * (kCrop + 1)];
  static_assert(kCrop * (kCrop + 1) >= 8 * kCrops && kCrops <= 256 && kCropThreads >= 512, "choose_levels");
  if (blockIdx.x == 0 && threadIdx.x == 0) *f.nroots = 0;
  const int level = crop_level<T, CONN>(m, blockIdx.x, s);
  bool last = false;
  if (threadIdx.x == 0) {
    c->crop[blockIdx.x] = level;
    __threadfence();
    last = atomicAdd(&c->crops_done, 1) == kCrops - 1;
    __threadfence();
  }
  if (__syncthreads_or(last)) choose_levels(tries, probe, c, s);
}

// Local pass of labelling `k`.  A CTA takes `per` rounds of tiles that follow one another.
template <typename T, int CONN>
__global__ void __launch_bounds__(32 * ccl::kLocalWarps)
    local_kernel(const __grid_constant__ Img m, int ntiles, int per, int k, ccl::Forest f, const FillCtl* c) {
  pdl_wait();
  pdl_release();
  if (!active(c, k)) return;
  __shared__ int s_nodes[ccl::kLocalWarps][ccl::kTile * ccl::kTile];
  __shared__ unsigned s_starts[ccl::kLocalWarps][ccl::kTile];
  const AtMost<T> cls{__ldcg(&c->level[k])};
  const int warp = threadIdx.x >> 5;
  for (int i = 0; i < per; ++i) {
    const int b = (blockIdx.x * per + i) * ccl::kLocalWarps + warp;
    if (b >= ntiles) break;
    ccl::local_tile<AtMost<T>, CONN>(cls, ccl::tile_in(m, b), f, s_nodes[warp], s_starts[warp]);
    __syncwarp();
  }
}

// Edge merge of labelling `k`; its bits are cleared on the way.
template <typename T, int CONN>
__global__ void __launch_bounds__(kThreads) merge_kernel(const __grid_constant__ Img m, int ntiles, int per, int k,
                                                         ccl::Forest f, unsigned* bits, int words, const FillCtl* c) {
  pdl_wait();
  pdl_release();
  if (!active(c, k)) return;
  const AtMost<T> cls{__ldcg(&c->level[k])};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) bits[i] = 0u;
  for (int i = 0; i < per; ++i) {
    const int e = (blockIdx.x * per + i) * kWarps + (threadIdx.x >> 5);
    if (e >= 2 * ntiles) break;
    ccl::merge_edge<AtMost<T>, CONN>(cls, ccl::tile_in(m, e >> 1), f.L, (e & 1) == 0);
    __syncwarp();
  }
}

// Marks the roots of the components that touch the image's border (the band: its two ends), and
// points the local roots at them (the band is too small for that to pay).
template <typename T>
__global__ void __launch_bounds__(kThreads) mark_kernel(const __grid_constant__ Img m, int k, ccl::Forest f, unsigned* bits,
                                                        const FillCtl* c) {
  pdl_wait();
  pdl_release();
  if (!active(c, k)) return;
  const AtMost<T> cls{__ldcg(&c->level[k])};
  if (k != kBand) ccl::flatten_roots(f, m.H * m.W);
  const int per = k == kBand ? 2 * m.H : 2 * m.W + 2 * m.H;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < per; i += gridDim.x * kThreads) {
    int y, x;
    if (k == kBand) y = i >> 1, x = i & 1 ? m.W - 1 : 0;
    else ccl::border_pixel(i, m.H, m.W, y, x);
    if (!cls(m, y, x)) continue;
    const int r = ccl::g_find(f.L, y * m.W + x);
    if (r >= 0) ccl::set_root_bit(bits, r);
  }
}

// Points of a grid over rows y0 .. y0 + rows and the inner half of the columns: how many are at or
// below the level, and how many of these are marked.  The last CTA to count its points decides what is
// labelled next.
template <typename T>
__device__ __forceinline__ void check_points(const Img& m, int k, const ccl::Forest& f, const unsigned* bits, int level,
                                             int y0, int rows, FillCtl* c) {
  if (blockIdx.x >= kCheckCtas) return;
  const int i = blockIdx.x * kThreads + threadIdx.x, gy = i / kCheckGrid, gx = i - gy * kCheckGrid;
  const int y = y0 + (int)(((int64_t)rows * gy) / kCheckGrid);
  const int x = m.W / 4 + (int)(((int64_t)(m.W / 2) * gx) / kCheckGrid);
  const bool in = value<T>(m, y, x) <= level;
  const int r = in ? ccl::g_find(f.L, y * m.W + x) : -1;
  const bool mark = r >= 0 && ((__ldcg(bits + (r >> 5)) >> (r & 31)) & 1u);
  const int a = __syncthreads_count(in), b = __syncthreads_count(mark);
  if (threadIdx.x != 0) return;
  atomicAdd(&c->low[k], a);
  atomicAdd(&c->joined[k], b);
  __threadfence();
  if (atomicAdd(&c->checked[k], 1) != kCheckCtas - 1) return;
  __threadfence();
  const int low = __ldcg(&c->low[k]), joined = __ldcg(&c->joined[k]);
  *f.nroots = 0;
  if (k == kBand) {
    c->go[0] = 8 * joined >= low;
  } else if (k + 1 < __ldcg(&c->n)) {
    // not when this level conducts, nor when it should have and marks next to nothing (unless the band says
    // that the highest level does)
    c->go[k + 1] = low == 0 || (2 * joined < low && (k < __ldcg(&c->expected) || 16 * joined >= low || __ldcg(&c->go[kBand])));
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) band_check_kernel(const __grid_constant__ Img m, ccl::Forest f,
                                                              const unsigned* bits, FillCtl* c) {
  pdl_wait();
  pdl_release();
  if (active(c, kBand)) check_points<T>(m, kBand, f, bits, __ldcg(&c->level[kBand]), 0, m.H, c);
}

// The start on this thread's four columns of rows y0 .. y1: the image on the border, max elsewhere,
// and `level` on the marked pixels.  JOINED: labels and bits are this level's; add: the plane holds the
// starts of lower levels already.
// Bound: the latency of three dependent loads a quad (label, root, bit).  The loads of each step are
// unconditional (clamped) so that they go out together, and a warp takes consecutive rows, so that
// the rows of a labelling tile find its roots in L1 (16384^2 u8, a noisy level: 635 us with neither,
// 378 with both).
template <typename T, bool JOINED>
__device__ __forceinline__ void write_rows(const Img& m, const int* L, const unsigned* bits, T* out, int level, bool add,
                                           int x, int y0, int y1) {
  constexpr T kMax = std::numeric_limits<T>::max();
  if (x >= m.W) return;
  const int n = min(4, m.W - x);
#pragma unroll 2
  for (int y = y0; y < y1; ++y) {
    const T* in = row_of<T>(m, y) + x;
    T* o = (T*)((char*)out + (int64_t)y * m.pitch) + x;
    const bool vec = n == 4 && ((uintptr_t)o & (4 * sizeof(T) - 1)) == 0;
    T v[4] = {kMax, kMax, kMax, kMax};
    if (JOINED && add) {
      if (vec) {
        const Quad<T> q = *(const Quad<T>*)o;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = q.v[k];
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = k < n ? o[k] : kMax;
      }
      if (v[0] != kMax && v[1] != kMax && v[2] != kMax && v[3] != kMax) continue;
    }
    if (JOINED) {
      int l[4], r[4];
      unsigned word[4];
      const int64_t i = (int64_t)y * m.W + x;
      if (n == 4 && (i & 3) == 0) {
        const int4 q = *(const int4*)(L + i);
        l[0] = q.x, l[1] = q.y, l[2] = q.z, l[3] = q.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) l[k] = k < n ? L[i + k] : -1;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) r[k] = L[max(l[k], 0)];
#pragma unroll
      for (int k = 0; k < 4; ++k) word[k] = bits[max(r[k], 0) >> 5];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (l[k] >= 0 && ((word[k] >> (r[k] & 31)) & 1u) && v[k] == kMax) v[k] = (T)level;
    }
    if (!JOINED || !add) {
      if (y == 0 || y == m.H - 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < n) v[k] = in[k];
      } else {
        if (x == 0) v[0] = in[0];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (x + k == m.W - 1) v[k] = in[k];
      }
    }
    if (vec) {
      *(Quad<T>*)o = Quad<T>{v[0], v[1], v[2], v[3]};
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n) o[k] = v[k];
    }
  }
}

// A warp's share of the plane: `per` stacked units of kUnitRows rows x 128 columns.
template <typename T, bool JOINED>
__device__ __forceinline__ void write_start(const Img& m, const int* L, const unsigned* bits, T* out, int level, bool add,
                                            int per) {
  const int nx = (m.W + 127) / 128;
  const int64_t u = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int yb = (int)(u / nx), xb = (int)(u - (int64_t)yb * nx);
  const int64_t y0 = (int64_t)yb * per * kUnitRows;
  if (y0 < m.H)
    write_rows<T, JOINED>(m, L, bits, out, level, add, 128 * xb + 4 * (threadIdx.x & 31), (int)y0,
                          (int)min((int64_t)m.H, y0 + per * kUnitRows));
}

// The start with level k added, and whether that level conducts.  Level 0 writes the whole plane: the
// plain marker if no level is tried.
template <typename T>
__global__ void __launch_bounds__(kThreads) level_kernel(const __grid_constant__ Img m, int per, int k, ccl::Forest f,
                                                         const unsigned* bits, T* out, FillCtl* c) {
  pdl_wait();
  pdl_release();
  if (!active(c, k)) {
    if (k == 0) write_start<T, false>(m, nullptr, nullptr, out, 0, false, per);
    return;
  }
  const int level = __ldcg(&c->level[k]);
  check_points<T>(m, k, f, bits, level, m.H / 4, m.H / 2, c);
  write_start<T, true>(m, f.L, bits, out, level, k > 0, per);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) plain_start_kernel(const __grid_constant__ Img m, int per, T* out) {
  write_start<T, false>(m, nullptr, nullptr, out, 0, false, per);
}

// CTAs of write_start, `per` units to a warp.
unsigned writer_ctas(const Img& m, int per) {
  const int64_t units = (int64_t)((m.W + 127) / 128) * ((m.H + (int64_t)per * kUnitRows - 1) / (per * kUnitRows));
  return (unsigned)((units + kWarps - 1) / kWarps);
}

template <typename T>
cudaError_t plain_start(const Img& m, T* out, cudaStream_t s) {
  plain_start_kernel<T><<<writer_ctas(m, 1), kThreads, 0, s>>>(m, 1, out);
  return cudaGetLastError();
}

template <typename T, int CONN>
cudaError_t level_start(const Img& m, int c_tiles, const ccl::Forest& f, unsigned* bits, int words, FillCtl* c, T* out,
                        cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(c, 0, sizeof(FillCtl), s);
  if (e != cudaSuccess) return e;
  // Small images: no band, since labelling the whole costs little more (4096^2 u8: band 60 us, level 210).
  const bool probe = (int64_t)m.H * m.W > kSmallPx;
  const int tries = probe ? kTries : kTries - 1;
  crop_kernel<T, CONN><<<kCrops, kCropThreads, 0, s>>>(m, tries, probe, f, c);
  e = cudaGetLastError();
  const auto label = [&](const Img& img, int tiles, int nwords, int k) {
    // rounds per CTA: large images have fewer CTAs, which a level that is not tried starts for nothing
    // (16384^2, local pass: 65536 CTAs take 1.20 ms, or 68 us to return at once; 16384 of four rounds 1.24
    // ms or 18 us; 1976 that take tiles in turn 1.42 ms)
    const int per = std::min(8, std::max(1, tiles / kTilesPerRound));
    const int warps = per * ccl::kLocalWarps, edges = per * kWarps;
    if (e == cudaSuccess)
      e = launch_dependent(local_kernel<T, CONN>, dim3((unsigned)((tiles + warps - 1) / warps)),
                           dim3(32 * ccl::kLocalWarps), s, img, tiles, per, k, f, (const FillCtl*)c);
    if (e == cudaSuccess)
      e = launch_dependent(merge_kernel<T, CONN>, dim3((unsigned)((2 * (int64_t)tiles + edges - 1) / edges)),
                           dim3(kThreads), s, img, tiles, per, k, f, bits, nwords, (const FillCtl*)c);
    if (e == cudaSuccess)
      e = launch_dependent(mark_kernel<T>, dim3(ccl::list_grid((int64_t)img.H * img.W)), dim3(kThreads), s, img, k, f,
                           bits, (const FillCtl*)c);
  };
  if (probe) {
    Img band = m;
    band.H = std::min(kBandRows, m.H / 8) & ~(ccl::kTile - 1);
    band.plane = (char*)m.plane + (int64_t)((m.H - band.H) / 2) * m.pitch;
    label(band, m.c_tiles_x * (band.H / ccl::kTile), (int)(((int64_t)band.H * band.W + 31) / 32), kBand);
    if (e == cudaSuccess)
      e = launch_dependent(band_check_kernel<T>, dim3(kCheckCtas), dim3(kThreads), s, band, f, (const unsigned*)bits, c);
  }
  const int per = c_tiles >= kTilesPerRound ? 8 : probe ? 4 : 1;
  const dim3 writers(std::max(writer_ctas(m, per), (unsigned)kCheckCtas));
  for (int k = 0; k < tries; ++k) {
    label(m, c_tiles, words, k);
    if (e == cudaSuccess)
      e = launch_dependent(level_kernel<T>, writers, dim3(kThreads), s, m, per, k, f, (const unsigned*)bits, out, c);
  }
  return e;
}

template <typename T>
cudaError_t start_typed(const Imgs& I, int c_tiles, const ccl::Forest& f, unsigned* bits, size_t bits_bytes, void* ctl,
                        void* out, int conn, cudaStream_t s) {
  const Img& m = I.one;
  if constexpr (std::is_integral<T>::value) {
    if (m.H >= kMinSide && m.W >= kMinSide) {
      const int words = (int)(bits_bytes / sizeof(unsigned));
      return conn == 8 ? level_start<T, 8>(m, c_tiles, f, bits, words, (FillCtl*)ctl, (T*)out, s)
                       : level_start<T, 4>(m, c_tiles, f, bits, words, (FillCtl*)ctl, (T*)out, s);
    }
  }
  return plain_start<T>(m, (T*)out, s);
}

}  // namespace

cudaError_t fill_start_launch(int dtype, const Imgs& I, int c_tiles, const ccl::Forest& f, unsigned* bits,
                              size_t bits_bytes, void* ctl, void* out, int conn, cudaStream_t s) {
  switch (dtype) {
    case NSGB_U8: return start_typed<uint8_t>(I, c_tiles, f, bits, bits_bytes, ctl, out, conn, s);
    case NSGB_U16: return start_typed<uint16_t>(I, c_tiles, f, bits, bits_bytes, ctl, out, conn, s);
    case NSGB_I32: return start_typed<int32_t>(I, c_tiles, f, bits, bits_bytes, ctl, out, conn, s);
    case NSGB_F32: return start_typed<float>(I, c_tiles, f, bits, bits_bytes, ctl, out, conn, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace nsgb
