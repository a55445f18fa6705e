// Euclidean distance transform of a u8 mask: for every pixel the distance to the nearest zero
// pixel (0 on zero pixels), the map the segmentation takes before its watershed
// (HistologicalEntities.cpp:341, OpenCV's CV_DIST_L2 / CV_DIST_MASK_PRECISE; the reference's own
// queue version is nscale::distanceTransform, MorphologicOperations.cpp:197-275, GPU
// nscale::gpu::distanceTransform, cuda/global_queue_dist.cu).  Exact: the squared distance is an
// integer, and the float result is the correctly rounded square root of it.  The reference's
// queue version propagates nearest zero pixels between 8-neighbours, which can settle on a zero
// pixel that is not the nearest; it is never closer than the exact distance.
//
// Near pass: one bit per pixel says where the zero pixels are, as 32-row column words
// (edt_zero_words).  A CTA takes a tile of 32 rows x 128 columns with 32 columns on either side,
// walks every column down and up through its word and the ones above and below it, and keeps the
// squared row distances of two rows in one 32-bit word of shared memory.  Each pixel then takes
// the minimum of k^2 + g(x +- k)^2 outward from its column, two rows at a time (min.u16x2 with
// three operands), until k^2 reaches both minima.  A squared distance of at most 32^2 found there
// is exact: no zero pixel further than 32 rows or columns away could be nearer.  Rows that hold a
// pixel further away are marked and done again by the far pass.
//   Bound: instructions issued (about 1.3 a pixel) beside the 5 bytes of a pixel.  4096^2 with
//   objects of tens of pixels: 58 us (the far pass, which used to do every row: 179 us).  A mask
//   whose rows are all marked takes both passes: with one zero per 100 x 100 pixels at 4096^2 it is
//   1020 us (1013 with the far pass alone; 1221 when the near pass stored a mark for every far pixel).
//
// Far pass, marked rows only (Meijster, Roerdink and Hesselink, 2000):
// (1) per column, the distance in rows to the nearest zero pixel of that column, g (INF when the
//     column has none; INF = rows + cols exceeds every real distance), from the same words.  Columns
//     are cut into 128-row chunks: one launch records each chunk's first and last zero row, the next
//     finds for each marked row the nearest zero rows within its word, its chunk or the chunks above
//     and below (threads of a warp take adjacent columns, so g is written coalesced);
// (2) per row, D^2(x) = min over x' of (x - x')^2 + g(x')^2, one CTA per row: each pixel that the
//     near pass left searches outward along the row and stops once the column offset alone
//     reaches its best squared distance (at most g(x) columns each way), which is cheap while the
//     row's mean g is small.  A row with a large mean g (far from every zero pixel, or crossing
//     columns without one) is done by the whole CTA by divide and conquer: the
//     matrix (x - i)^2 + g(i)^2 is Monge, so the leftmost minimising column A(x) never
//     decreases with x, and the row minimum at the midpoint of two computed positions a < b
//     only needs the columns A(a) .. A(b).  Level by level (log2 W levels) every position's
//     candidate columns are laid end to end and split evenly over the threads, each keeping
//     one running minimum per position it touches (64-bit keys: D^2 above the column, so
//     atomicMin keeps the leftmost minimum).  Rows wider than the shared-memory tables
//     (12288 columns) fall back to the lower envelope of the parabolas (Meijster) on one
//     thread.  All three are exact integer arithmetic.
// Output: the distance (float), or the basins of the watershed step (HistologicalEntities.cpp:
// 347-356): -distance on mask pixels, -FLT_MAX elsewhere.  No zero pixel at all: +inf.
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "edt.cuh"
#include "launch.cuh"

namespace nsgb {

namespace {

constexpr int kThreads = 64;  // column passes: adjacent columns per block
constexpr int kChunk = 128;   // rows per column chunk

// ---- Near pass.

constexpr int kNear = 32;       // rows of a tile and of a word; columns of halo on each side
constexpr int kNearCols = 128;
// Threads of a near tile.  An image of few tiles leaves the device to their latency: there twice the
// threads take half of the rows each (513 x 700 with far pixels all over: 9.9 -> 7.5 us).
constexpr int kNearThreads = 256, kNearThreadsFew = 512, kNearFewTiles = 304;
constexpr uint32_t kNearInf = 60000;  // a squared row distance beyond the near pass; + 32^2 < 2^16

// Words of 32 rows: bit r of words[(y / 32) * W + x] is set where pixel (y + r, x) is zero.  Four
// columns per thread; the four rows of a word's byte by byte: a byte's bits are eight rows.  Clears the
// marks of its rows on the way.
template <bool VEC>
__global__ void __launch_bounds__(128) edt_zero_words(const uint8_t* __restrict__ mask, int64_t pitch, int H, int W,
                                                      uint32_t* __restrict__ words, int* __restrict__ far,
                                                      int* any_far) {
  pdl_release();
  const int per = (W + 511) / 512, c = blockIdx.x / per;
  if ((int)blockIdx.x == c * per && threadIdx.x < kNear && kNear * c + threadIdx.x < H) far[kNear * c + threadIdx.x] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *any_far = 0;
  const int x = 4 * ((blockIdx.x - c * per) * blockDim.x + threadIdx.x);
  if (x >= W) return;
  const int y0 = kNear * c;
  const int last = H - 1 - y0;  // rows past the image repeat the last one; their bits are unused
  uint32_t px[kNear];           // all loads go out before the first is used
#pragma unroll
  for (int r = 0; r < kNear; ++r) {
    const uint8_t* p = mask + (int64_t)(y0 + min(r, last)) * pitch + x;
    if (VEC && x + 4 <= W) {
      px[r] = __ldg((const uint32_t*)p);
    } else {
      px[r] = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) px[r] |= (uint32_t)__ldg(p + min(b, W - 1 - x)) << (8 * b);
    }
  }
  uint32_t rows8[4];  // byte k: eight rows of column x + k
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t acc = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t w = px[8 * q + r];
      // bit 7 of every zero byte
      const uint32_t z = ~(((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
      acc |= z >> (7 - r);
    }
    rows8[q] = acc;
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    if (x + b >= W) break;
    uint32_t v = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) v |= ((rows8[q] >> (8 * b)) & 0xFFu) << (8 * q);
    if (last < kNear - 1) v &= (2u << last) - 1u;
    words[(int64_t)c * W + x + b] = v;
  }
}

__device__ __forceinline__ float near_value(uint32_t d2, bool basins) {
  if (d2 == 0u) return basins ? -FLT_MAX : 0.f;
  const float d = sqrtf((float)d2);
  return basins ? -d : d;
}

// Output of every pixel within 32 of a zero pixel; where a row holds another, its bit in the row's far
// words (W words apart), far[y] and *any_far.  (Marks are collected per CTA: stored by every pixel they were
// 0.2 ms of a 4096^2 mask with most pixels far.)
template <bool BASINS, int THREADS>
__global__ void __launch_bounds__(THREADS) edt_near(const uint32_t* __restrict__ words, int nwords,
                                                         float* __restrict__ out, int64_t pitch_out, int H, int W,
                                                         uint32_t* __restrict__ far_words, int* __restrict__ far,
                                                         int* any_far) {
  pdl_wait();
  pdl_release();
  constexpr int kCols = kNearCols + 2 * kNear;
  __shared__ uint32_t s[kNear / 2][kCols];  // rows 2 j (low half) and 2 j + 1 (high half), squared
  __shared__ int s_far[kNear];
  const int per = (W + kNearCols - 1) / kNearCols, c = blockIdx.x / per;
  const int x0 = (blockIdx.x - c * per) * kNearCols, y0 = c * kNear;
  bool seen = false;
  if (threadIdx.x < kNear) s_far[threadIdx.x] = 0;
  if (threadIdx.x < kCols) {
    const int x = x0 - kNear + threadIdx.x;
    uint32_t z = 0, above = 0, below = 0;
    if (x >= 0 && x < W) {
      z = __ldg(words + (int64_t)c * W + x);
      if (c > 0) above = __ldg(words + (int64_t)(c - 1) * W + x);
      if (c + 1 < nwords) below = __ldg(words + (int64_t)(c + 1) * W + x);
    }
    seen = (z | above | below) != 0u;
    uint32_t g[kNear];
    uint32_t d = above ? (uint32_t)__clz(above) : 4 * kNear;  // rows from the last zero above to row -1
#pragma unroll
    for (int r = 0; r < kNear; ++r) {
      d = (z >> r) & 1u ? 0u : d + 1u;
      g[r] = d;
    }
    d = below ? (uint32_t)__ffs(below) - 1u : 4 * kNear;
#pragma unroll
    for (int r = kNear - 1; r >= 0; --r) {
      d = (z >> r) & 1u ? 0u : d + 1u;
      g[r] = min(g[r], d);
      g[r] = g[r] <= kNear ? g[r] * g[r] : kNearInf;
    }
#pragma unroll
    for (int j = 0; j < kNear / 2; ++j) s[j][threadIdx.x] = g[2 * j] | (g[2 * j + 1] << 16);
  }
  if (!__syncthreads_or(seen)) {  // no zero pixel anywhere near
    if (threadIdx.x < kNear && y0 + threadIdx.x < H) far[y0 + threadIdx.x] = 1;
    if (threadIdx.x == 0) *any_far = 1;
    constexpr int kWords = kNearCols / 32;
    const int y = y0 + threadIdx.x / kWords, x = x0 + 32 * (threadIdx.x % kWords);
    if (threadIdx.x < kNear * kWords && y < H && x < W) far_words[(int64_t)y * W + x / 32] = 0xFFFFFFFFu;
    return;
  }
  const int x = x0 + (threadIdx.x & (kNearCols - 1));
  for (int j = threadIdx.x / kNearCols; j < kNear / 2; j += THREADS / kNearCols) {  // the same for a warp
    const int y = y0 + 2 * j;
    if (y >= H) break;
    const uint32_t* row = s[j] + kNear + (threadIdx.x & (kNearCols - 1));
    uint32_t best = row[0];
    for (int k = 1; k <= kNear; k += 4) {
      if (!((uint32_t)(k * k) < max(best & 0xFFFFu, best >> 16))) break;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t kk = (uint32_t)((k + q) * (k + q)) * 0x10001u;
        best = __vimin3_u16x2(best, row[-(k + q)] + kk, row[k + q] + kk);
      }
    }
    const uint32_t d[2] = {best & 0xFFFFu, best >> 16};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (y + h >= H) break;
      const bool in = x < W, is_far = d[h] > kNear * kNear;
      if (in && !is_far) *((float*)((char*)out + (int64_t)(y + h) * pitch_out) + x) = near_value(d[h], BASINS);
      const unsigned word = __ballot_sync(NSGB_FULL, in && is_far);
      if ((threadIdx.x & 31) == 0 && in) {
        far_words[(int64_t)(y + h) * W + x / 32] = word;
        if (word) s_far[2 * j + h] = 1;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < kNear) {
    const bool mark = s_far[threadIdx.x] != 0;
    if (mark) far[y0 + threadIdx.x] = 1;
    if (__any_sync(NSGB_FULL, mark) && threadIdx.x == 0) *any_far = 1;
  }
}

// ---- Far pass.

constexpr int kChunkWords = kChunk / kNear;

// First and last zero row of every (column, chunk), -1 when none.
__global__ void __launch_bounds__(kThreads) edt_chunk_zeros(const uint32_t* __restrict__ words, int nwords, int W,
                                                            int* __restrict__ first0, int* __restrict__ last0,
                                                            const int* __restrict__ any_far) {
  pdl_wait();
  pdl_release();
  if (*any_far == 0) return;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= W) return;
  const int c = blockIdx.y;
  int f = -1, l = -1;
#pragma unroll
  for (int q = 0; q < kChunkWords; ++q) {
    const int k = c * kChunkWords + q;
    const uint32_t w = k < nwords ? __ldg(words + (int64_t)k * W + x) : 0u;
    if (w) {
      if (f < 0) f = k * kNear + __ffs(w) - 1;
      l = k * kNear + 31 - __clz(w);
    }
  }
  first0[(int64_t)c * W + x] = f;
  last0[(int64_t)c * W + x] = l;
}

// g of one row, `up` and `down` its column's zero pixels of the word at or above and at or below the row.
__device__ __forceinline__ int row_distance(uint32_t up, uint32_t down, int y, int above, int below, int inf) {
  const int du = up ? __clz(up) : above >= 0 ? y - above : inf;
  const int dd = down ? __ffs(down) - 1 : below >= 0 ? below - y : inf;
  return min(du, dd);
}

// g for the marked rows of one (column, chunk), from the words of zero pixels: nearest zero row above and
// below, in the chunk or in the chunks above and below it.  (Walked pixel by pixel down and up, with g
// written, read and written again, this pass took 59 us at 4096^2, and the one before it another 16 MB of
// mask.)
__global__ void __launch_bounds__(kThreads) edt_columns(const uint32_t* __restrict__ words, int nwords, int H, int W,
                                                        const int* __restrict__ first0, const int* __restrict__ last0,
                                                        int* __restrict__ g, const int* __restrict__ far,
                                                        const int* __restrict__ any_far) {
  pdl_wait();
  pdl_release();
  if (*any_far == 0) return;
  const int c = blockIdx.y, nc = gridDim.y, lane = threadIdx.x & 31;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t marked[kChunkWords];  // rows of this chunk that the far pass does
  bool any = false;
#pragma unroll
  for (int q = 0; q < kChunkWords; ++q) {
    const int y = c * kChunk + q * kNear + lane;
    marked[q] = __ballot_sync(NSGB_FULL, y < H && __ldg(far + (y < H ? y : 0)) != 0);
    any = any || marked[q] != 0u;
  }
  if (!any || x >= W) return;
  const int inf = H + W;
  int above = -1, below = -1;  // nearest zero rows outside the chunk
  for (int k = c - 1; k >= 0 && above < 0; --k) above = __ldg(last0 + (int64_t)k * W + x);
  for (int k = c + 1; k < nc && below < 0; ++k) below = __ldg(first0 + (int64_t)k * W + x);
  uint32_t w[kChunkWords];
#pragma unroll
  for (int q = 0; q < kChunkWords; ++q) {
    const int k = c * kChunkWords + q;
    w[q] = k < nwords ? __ldg(words + (int64_t)k * W + x) : 0u;
  }
#pragma unroll
  for (int q = 0; q < kChunkWords; ++q) {
    const int y0 = c * kChunk + q * kNear;
    if (marked[q]) {
      int next = below;  // nearest zero row below the word
#pragma unroll
      for (int p = kChunkWords - 1; p > q; --p)
        if (w[p]) next = c * kChunk + p * kNear + __ffs(w[p]) - 1;
#pragma unroll 8
      for (int r = 0; r < kNear; ++r) {
        if (!((marked[q] >> r) & 1u)) continue;  // the same for a warp
        g[(int64_t)(y0 + r) * W + x] = row_distance(w[q] << (31 - r), w[q] >> r, y0 + r, above, next, inf);
      }
    }
    if (w[q]) above = y0 + 31 - __clz(w[q]);
  }
}

// The same in one launch for images of up to kFewWords words of rows: a thread per (column, word) loads the
// column's words, all at once.  A short image leaves the device to the latency of the two launches above,
// each of few CTAs (513 x 700: 15 us of chunks and columns, this 6).
constexpr int kFewWords = 32;
__global__ void __launch_bounds__(kThreads) edt_columns_few(const uint32_t* __restrict__ words, int nwords, int H, int W,
                                                            int* __restrict__ g, const int* __restrict__ far,
                                                            const int* __restrict__ any_far) {
  pdl_wait();
  pdl_release();
  if (*any_far == 0) return;
  const int c = blockIdx.y, y0 = c * kNear, lane = threadIdx.x & 31;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, xc = min(x, W - 1);
  uint32_t w[kFewWords];
#pragma unroll
  for (int k = 0; k < kFewWords; ++k) w[k] = k < nwords ? __ldg(words + (int64_t)k * W + xc) : 0u;
  const uint32_t marked = __ballot_sync(NSGB_FULL, y0 + lane < H && __ldg(far + min(y0 + lane, H - 1)) != 0);
  if (!marked || x >= W) return;
  int above = -1, below = -1;
  uint32_t own = 0u;
#pragma unroll
  for (int k = 0; k < kFewWords; ++k) {
    if (k < c && w[k]) above = k * kNear + 31 - __clz(w[k]);
    if (k == c) own = w[k];
    if (k > c && w[k] && below < 0) below = k * kNear + __ffs(w[k]) - 1;
  }
  for (uint32_t m = marked; m; m &= m - 1u) {
    const int r = __ffs(m) - 1;
    g[(int64_t)(y0 + r) * W + x] = row_distance(own << (31 - r), own >> r, y0 + r, above, below, H + W);
  }
}

__device__ __forceinline__ int64_t sq(int64_t v) { return v * v; }

// floor(a / b) for b > 0.
__device__ __forceinline__ int64_t floor_div(int64_t a, int64_t b) {
  const int64_t q = a / b;
  return (a % b != 0 && a < 0) ? q - 1 : q;
}

__device__ __forceinline__ float root(int64_t d2) {
  return d2 < (1ll << 24) ? sqrtf((float)d2) : (float)sqrt((double)d2);
}

template <bool BASINS>
__device__ __forceinline__ void store_px(float* o, const uint8_t* mrow, int x, int64_t d2, int64_t inf2) {
  const float d = d2 >= inf2 ? INFINITY : root(d2);
  if (BASINS) o[x] = __ldg(mrow + x) != 0 ? -d : -FLT_MAX;
  else o[x] = d;
}

// One row by the lower envelope of its parabolas (one thread; stacks s, t in the workspace).
template <bool BASINS>
__device__ void envelope_row(const int* __restrict__ gr, int* s, int* t, float* o, const uint8_t* mrow, int W,
                             int64_t inf2) {
  int q = 0;
  s[0] = 0;
  t[0] = 0;
  int64_t gs = sq(__ldg(gr));  // g(s[q])^2
  for (int u = 1; u < W; ++u) {
    const int64_t gu = sq(__ldg(gr + u));
    // pop while the top parabola is above u's at the top's start t[q]
    while (q >= 0 && sq((int64_t)t[q] - s[q]) + gs > sq((int64_t)t[q] - u) + gu) {
      --q;
      if (q >= 0) gs = sq(__ldg(gr + s[q]));
    }
    if (q < 0) {
      q = 0;
      s[0] = u;
      t[0] = 0;
      gs = gu;
    } else {
      // first x at which u's parabola is below s[q]'s: 1 + floor(sep)
      const int64_t sep = floor_div(sq((int64_t)u) - sq((int64_t)s[q]) + gu - gs, 2 * ((int64_t)u - s[q]));
      const int64_t w = 1 + sep;
      if (w < W) {
        ++q;
        s[q] = u;
        t[q] = (int)w;
        gs = gu;
      }
    }
  }
  int64_t gq = sq(__ldg(gr + s[q]));
  for (int x = W - 1; x >= 0; --x) {
    store_px<BASINS>(o, mrow, x, sq((int64_t)x - s[q]) + gq, inf2);
    if (x == t[q] && q > 0) {
      --q;
      gq = sq(__ldg(gr + s[q]));
    }
  }
}

constexpr int kRowThreads = 256;
// A row whose mean g exceeds this takes the divide and conquer instead of the per-pixel search.
constexpr int64_t kMeanG = 32;
// Widest row for the divide and conquer's shared-memory tables (8 bytes per column).
constexpr int kDcMaxW = 12288;

__device__ __forceinline__ int dc_levels(int W) {
  int L = 1;
  while ((1 << L) < W + 1) ++L;
  return L;
}

// Exclusive prefix sum of a[0 .. n) in place by the whole CTA; returns the total.
__device__ int block_exclusive_scan(int* a, int n) {
  __shared__ int s_warp[kRowThreads / 32];
  __shared__ int s_total;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int per = (n + kRowThreads - 1) / kRowThreads;
  const int b = min(n, tid * per), e = min(n, b + per);
  int sum = 0;
  for (int k = b; k < e; ++k) sum += a[k];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(NSGB_FULL, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  int base = 0;
  for (int w = 0; w < wid; ++w) base += s_warp[w];
  if (tid == kRowThreads - 1) s_total = base + incl;
  int run = base + incl - sum;
  for (int k = b; k < e; ++k) {
    const int v = a[k];
    a[k] = run;
    run += v;
  }
  __syncthreads();
  return s_total;
}

// Divide and conquer over the row (see the file comment).  Level l computes the positions
// x = (2k + 1) h - 1, h = 2^(L-1-l), whose neighbours x - h and x + h were computed before (or
// lie outside the row: A = 0 on the left, W - 1 on the right).  Shared memory: A (u16 per
// column), the level's keys (u64 per position) and candidate offsets (int per position + 1).
template <bool BASINS>
__device__ void dc_row(const int* __restrict__ gr, float* o, const uint8_t* mrow, int W, int64_t inf2,
                       unsigned char* smem) {
  uint16_t* A = (uint16_t*)smem;
  const int max_nodes = W / 2 + 1;
  unsigned long long* key = (unsigned long long*)(smem + (((size_t)W * 2 + 15) & ~(size_t)15));
  int* off = (int*)(key + max_nodes);
  const int L = dc_levels(W);
  const int tid = threadIdx.x;
  for (int l = 0; l < L; ++l) {
    const int h = 1 << (L - 1 - l);
    const int n = (W / h + 1) / 2;  // positions of this level inside the row
    for (int k = tid; k < n; k += kRowThreads) {
      const int x = (2 * k + 1) * h - 1;
      const int lo = x - h < 0 ? 0 : A[x - h];
      const int hi = x + h >= W ? W - 1 : A[x + h];
      off[k] = hi - lo + 1;
      key[k] = ~0ull;
    }
    __syncthreads();
    const int total = block_exclusive_scan(off, n);
    if (tid == 0) off[n] = total;
    __syncthreads();
    const int chunk = (total + kRowThreads - 1) / kRowThreads;
    int j = tid * chunk;
    const int end = min(total, j + chunk);
    if (j < end) {
      // the position holding candidate j: the last k with off[k] <= j
      int a = 0, b = n - 1;
      while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (off[m] <= j) a = m;
        else b = m - 1;
      }
      int k = a;
      while (j < end) {
        const int x = (2 * k + 1) * h - 1;
        const int lo = x - h < 0 ? 0 : A[x - h];
        const int stop = min(end, off[k + 1]);
        unsigned long long best = ~0ull;
        for (; j < stop; ++j) {
          const int i = lo + (j - off[k]);
          const unsigned long long d2 = (unsigned long long)(sq((int64_t)x - i) + sq(__ldg(gr + i)));
          const unsigned long long kk = (d2 << 24) | (unsigned long long)i;
          best = kk < best ? kk : best;
        }
        atomicMin(&key[k], best);
        ++k;
      }
    }
    __syncthreads();
    for (int k = tid; k < n; k += kRowThreads) {
      const int x = (2 * k + 1) * h - 1;
      const unsigned long long kk = key[k];
      A[x] = (uint16_t)(kk & 0xFFFFFFull);
      store_px<BASINS>(o, mrow, x, (int64_t)(kk >> 24), inf2);
    }
    __syncthreads();
  }
}

// One CTA per row.  D(x) <= g(x), so a pixel's search along the row stops after at most g(x)
// columns each way (once k^2 reaches the best squared distance so far); when the row's g sum
// keeps that work small (mean g <= kMeanG) all threads search their pixels, otherwise the CTA
// runs the divide and conquer (`dc`: the row fits the shared tables and its squared distances
// fit the 40-bit keys), or one thread builds the row's lower envelope.

template <bool BASINS>
__global__ void __launch_bounds__(kRowThreads) edt_rows(const uint8_t* __restrict__ mask, int64_t pitch_in,
                                                        const int* __restrict__ g, int* __restrict__ stack_s,
                                                        int* stack_t, float* __restrict__ out,
                                                        int64_t pitch_out, int H, int W, bool dc,
                                                        const int* __restrict__ far, const int* __restrict__ any_far) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char dc_smem[];
  __shared__ long long s_sum[kRowThreads / 32];
  if (*any_far == 0) return;
  const int64_t inf2 = sq((int64_t)H + W);
  for (int y = blockIdx.x; y < H; y += gridDim.x) {
    if (__ldg(far + y) == 0) continue;  // the same for the whole CTA
    const int* gr = g + (int64_t)y * W;
    float* o = (float*)((char*)out + (int64_t)y * pitch_out);
    const uint8_t* mrow = mask + (int64_t)y * pitch_in;
    long long sum = 0;
    for (int x = threadIdx.x; x < W; x += kRowThreads) sum += __ldg(gr + x);
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(NSGB_FULL, sum, off);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    long long total = 0;
#pragma unroll
    for (int k = 0; k < kRowThreads / 32; ++k) total += s_sum[k];
    if (total <= kMeanG * W) {
      const int* far_word = stack_t + (int64_t)y * W;  // the near pass's: the other pixels are done
      for (int x = threadIdx.x; x < W; x += kRowThreads) {
        if (!((__ldg(far_word + x / 32) >> (x & 31)) & 1)) continue;
        const int64_t gx = __ldg(gr + x);
        int64_t best = gx * gx;
        for (int64_t k = 1; k < W && k * k < best; ++k) {
          if (x - k >= 0) best = min(best, k * k + sq(__ldg(gr + x - k)));
          if (x + k < W) best = min(best, k * k + sq(__ldg(gr + x + k)));
        }
        store_px<BASINS>(o, mrow, x, best, inf2);
      }
    } else if (dc) {
      dc_row<BASINS>(gr, o, mrow, W, inf2, dc_smem);
    } else if (threadIdx.x == 0) {
      envelope_row<BASINS>(gr, stack_s + (int64_t)y * W, stack_t + (int64_t)y * W, o, mrow, W, inf2);
    }
    __syncthreads();  // s_sum is rewritten for the next row
  }
}

}  // namespace

size_t edt_workspace_bytes(int64_t rows, int64_t cols) {
  const size_t plane = ((size_t)rows * (size_t)cols * sizeof(int) + 255) & ~(size_t)255;
  const size_t chunks = ((size_t)((rows + kChunk - 1) / kChunk) * (size_t)cols * sizeof(int) + 255) & ~(size_t)255;
  return 256 + 3 * plane + 2 * chunks + 256 + sizeof(int) * (size_t)rows;
}

cudaError_t edt_launch(const uint8_t* mask, int64_t pitch_in, float* out, int64_t pitch_out, int rows, int cols,
                       bool basins, void* ws, cudaStream_t s) {
  const size_t plane = ((size_t)rows * (size_t)cols * sizeof(int) + 255) & ~(size_t)255;
  const int nchunks = (rows + kChunk - 1) / kChunk;
  const size_t chunks = ((size_t)nchunks * (size_t)cols * sizeof(int) + 255) & ~(size_t)255;
  char* p = (char*)ws + 256;
  int* g = (int*)p;
  int* st_s = (int*)(p + plane);
  int* st_t = (int*)(p + 2 * plane);
  int* first0 = (int*)(p + 3 * plane);
  int* last0 = (int*)(p + 3 * plane + chunks);
  // The near pass's words live in a plane of the envelope's stacks, which only the far pass uses.
  const int nwords = (rows + kNear - 1) / kNear;
  uint32_t* words = (uint32_t*)st_s;
  int* any_far = (int*)(p + 3 * plane + 2 * chunks);
  int* far = any_far + 64;
  // The far words lie in each row's part of the other stack plane: a row takes either them or the stacks.
  uint32_t* far_words = (uint32_t*)st_t;
  cudaError_t e = cudaSuccess;
  const unsigned wgrid = (unsigned)nwords * (unsigned)((cols + 511) / 512);
  const unsigned ngrid = (unsigned)nwords * (unsigned)((cols + kNearCols - 1) / kNearCols);
  const bool few = ngrid <= kNearFewTiles;
  if ((uintptr_t)mask % 4 == 0 && pitch_in % 4 == 0)
    edt_zero_words<true><<<wgrid, 128, 0, s>>>(mask, pitch_in, rows, cols, words, far, any_far);
  else
    edt_zero_words<false><<<wgrid, 128, 0, s>>>(mask, pitch_in, rows, cols, words, far, any_far);
  e = cudaGetLastError();
  if (e == cudaSuccess)
    e = launch_dependent(few ? (basins ? edt_near<true, kNearThreadsFew> : edt_near<false, kNearThreadsFew>)
                             : (basins ? edt_near<true, kNearThreads> : edt_near<false, kNearThreads>),
                         dim3(ngrid), dim3(few ? kNearThreadsFew : kNearThreads), s, (const uint32_t*)words, nwords, out, pitch_out, rows, cols, far_words, far, any_far);
  const dim3 cgrid((cols + kThreads - 1) / kThreads, nchunks);
  if (nwords <= kFewWords) {
    if (e == cudaSuccess)
      e = launch_dependent(edt_columns_few, dim3(cgrid.x, nwords), dim3(kThreads), s, (const uint32_t*)words, nwords, rows,
                           cols, g, (const int*)far, (const int*)any_far);
  } else {
    if (e == cudaSuccess)
      e = launch_dependent(edt_chunk_zeros, cgrid, dim3(kThreads), s, (const uint32_t*)words, nwords, cols, first0,
                           last0, (const int*)any_far);
    if (e == cudaSuccess)
      e = launch_dependent(edt_columns, cgrid, dim3(kThreads), s, (const uint32_t*)words, nwords, rows, cols,
                           (const int*)first0, (const int*)last0, g, (const int*)far, (const int*)any_far);
  }
  const int rblocks = rows < (1 << 20) ? rows : (1 << 20);
  // divide and conquer: tables fit (u16 columns, 24-bit column field) and 2 (H + W)^2 < 2^40
  const bool dc = cols <= kDcMaxW && (int64_t)rows + cols < (1 << 19);
  const size_t smem = dc ? (((size_t)cols * 2 + 15) & ~(size_t)15) + (size_t)(cols / 2 + 1) * 8 +
                               (size_t)(cols / 2 + 2) * 4
                         : 0;
  const auto rows_kernel = basins ? edt_rows<true> : edt_rows<false>;
  if (e == cudaSuccess && smem > 48 * 1024)
    e = cudaFuncSetAttribute(rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = launch_dependent_smem(rows_kernel, dim3(rblocks), dim3(kRowThreads), smem, s, mask, pitch_in, (const int*)g, st_s,
                              st_t, out, pitch_out, rows, cols, dc, (const int*)far, (const int*)any_far);
  return e;
}

}  // namespace nsgb
