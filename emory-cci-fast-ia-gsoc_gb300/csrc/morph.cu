// Flat grayscale erosion and dilation of u8 images by a k x k structuring element, and the
// opening nscale::morphOpen<unsigned char> builds from them (src/segment/MorphologicOperations.cpp:
// 2459-2493: copyMakeBorder by (k-1)/2 with 255, cv::erode, crop; copyMakeBorder with 0,
// cv::dilate, crop).  OpenCV's erode / dilate take, at (y, x), the min / max of
// src(y + i - bw, x + j - bw) over the element's non-zero (i, j), bw = (k-1)/2 (the element is
// not reflected for the dilation); pixels outside the image read the padding value.
//
// One CTA computes a 128-row x 128-column output tile, four pixels to a 32-bit word, one word
// column per lane, eight rows per warp.  The input rows the tile needs (128 + 2 bw, with 32 columns
// of halo on each side) are staged in shared memory once, padding values filled in; the word at
// any column offset is one funnel shift of two staged words.
//
// Byte-wise min / max is emulated on this device (several instructions per word), 16-bit pairs are
// native (min.u16x2, also with three operands).  The min of two 16-bit lanes has the min of their
// high bytes as its high byte whatever the low bytes hold, so a word of four pixels is folded as
// two words -- W(s), the word starting at column offset s, whose lanes carry pixels 1 and 3 on top,
// and W(s - 1), whose lanes carry pixels 0 and 2 on top -- without any unpacking.  W(s) serves
// offset s for the odd pixels and offset s + 1 for the even ones, so a widening run needs one
// funnel shift per new column.
//
// Fast path (every element row is one run of columns centred on the middle column: disks,
// rectangles, diamonds): every staged row's run grows in registers from radius 0 outwards; where
// element rows of a radius exist the row's word at that radius goes to a shared plane (four radii,
// one per plane, between two barriers), and the element rows of that radius fold the plane's rows
// into the per-row accumulators.  A vertical run of eight or more element rows of one radius is a
// sliding window: the rows common to a thread's eight outputs are folded once.
// Other elements, in a kernel of their own: two folds (odd and even pixels) per element pixel, of words
// that the eight outputs of a thread and the two parities share.
//
// Bound: instructions issued.  4096^2 with the 19 x 19 disk: 49 us per pass at 66% of
// issue cycles (the byte-wise form, one radius per barrier pair and 64-row tiles, took 102 us; this
// form with 64-row tiles and word-wise staging 75 us).
#include <string.h>

#include "common.cuh"
#include "morph.cuh"

namespace nsgb {

namespace {

constexpr int kTileRows = 128;
constexpr int kTileWords = 32;   // 128 columns
constexpr int kHaloWords = 8;    // 32 columns each side: covers offsets up to 31
constexpr int kRowWords = kTileWords + 2 * kHaloWords;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsPerWarp = kTileRows / kWarps;
constexpr int kGroup = 4;  // radii between two barriers, one shared plane each
constexpr int kMaxStageRows = kTileRows + 2 * (kMorphMaxK / 2);
constexpr int kMaxRowsOfWarp = (kMaxStageRows + kWarps - 1) / kWarps;  // staged rows widened by one warp

template <bool MAX>
__device__ __forceinline__ uint32_t fold(uint32_t a, uint32_t b) {
  return MAX ? vmax_u16x2(a, b) : vmin_u16x2(a, b);
}
template <bool MAX>
__device__ __forceinline__ uint32_t fold3(uint32_t a, uint32_t b, uint32_t c) {
  return MAX ? __vimax3_u16x2(a, b, c) : __vimin3_u16x2(a, b, c);
}

// Four pixels under fold: `odd` has pixels 1 and 3 in its high bytes, `even` pixels 0 and 2.
struct Quad {
  uint32_t odd, even;
};
template <bool MAX>
__device__ __forceinline__ void fold_quad(Quad& a, uint32_t w) {
  a.odd = fold<MAX>(a.odd, w);
  a.even = fold<MAX>(a.even, w << 8);
}
__device__ __forceinline__ uint32_t pixels(const Quad& q) { return __byte_perm(q.even, q.odd, 0x7351); }

// The element rows of radius r, from their plane, into the eight outputs of this thread (tile
// rows j0 ..; element row i of output j is plane row j + i).
template <bool MAX>
__device__ __forceinline__ void fold_rows(Quad (&acc)[kRowsPerWarp], const uint32_t* plane, const MorphElement& e,
                                          int r) {
  const int end = e.first_run[r + 1];
  for (int u = e.first_run[r]; u < end; ++u) {
    const int n = e.run_len[u];
    const uint32_t* p = plane + e.run_row[u] * kTileWords;
    if (n == 1 && u + 1 < end && e.run_len[u + 1] == 1) {  // two single rows (the two sides of a disk) at once
      ++u;
      const uint32_t* p2 = plane + e.run_row[u] * kTileWords;
#pragma unroll
      for (int j = 0; j < kRowsPerWarp; ++j) {
        const uint32_t v = p[j * kTileWords], w = p2[j * kTileWords];
        acc[j].odd = fold3<MAX>(acc[j].odd, v, w);
        acc[j].even = fold3<MAX>(acc[j].even, v << 8, w << 8);
      }
      continue;
    }
    if (n < kRowsPerWarp) {
      for (int q = 0; q < n; ++q, p += kTileWords) {
#pragma unroll
        for (int j = 0; j < kRowsPerWarp; ++j) fold_quad<MAX>(acc[j], p[j * kTileWords]);
      }
      continue;
    }
    // output j takes plane rows j .. j + n - 1: rows 7 .. n - 1 are common to all eight, `c` grows
    // upwards from them (row j first), `d` downwards (row n + j - 1)
    Quad c = {p[(kRowsPerWarp - 1) * kTileWords], p[(kRowsPerWarp - 1) * kTileWords] << 8};
    for (int q = kRowsPerWarp; q < n; ++q) fold_quad<MAX>(c, p[q * kTileWords]);
    Quad up[kRowsPerWarp];
#pragma unroll
    for (int j = kRowsPerWarp - 1; j >= 0; --j) {
      if (j < kRowsPerWarp - 1) fold_quad<MAX>(c, p[j * kTileWords]);
      up[j] = c;
    }
    acc[0].odd = fold<MAX>(acc[0].odd, up[0].odd);
    acc[0].even = fold<MAX>(acc[0].even, up[0].even);
    Quad d = {p[n * kTileWords], p[n * kTileWords] << 8};
#pragma unroll
    for (int j = 1; j < kRowsPerWarp; ++j) {
      if (j > 1) fold_quad<MAX>(d, p[(n + j - 1) * kTileWords]);
      acc[j].odd = fold3<MAX>(acc[j].odd, up[j].odd, d.odd);
      acc[j].even = fold3<MAX>(acc[j].even, up[j].even, d.even);
    }
  }
}

// MAX = false: erosion, padding 255; MAX = true: dilation, padding 0.  CENTRED: the fast path (a kernel of
// its own: fetched cold, one with both paths took 5 us longer a pass).  Dynamic shared memory:
// morph_smem(e) bytes.
template <bool MAX, bool CENTRED>
__global__ void __launch_bounds__(kThreads, 2) morph_kernel(const uint8_t* __restrict__ in, int64_t pitch_in,
                                                         bool in_words, bool in_quads, uint8_t* __restrict__ out,
                                                         int64_t pitch_out, bool out_words, int H, int W,
                                                         const __grid_constant__ MorphElement e) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t pad_byte = MAX ? 0u : 255u;
  const uint32_t pad = MAX ? 0u : 0xFFFFFFFFu;
  const int bw = e.bw;
  const int x0 = blockIdx.x * 4 * kTileWords;
  const int rows_in = kTileRows + 2 * bw;
  uint32_t* const S = smem;                                  // [rows_in][kRowWords]
  uint32_t* const R = smem + rows_in * kRowWords;            // [kGroup][rows_in][kTileWords]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // tile rows stride by the grid's y extent (65535 at most)
  for (int64_t ty = blockIdx.y; ty * kTileRows < H; ty += gridDim.y) {
    const int y0 = (int)(ty * kTileRows);
    if (in_quads && x0 >= 4 * kHaloWords && x0 + 4 * (kTileWords + kHaloWords) <= W) {
      // columns all inside: 16 bytes at a time
      constexpr int kRowQuads = kRowWords / 4;
#pragma unroll 4
      for (int k = threadIdx.x; k < rows_in * kRowQuads; k += kThreads) {
        const int i = k / kRowQuads, q = k - i * kRowQuads;
        const int y = y0 - bw + i;
        uint4 v = make_uint4(pad, pad, pad, pad);
        if (y >= 0 && y < H) v = __ldg((const uint4*)(in + (int64_t)y * pitch_in + x0 - 4 * kHaloWords) + q);
        *(uint4*)(S + i * kRowWords + 4 * q) = v;
      }
    } else {
#pragma unroll 2
      for (int i = warp; i < rows_in; i += kWarps) {
        const int y = y0 - bw + i;
        const bool row_in = y >= 0 && y < H;
        const uint8_t* row = in + (int64_t)(row_in ? y : 0) * pitch_in;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int wd = lane + 32 * q;
          if (wd >= kRowWords) break;
          const int xb = x0 + 4 * (wd - kHaloWords);
          uint32_t v = pad;
          if (row_in) {
            if (in_words && xb >= 0 && xb + 4 <= W) {
              v = __ldg((const uint32_t*)(row + xb));
            } else if (xb + 4 > 0 && xb < W) {
              v = 0;
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                const int x = xb + b;
                v |= (x >= 0 && x < W ? (uint32_t)__ldg(row + x) : pad_byte) << (8 * b);
              }
            }
          }
          S[i * kRowWords + wd] = v;
        }
      }
    }
    __syncthreads();

    Quad acc[kRowsPerWarp];
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) acc[j] = Quad{pad, pad};
    const int j0 = warp * kRowsPerWarp;  // this warp's first output row in the tile

    if constexpr (CENTRED) {
      // radius 0: the staged rows themselves
      if (e.radii & 1u) {
        for (int i = warp; i < rows_in; i += kWarps) R[i * kTileWords + lane] = S[i * kRowWords + kHaloWords + lane];
        __syncthreads();
        fold_rows<MAX>(acc, R + j0 * kTileWords + lane, e, 0);
        __syncthreads();
      }
      Quad run[kMaxRowsOfWarp];
#pragma unroll
      for (int t = 0; t < kMaxRowsOfWarp; ++t) {
        const int i = warp + t * kWarps;
        if (i >= rows_in) break;
        const uint32_t* row = S + i * kRowWords + kHaloWords + lane;
        run[t] = Quad{row[0], __funnelshift_r(row[-1], row[0], 24)};
      }
      for (int r = 0; r < e.max_radius; r += kGroup) {  // radii r + 1 .. r + 4
        const uint32_t used = (e.radii >> r) >> 1;
        const int last = e.max_radius - r;  // radii of this group that exist, if below 4
        // words r/4 + 2 left to r/4 + 1 right of the lane's.  The last group reads up to 32 columns
        // left and right (the halo); a word beyond it only serves radii that do not exist.
        const int g = r / kGroup, g2 = min(g + 2, kHaloWords);
#pragma unroll
        for (int t = 0; t < kMaxRowsOfWarp; ++t) {
          const int i = warp + t * kWarps;
          if (i >= rows_in) break;
          const uint32_t* c = S + i * kRowWords + kHaloWords + lane;
          uint32_t* o = R + i * kTileWords + lane;
          const uint32_t l0 = c[-g], l1 = c[-g - 1], l2 = c[-g2];
          const uint32_t r0 = c[g], r1 = c[g + 1];
          // W(-r-1) .. W(-r-5) and W(r) .. W(r+4)
          const uint32_t w1 = __funnelshift_r(l1, l0, 16), v1 = __funnelshift_r(r0, r1, 8);
          run[t].odd = fold3<MAX>(run[t].odd, __funnelshift_r(l1, l0, 24), v1);
          run[t].even = fold3<MAX>(run[t].even, w1, r0);
          if (used & 1u) o[0] = pixels(run[t]);
          if (last == 1) continue;
          const uint32_t w2 = __funnelshift_r(l1, l0, 8), v2 = __funnelshift_r(r0, r1, 16);
          run[t].odd = fold3<MAX>(run[t].odd, w1, v2);
          run[t].even = fold3<MAX>(run[t].even, w2, v1);
          if (used & 2u) o[rows_in * kTileWords] = pixels(run[t]);
          if (last == 2) continue;
          const uint32_t v3 = __funnelshift_r(r0, r1, 24);
          run[t].odd = fold3<MAX>(run[t].odd, w2, v3);
          run[t].even = fold3<MAX>(run[t].even, l1, v2);
          if (used & 4u) o[2 * rows_in * kTileWords] = pixels(run[t]);
          if (last == 3) continue;
          run[t].odd = fold3<MAX>(run[t].odd, l1, r1);
          run[t].even = fold3<MAX>(run[t].even, __funnelshift_r(l2, l1, 24), v3);
          if (used & 8u) o[3 * rows_in * kTileWords] = pixels(run[t]);
        }
        if ((used & 15u) == 0) continue;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kGroup; ++q)
          if ((used >> q) & 1u) fold_rows<MAX>(acc, R + (q * rows_in + j0) * kTileWords + lane, e, r + 1 + q);
        __syncthreads();
      }
    } else {
      // Any element, row by row: each word that a row's columns reach is loaded once for the eight outputs,
      // and the word at each used column offset formed once, for the odd pixels at that offset and the
      // even ones at the next (a word formed anew for each element pixel and parity took 2.0 ms for an opening
      // of 4096^2 by a random 19 x 19 element, 0.55 now).
      const int wd0 = -((e.bw + 4) / 4);  // the word of offset -bw - 1, below
      for (int kr = 0; kr < e.k; ++kr) {
        const uint64_t bits = e.row_bits[kr];  // bit i: offset i - bw for odd pixels, i - bw - 1 for even ones
        if (!bits) continue;
        const uint32_t* row = S + (j0 + kr) * kRowWords + kHaloWords + lane;
        uint32_t cur[kRowsPerWarp], next[kRowsPerWarp];
        bool loaded = false;  // next holds the word that becomes cur
        for (int wd = wd0; 4 * wd <= e.bw; ++wd) {
          const int i0 = 4 * wd + e.bw + 1;  // bit of the word's first offset for even pixels; -3 or more
          const unsigned even = (unsigned)(i0 >= 0 ? bits >> i0 : bits << -i0) & 15u;
          const unsigned odd = (unsigned)(i0 >= 1 ? bits >> (i0 - 1) : bits << (1 - i0)) & 15u;
          if (!(even | odd)) {
            loaded = false;
            continue;
          }
#pragma unroll
          for (int j = 0; j < kRowsPerWarp; ++j) {
            cur[j] = loaded ? next[j] : row[j * kRowWords + wd];
            next[j] = row[j * kRowWords + wd + 1];
          }
          loaded = true;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (!(((even | odd) >> q) & 1u)) continue;
            uint32_t w[kRowsPerWarp];
#pragma unroll
            for (int j = 0; j < kRowsPerWarp; ++j) w[j] = q ? __funnelshift_r(cur[j], next[j], 8 * q) : cur[j];
            if ((odd >> q) & 1u) {
#pragma unroll
              for (int j = 0; j < kRowsPerWarp; ++j) acc[j].odd = fold<MAX>(acc[j].odd, w[j]);
            }
            if ((even >> q) & 1u) {
#pragma unroll
              for (int j = 0; j < kRowsPerWarp; ++j) acc[j].even = fold<MAX>(acc[j].even, w[j]);
            }
          }
        }
      }
    }

    const int xb = x0 + 4 * lane;
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) {
      const int y = y0 + j0 + j;
      if (y >= H || xb >= W) break;
      const uint32_t v = pixels(acc[j]);
      uint8_t* o = out + (int64_t)y * pitch_out + xb;
      if (out_words && xb + 4 <= W) {
        *(uint32_t*)o = v;
      } else {
        for (int b = 0; b < 4 && xb + b < W; ++b) o[b] = (uint8_t)(v >> (8 * b));
      }
    }
    __syncthreads();  // the next tile restages S
  }
}

// Staged rows, and the planes of the centred path: four, or as many as there are radii above 0 (the 3 x 3
// elements then need no more than the 48 KB that a launch has without asking).
size_t morph_smem(const MorphElement& e) {
  const size_t rows_in = kTileRows + 2 * (size_t)e.bw;
  const size_t planes = e.centred ? (e.max_radius < 1 ? 1 : e.max_radius < kGroup ? e.max_radius : kGroup) : 0;
  return sizeof(uint32_t) * rows_in * (kRowWords + planes * kTileWords);
}

bool words_ok(const void* p, int64_t pitch) { return ((uintptr_t)p % 4) == 0 && pitch % 4 == 0; }
bool quads_ok(const void* p, int64_t pitch) { return ((uintptr_t)p % 16) == 0 && pitch % 16 == 0; }

}  // namespace

bool morph_element(const uint8_t* kernel, int k, MorphElement* e) {
  if (!kernel || !e || k < 3 || k > kMorphMaxK || k % 2 == 0) return false;
  memset(e, 0, sizeof(*e));
  e->k = k;
  e->bw = (k - 1) / 2;
  e->centred = 1;
  e->max_radius = 0;
  bool any = false;
  for (int i = 0; i < k; ++i) {
    uint64_t bits = 0;
    for (int j = 0; j < k; ++j)
      if (kernel[i * k + j]) bits |= 1ull << j;
    e->row_bits[i] = bits;
    e->radius[i] = -1;
    if (!bits) continue;
    any = true;
    const int lo = __builtin_ctzll(bits), hi = 63 - __builtin_clzll(bits);
    const bool run = __builtin_popcountll(bits) == hi - lo + 1;
    if (run && lo + hi == 2 * e->bw) {
      const int r = e->bw - lo;
      e->radius[i] = (int8_t)r;
      e->radii |= 1u << r;
      if (r > e->max_radius) e->max_radius = r;
    } else {
      e->centred = 0;
    }
  }
  int runs = 0;
  for (int r = 0; r <= kMorphMaxK / 2; ++r) {
    e->first_run[r] = (uint8_t)runs;
    for (int i = 0; i < k; ++i) {
      if (e->radius[i] != r) continue;
      if (i > 0 && e->radius[i - 1] == r) {
        ++e->run_len[runs - 1];
      } else {
        e->run_row[runs] = (uint8_t)i;
        e->run_len[runs++] = 1;
      }
    }
  }
  e->first_run[kMorphMaxK / 2 + 1] = (uint8_t)runs;
  return any;
}

cudaError_t morph_open_launch(const uint8_t* in, int64_t pitch_in, uint8_t* out, int64_t pitch_out, int rows,
                              int cols, const MorphElement& e, uint8_t* tmp, cudaStream_t s) {
  const int64_t pitch_tmp = ((int64_t)cols + 127) & ~(int64_t)127;
  const int tiles_y = (rows + kTileRows - 1) / kTileRows;
  const dim3 grid((cols + 4 * kTileWords - 1) / (4 * kTileWords), tiles_y < 65535 ? tiles_y : 65535);
  const size_t smem = morph_smem(e);
  const auto erode = e.centred ? morph_kernel<false, true> : morph_kernel<false, false>;
  const auto dilate = e.centred ? morph_kernel<true, true> : morph_kernel<true, false>;
  if (smem > 48 * 1024) {
    cudaError_t r = cudaFuncSetAttribute(erode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r == cudaSuccess) r = cudaFuncSetAttribute(dilate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
  }
  erode<<<grid, kThreads, smem, s>>>(in, pitch_in, words_ok(in, pitch_in), quads_ok(in, pitch_in), tmp, pitch_tmp, true,
                                     rows, cols, e);
  dilate<<<grid, kThreads, smem, s>>>(tmp, pitch_tmp, true, true, out, pitch_out, words_ok(out, pitch_out), rows, cols, e);
  return cudaGetLastError();
}

size_t morph_open_workspace_bytes(int64_t rows, int64_t cols) {
  return 256 + (size_t)rows * (size_t)(((cols + 127) / 128) * 128);
}

}  // namespace nsgb
