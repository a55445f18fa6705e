// Union-find connected-component labelling on GB300 (internal templates).
//
// Reference semantics: ConnComponents::label (fastIA-master/src/segment/ConnComponents.cpp:
// 52-86) joins equal-valued non-zero neighbours (left, up, and up-left / up-right for
// 8-connectivity) and always hooks the larger root under the smaller one (merge, 34-43), so
// every component ends labelled with its smallest raster index; background is bgval.  The GPU
// reference (cuda/ccl_uf.cu:64-157, UF_local / UF_global / UF_final) uses the same
// min-index rule with atomicMin.  This implementation keeps that rule (so labels are
// bit-identical) with its own schedule:
//   1. ccl_local: 32x32 tile per warp; rows as bit masks from ballots, runs joined by pointer
//      jumping and (for the few that touch two runs above) unions in shared memory; writes the
//      tile-local root's global index, lists the local roots and (optionally) their areas.
//   2. ccl_merge: one warp per tile edge joins runs that touch across the edge (global
//      atomicMin hooking; a failed hook retries with the new parent).
//   3. ccl_flatten_roots: every local root points directly at its global root and passes its
//      area on, so any pixel's root is L[L[i]]; seed kernels set a bit on the roots.
// Roots are exactly the pixels with L[i] == i.  Classifiers (the `Cls` template argument)
// return a pixel's class (0 = background; equal non-zero classes are joined), so the same
// kernels serve bwlabel (class = pixel value), hole filling (class = "not foreground"),
// binary reconstruction and bwselect (class = "mask non-zero").
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <climits>
#include <type_traits>

#include "batch.cuh"
#include "common.cuh"
#include "launch.cuh"

namespace nsgb {
namespace ccl {

constexpr int kTile = 32;      // tile edge (pixels)

// Connectivity codes.  4 and 8 join every class alike.  The two dual codes label two classes
// in one forest: kConnFg8Bg4 joins class 1 with 8-connectivity and class 2 with 4-connectivity,
// kConnFg4Bg8 the other way round (the pairs for which a binary image's components form a
// tree by enclosure).
constexpr int kConnFg8Bg4 = 84;
constexpr int kConnFg4Bg8 = 48;

// Whether pixels of class c join their diagonal neighbours of the same class.
template <int CONN>
__device__ __forceinline__ bool joins_diagonally(uint32_t c) {
  if constexpr (CONN == 8) return true;
  else if constexpr (CONN == 4) return false;
  else if constexpr (CONN == kConnFg8Bg4) return c == 1u;
  else return c == 2u;
}
constexpr int kLocalWarps = 4;  // labelling tiles (one warp each) per CTA of ccl_local
constexpr int kMergeTiles = 4;  // labelling tiles (two warps each) per CTA of ccl_merge
constexpr int kManyAlone = 256; // single pixels of a tile from which they are treated apart

// Tile-local forest of one warp (shared memory, 1024 words).  Node i = 32 * row + column; its
// word sits at s[i ^ (i >> 5)], so the same column of 32 rows lies in 32 banks.  A word holds the
// parent in its low 10 bits; the area of a root is added above bit 16 once the unions are done.
constexpr int kNodeMask = kTile * kTile - 1;
__device__ __forceinline__ int node_at(int i) { return i ^ (i >> 5); }

// Root of x, halving the path on the way (every node on it is re-pointed to its grandparent; a
// concurrent hook of a root is never overwritten because roots are not written here).  FINAL: the
// unions are done and other lanes write final roots into these words, so a re-pointing is an
// atomicMin (a parent only ever moves to a smaller node, and the root is the smallest of all).
template <bool FINAL = false>
__device__ __forceinline__ int s_find(volatile int* s, int x) {
  for (;;) {
    const int p = s[node_at(x)] & kNodeMask;
    if (p == x) return x;
    const int g = s[node_at(p)] & kNodeMask;
    if (g == p) return p;
    if (FINAL) atomicMin((int*)&s[node_at(x)], g);
    else s[node_at(x)] = g;
    x = g;
  }
}

__device__ __forceinline__ void s_union(int* s, int a, int b) {
  for (;;) {
    a = s_find(s, a);
    b = s_find(s, b);
    if (a == b) return;
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&s[node_at(a)], b);
    if (old == a) return;
    a = old;
  }
}

// Root of x in the global forest with path halving.  The halving write is an atomicMin: a
// parent link only ever moves to a smaller index (an ancestor), so it can never undo another
// thread's write of the root itself (the smallest index on the path).
// A background entry (-1) on the path means the forest is inconsistent with the classifier
// (never in a correct labelling); the walk then stops with -1 instead of reading before L.
__device__ __forceinline__ int g_find(int* L, int x) {
  for (;;) {
    const int p = ld_relaxed(L + x);
    if (p == x) return x;
    if (p < 0) return -1;
    const int g = ld_relaxed(L + p);
    if (g == p) return p;
    if (g < 0) return -1;
    atomicMin(L + x, g);
    x = g;
  }
}

__device__ __forceinline__ void g_union(int* L, int a, int b) {
  for (;;) {
    a = g_find(L, a);
    b = g_find(L, b);
    if (a == b || a < 0 || b < 0) return;
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&L[a], b);
    if (old == a) return;
    a = old;
  }
}

// Output of a labelling over a batch of images: L (int32, one dense plane per image at
// Img::px_base, pixel index = px_base + y*W + x; -1 = background).  Every foreground pixel
// points at its tile-local root and, after ccl_flatten_roots, every local root points at the
// global root, so root(i) = L[L[i]] (one hop).  Indices are global (px_base included), so a
// root is px_base + the smallest raster index of the component.  A (optional) holds the pixel
// count of each local root, then of each global root.  `roots` lists the local roots,
// `nroots` counts them.
struct Forest {
  int* L;
  int* A;
  int* roots;
  int* nroots;
};

__device__ __forceinline__ int root_of(const int* L, int64_t i) {
  const int l = __ldcg(L + i);
  return l < 0 ? -1 : __ldcg(L + l);
}

// The same, for kernels that do not write L: the second load goes through L1, where the
// pixels of one run (and of one component in a tile) find their shared root.
__device__ __forceinline__ int root_of_ro(const int* L, int64_t i) {
  const int l = __ldg(L + i);
  return l < 0 ? -1 : __ldg(L + l);
}

// Labelling tile `b`: image, tile origin.
struct TileAt {
  Img m;
  int x0, y0;
};
__device__ __forceinline__ TileAt tile_in(const Img& m, int b) {
  TileAt t;
  t.m = m;
  const int lt = b - t.m.c_tile_base;
  const int ty = lt / t.m.c_tiles_x;
  t.x0 = (lt - ty * t.m.c_tiles_x) * kTile;
  t.y0 = ty * kTile;
  return t;
}
__device__ __forceinline__ TileAt tile_at(const Imgs& I, int b) {
  return tile_in(img_at(I, img_of_tile(I, b, I.c_img, I.c_per, CTileBase())), b);
}

// Width of the class values a classifier produces: 8 bits unless it declares `class_t`
// (the float plateau classifier needs all 32 bits of a value).
template <class Cls, class = void>
struct class_type {
  using type = uint8_t;
};
template <class Cls>
struct class_type<Cls, std::void_t<typename Cls::class_t>> {
  using type = typename Cls::class_t;
};

// What a classifier's values can be (`Cls::kKind`): any value, background 0 or class 1, class 1
// or class 2 (no background inside the image), or class 0 / 1 given as 32 pixels of a row at once
// (row_bits).
enum ClassKind { kAnyClass, kOneClass, kTwoClasses, kRowBits };

// The rows of a labelling tile as bit masks (bit = column), lane = row: the foreground, the run
// starts, and the pixels at which a union with the row above is due -- straight up, up-left, up-right.
struct RowMasks {
  unsigned fg, start, up, ul, ur;
};

__device__ __forceinline__ unsigned above(unsigned m, int lane) {
  const unsigned u = __shfl_up_sync(NSGB_FULL, m, 1);
  return lane ? u : 0u;
}

// One class (mask m of this lane's row): a pair of touching runs of adjacent rows is joined once,
// at the first column of their overlap, or diagonally past an end of the lower run where the
// pixel above that end is not of the class.
__device__ __forceinline__ void class_masks(unsigned m, bool diag, int lane, RowMasks& k) {
  const unsigned u = above(m, lane), st = m & ~(m << 1), c = m & u;
  k.fg |= m;
  k.start |= st;
  k.up |= c & ~(c << 1);
  if (diag) {
    k.ul |= st & (u << 1) & ~u;
    k.ur |= m & ~(m >> 1) & (u >> 1) & ~u;
  }
}

// Any classes: the rows are classified once more, pixel values in hand.  Touching equal pixels
// are joined where either run starts, or where the overlap does; diagonals as above.
template <int CONN, class Cls>
__device__ __forceinline__ RowMasks any_masks(const Cls& cls, const TileAt& T, int rows_in, int gx, int lane) {
  RowMasks k = {0u, 0u, 0u, 0u, 0u};
  unsigned same_left = 0, same_up = 0, same_ul = 0, same_ur = 0;
  uint32_t prev = 0, prev_left = 0;
  const int cx = min(gx, T.m.W - 1);  // loads without a predicate, dropped past the edge (see local_tile)
#pragma unroll 8
  for (int r = 0; r < kTile; ++r) {
    const uint32_t p = (uint32_t)cls(T.m, T.y0 + min(r, rows_in - 1), cx);
    const uint32_t v = r < rows_in && gx < T.m.W ? p : 0u;
    const uint32_t left = __shfl_up_sync(NSGB_FULL, v, 1);
    const bool fg = v != 0u;
    const unsigned f = __ballot_sync(NSGB_FULL, fg);
    const unsigned sl = __ballot_sync(NSGB_FULL, fg && lane > 0 && left == v);
    const unsigned su = __ballot_sync(NSGB_FULL, fg && prev == v);  // prev is 0 for the first row
    unsigned sul = 0, sur = 0;
    if constexpr (CONN != 4) {
      const uint32_t prev_right = __shfl_down_sync(NSGB_FULL, prev, 1);
      const bool d = fg && joins_diagonally<CONN>(v);
      sul = __ballot_sync(NSGB_FULL, d && lane > 0 && prev_left == v);
      sur = __ballot_sync(NSGB_FULL, d && lane < 31 && prev_right == v);
    }
    if (lane == r) {
      k.fg = f;
      same_left = sl;
      same_up = su;
      same_ul = sul;
      same_ur = sur;
    }
    prev = v;
    prev_left = left;
  }
  k.start = k.fg & ~same_left;
  const unsigned start_above = above(k.start, lane);
  k.up = same_up & (~(same_up << 1) | k.start | start_above);
  k.ul = same_ul & k.start & ~same_up;
  k.ur = same_ur & ~(same_left >> 1) & ~same_up;
  return k;
}

// Column of the start at or before column x.
__device__ __forceinline__ int start_at(unsigned starts, int x) { return 31 - __clz(starts & (0xFFFFFFFFu >> (31 - x))); }

// Steps (3) to (6) of a tile with both runs and background or several classes.  ALONE: `alone` are single
// pixels without a contact, components of their own; they take no part in (3) to (5) and are labelled and
// listed in (6), a row at a time.
template <bool ALONE>
__device__ __forceinline__ void finish_tile(const RowMasks& k, unsigned alone, const Forest& f, int* s, unsigned* starts,
                                            int x0, int y0, int W, int pb, int rows_in, int* Lt) {
  const int lane = threadIdx.x & 31, gx = x0 + lane;

  // (3) contacts, lane = row
  const int row = kTile * lane;
  const unsigned runs = ALONE ? k.start & ~alone : k.start;
  const unsigned start_above = above(k.start, lane);
  unsigned up = k.up, ul = k.ul, ur = k.ur;
  for (unsigned w = runs; w; w &= w - 1u) {
    const int x = __ffs(w) - 1;
    const unsigned next = (k.start | ~k.fg) & ~(0xFFFFFFFFu >> (31 - x));  // first column past the run
    const unsigned run = (next ? (next & (0u - next)) - 1u : 0xFFFFFFFFu) & (0xFFFFFFFFu << x);
    int c = -1;  // the column above of the run's first contact
    unsigned t;
    if ((ul >> x) & 1u) {
      ul &= ~(1u << x);
      c = x - 1;
    } else if ((t = up & run) != 0u) {
      up &= ~(t & (0u - t));
      c = __ffs(t) - 1;
    } else if ((t = ur & run) != 0u) {
      ur &= ~t;
      c = __ffs(t);
    }
    s[node_at(row + x)] = c >= 0 ? row - kTile + start_at(start_above, c) : row + x;
  }
  __syncwarp();
  for (;;) {
    bool moved = false;
    for (unsigned w = runs; w; w &= w - 1u) {
      volatile int* v = s;
      const int i = node_at(row + __ffs(w) - 1);
      const int p = v[i], g = v[node_at(p)];
      if (g != p) {
        v[i] = g;
        moved = true;
      }
    }
    if (!__any_sync(NSGB_FULL, moved)) break;
  }
  if (__any_sync(NSGB_FULL, (up | ul | ur) != 0u)) {
    int d = 0;
    for (;;) {
      if (up == 0u) {
        if (ul) {
          up = ul, ul = 0u, d = -1;
        } else if (ur) {
          up = ur, ur = 0u, d = 1;
        } else {
          break;
        }
      }
      const int x = __ffs(up) - 1;
      up &= up - 1u;
      s_union(s, row + start_at(k.start, x), row - kTile + start_at(start_above, x + d));
    }
    __syncwarp();
  }

  // (4) every run points at its root; run lengths add up at the roots (above bit 16)
  unsigned is_root = 0u;
  for (unsigned w = runs; w; w &= w - 1u) {
    const int x = __ffs(w) - 1, i = row + x;
    const int r = s_find<true>(s, i);
    if (r == i) is_root |= 1u << x;
    else atomicMin(&s[node_at(i)], r);
    if (f.A) {
      const unsigned stop = (k.start | ~k.fg) & ~(0xFFFFFFFFu >> (31 - x));
      atomicAdd(&s[node_at(r)], ((stop ? __ffs(stop) - 1 : 32) - x) << 16);
    }
  }
  __syncwarp();

  // (5) the tile's local roots go to the list with one atomic, and every run start (background
  // runs included) gets the label of its pixels.  A lane touches only the nodes of its own row.
  const int nr = __popc(is_root) + (ALONE ? __popc(alone) : 0);
  int incl = nr;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(NSGB_FULL, incl, o);
    if (lane >= o) incl += v;
  }
  int base = 0;
  if (lane == 31) base = atomicAdd(f.nroots, incl);
  base = __shfl_sync(NSGB_FULL, base, 31) + incl - nr;
  const unsigned every = k.start | (~k.fg & ((k.fg << 1) | 1u));
  starts[lane] = ALONE ? k.start : every;
  for (unsigned w = ALONE ? runs : every; w; w &= w - 1u) {
    const int x = __ffs(w) - 1;
    int* const node = &s[node_at(row + x)];
    int label = -1;
    if ((k.fg >> x) & 1u) {
      const int v = *node, q = v & kNodeMask;
      label = pb + (y0 + (q >> 5)) * W + x0 + (q & 31);
      if ((is_root >> x) & 1u) {
        f.roots[base++] = label;
        if (f.A) f.A[label] = v >> 16;
      }
    }
    *node = label;
  }
  __syncwarp();

  // (6) labels, lane = column
  const unsigned upto = 0xFFFFFFFFu >> (31 - lane);
  if constexpr (!ALONE) {
    if (gx < W) {
#pragma unroll 8
      for (int r = 0; r < rows_in; ++r, Lt += W) *Lt = s[node_at(kTile * r + 31 - __clz(starts[r] & upto))];
    }
  } else {
#pragma unroll 4
    for (int r = 0; r < rows_in; ++r, Lt += W) {
      const unsigned one = __shfl_sync(NSGB_FULL, alone, r), fg = __shfl_sync(NSGB_FULL, k.fg, r);
      const int at = __shfl_sync(NSGB_FULL, base, r);
      int label = -1;
      if ((one >> lane) & 1u) {
        label = pb + (y0 + r) * W + gx;
        f.roots[at + __popc(one & (upto >> 1))] = label;
        if (f.A) f.A[label] = 1;
      } else if ((fg >> lane) & 1u) {
        label = s[node_at(kTile * r + 31 - __clz(starts[r] & upto))];
      }
      if (gx < W) *Lt = label;
    }
  }
}

// Tile-local labelling: one warp per 32 x 32 tile.  The pixels of a row become bit masks (ballots
// over lane = column; lane r keeps row r), and from there on lane = row works on whole runs with
// bit operations.  Runs of equal class along a row start out joined (node = run start).  A pair of
// touching runs of adjacent rows is one contact:
//   - each run's first contact is a plain store (its parent is the run above; parents are smaller,
//     so this is a forest), and pointer jumping in lockstep flattens it in at most five rounds --
//     for blobs that is nearly all there is;
//   - the remaining contacts (a run that touches two runs above) are unions in shared memory.
// Each run then adds its length to its root's area and puts its label at its start, and the
// labels are written lane = column, every pixel through the start of its run.
//
// Bound: instructions issued (63% of cycles).  The kernel it replaced (a 256-thread CTA per tile,
// unions, finds and area counts per pixel) issued about 5200 warp instructions per mixed tile,
// this one 1200 (one class) to 1450 (two).  4096^2 u8, cold: two classes with areas 102 -> 38 us,
// a 0 / 255 mask 76 -> 32 us; from a bit plane, 47 Mpixel of uneven tiles: 109 -> 70 us.
//
// `s` (1024 words) and `starts` (32) are the warp's own shared memory.
template <class Cls, int CONN>
__device__ __forceinline__ void local_tile(const Cls& cls, const TileAt& T, const Forest& f, int* s, unsigned* starts) {
  const int lane = threadIdx.x & 31;
  const int x0 = T.x0, y0 = T.y0, W = T.m.W, pb = T.m.px_base;
  const int gx = x0 + lane;
  const unsigned cols_in = W - x0 >= 32 ? 0xFFFFFFFFu : (1u << (W - x0)) - 1u;
  const int rows_in = min(kTile, T.m.H - y0);

  // (1) lane r: the masks of row r
  RowMasks k = {0u, 0u, 0u, 0u, 0u};
  if constexpr (Cls::kKind == kRowBits) {
    const unsigned m = lane < rows_in ? cls.row_bits(T.m, y0 + lane, x0) & cols_in : 0u;
    class_masks(m, joins_diagonally<CONN>(1u), lane, k);
  } else if constexpr (Cls::kKind == kAnyClass && sizeof(typename class_type<Cls>::type) > 1) {
    k = any_masks<CONN>(cls, T, rows_in, gx, lane);
  } else {
    unsigned m = 0;
    uint32_t any = 0u, all = ~0u;  // of the non-zero values (kAnyClass)
    // Past the image edge the last row or column is read again and masked off below: loads
    // without a predicate all go out before the first ballot (guarded ones came one by one:
    // 71 against 30 us for the two classes of a 4096^2 u8 tile).
    const int cx = min(gx, W - 1);
#pragma unroll
    for (int r = 0; r < kTile; ++r) {
      const uint32_t v = (uint32_t)cls(T.m, y0 + min(r, rows_in - 1), cx);
      if constexpr (Cls::kKind == kAnyClass) {
        any |= v;
        all &= v ? v : ~0u;
      }
      const unsigned w = __ballot_sync(NSGB_FULL, Cls::kKind == kTwoClasses ? v == 1u : v != 0u);
      if (lane == r) m = w;
    }
    m = lane < rows_in ? m & cols_in : 0u;
    // one non-zero class in the whole tile (a 0 / 255 mask), or several
    if (Cls::kKind == kAnyClass &&
        (__reduce_or_sync(NSGB_FULL, any) & ~__reduce_and_sync(NSGB_FULL, all)) != 0u) {
      k = any_masks<CONN>(cls, T, rows_in, gx, lane);
    } else {
      class_masks(m, joins_diagonally<CONN>(1u), lane, k);
      if constexpr (Cls::kKind == kTwoClasses)
        class_masks(lane < rows_in ? cols_in & ~m : 0u, joins_diagonally<CONN>(2u), lane, k);
    }
  }

  int* Lt = f.L + pb + (int64_t)y0 * W + gx;  // this lane's column of the tile
  // (2) a tile without foreground, or one solid class: no unions
  const bool empty = __all_sync(NSGB_FULL, k.fg == 0u);
  const bool solid = __all_sync(NSGB_FULL, k.fg == 0xFFFFFFFFu && k.start == 1u && (lane == 0 || k.up == 1u));
  if (empty || solid) {
    const int g0 = pb + y0 * W + x0;
    const int v = solid ? g0 : -1;
    if (gx < W) {
#pragma unroll 8
      for (int r = 0; r < rows_in; ++r, Lt += W) *Lt = v;
    }
    if (solid && lane == 0) {
      f.roots[atomicAdd(f.nroots, 1)] = g0;
      if (f.A) f.A[g0] = kTile * kTile;
    }
    return;
  }

  // Single pixels without a contact are treated apart where they are many.  (A lane takes the runs of its row one
  // after another: a tile of single pixels, such as the plateaus of a float image or a checkerboard, was 32
  // steps in each of (3) to (5).  4096^2 u8, 8-connected 256-valued noise 119 -> 86 us, 4-connected
  // checkerboard 170 -> 51; 4 float planes of 1024^2 58 -> 49.)  Classifiers of one class and of two see
  // masks, where they are few.
  if constexpr (Cls::kKind == kAnyClass) {
    const unsigned touches = k.up | (k.ul >> 1) | (k.ur << 1);  // columns of the row above
    const unsigned below = __shfl_down_sync(NSGB_FULL, touches, 1);
    const unsigned single = k.start & (((k.start | ~k.fg) >> 1) | 0x80000000u);
    const unsigned alone = single & ~(k.up | k.ul | k.ur | (lane < 31 ? below : 0u));
    if (__reduce_add_sync(NSGB_FULL, __popc(alone)) >= kManyAlone) {
      finish_tile<true>(k, alone, f, s, starts, x0, y0, W, pb, rows_in, Lt);
      return;
    }
  }
  finish_tile<false>(k, 0u, f, s, starts, x0, y0, W, pb, rows_in, Lt);
}

template <class Cls, int CONN>
__global__ void __launch_bounds__(32 * kLocalWarps) ccl_local(Cls cls, Imgs I, Forest f, int ntiles) {
  pdl_wait();
  pdl_release();
  __shared__ int s_nodes[kLocalWarps][kTile * kTile];
  __shared__ unsigned s_starts[kLocalWarps][kTile];
  const int b = blockIdx.x * kLocalWarps + (threadIdx.x >> 5);
  if (b >= ntiles) return;  // whole warp; the warps of a CTA are independent
  local_tile<Cls, CONN>(cls, tile_at(I, b), f, s_nodes[threadIdx.x >> 5], s_starts[threadIdx.x >> 5]);
}

// Joins runs across tile edges.  Two warps per labelling tile: warp 0 takes the bottom edge
// (row y0+31 against row y0+32), warp 1 the right edge (column x0+31 against column x0+32, the
// same logic transposed).  With `a` = the pixel on this side and `b` its partner across the
// edge, runs of equal class along the edge are found with ballots, and a union is made only
// where a run on the far side starts or where a near-side run starts under a far-side run,
// plus the two diagonal ends of each far-side run for 8-connectivity.
template <class Cls, int CONN>
__device__ __forceinline__ void merge_edge(const Cls& cls, const TileAt& T, int* L, bool bottom) {
  const int x0 = T.x0, y0 = T.y0, H = T.m.H, W = T.m.W, pb = T.m.px_base;
  const int lane = threadIdx.x & 31;
  // coordinates of the near pixel (a) and the far pixel (b) for this lane
  int ay, ax, by, bx;
  if (bottom) {
    ay = y0 + kTile - 1;
    ax = x0 + lane;
    by = ay + 1;
    bx = ax;
    if (by >= H) return;  // whole warp: no tile below
  } else {
    ax = x0 + kTile - 1;
    ay = y0 + lane;
    bx = ax + 1;
    by = ay;
    if (bx >= W) return;
  }
  const bool in_a = ay < H && ax < W;
  const bool in_b = by < H && bx < W;
  const uint32_t ca = in_a ? cls(T.m, ay, ax) : 0u;
  const uint32_t cb = in_b ? cls(T.m, by, bx) : 0u;
  // runs along the edge (lane order) on each side
  const uint32_t ca_prev = __shfl_up_sync(NSGB_FULL, ca, 1);
  const uint32_t cb_prev = __shfl_up_sync(NSGB_FULL, cb, 1);
  const uint32_t cb_next = __shfl_down_sync(NSGB_FULL, cb, 1);
  const bool a_start = ca != 0 && !(lane > 0 && ca_prev == ca);
  const bool b_start = cb != 0 && !(lane > 0 && cb_prev == cb);
  const bool b_end = cb != 0 && !(lane < 31 && cb_next == cb);
  if (cb == 0) return;
  const int qb = pb + by * W + bx;
  if (ca == cb && (a_start || b_start)) g_union(L, qb, pb + ay * W + ax);
  // Diagonal partners one step before the start / after the end of the far-side run.  When
  // the near pixel at this lane has the far run's class, the partner (its neighbour along the
  // edge) is joined to it by the near tile's own labelling or by the next tile's edge merge,
  // and the near pixel is joined to the far run here: the diagonal union adds nothing.
  if (ca != cb && joins_diagonally<CONN>(cb)) {
    if (b_start) {
      const int dy = bottom ? ay : ay - 1, dx = bottom ? ax - 1 : ax;
      if (dy >= 0 && dx >= 0 && dy < H && dx < W && cls(T.m, dy, dx) == cb) g_union(L, qb, pb + dy * W + dx);
    }
    if (b_end) {
      const int dy = bottom ? ay : ay + 1, dx = bottom ? ax + 1 : ax;
      if (dy < H && dx < W && cls(T.m, dy, dx) == cb) g_union(L, qb, pb + dy * W + dx);
    }
  }
}

template <class Cls, int CONN>
__global__ void __launch_bounds__(64 * kMergeTiles) ccl_merge(Cls cls, Imgs I, Forest f, int ntiles) {
  pdl_wait();
  pdl_release();
  const int b = blockIdx.x * kMergeTiles + (threadIdx.x >> 6);
  if (b < ntiles) merge_edge<Cls, CONN>(cls, tile_at(I, b), f.L, ((threadIdx.x >> 5) & 1) == 0);
}

// Every local root points directly at its global root; local-root areas move into the root.
// Four list entries per thread and iteration, their loads issued together: most local roots
// are global roots already (one load to see it), so the kernel is load-latency bound.  The
// area adds of a warp are summed per root first (one atomic per root and warp): the local
// roots of a giant component, one per labelling tile, all add into the same word.
__device__ __forceinline__ void flatten_roots(const Forest& f, int max_roots) {
  const int n = min(__ldcg(f.nroots), max_roots);
  const int stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 - lane < n; k0 += 4 * stride) {
    int lr[4], p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) lr[j] = k0 + j * stride < n ? __ldcg(f.roots + k0 + j * stride) : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = lr[j] >= 0 ? __ldcg(f.L + lr[j]) : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int r = -1, a = 0;
      if (lr[j] >= 0 && p[j] != lr[j]) {
        r = g_find(f.L, lr[j]);
        if (r >= 0 && r != lr[j]) {
          atomicMin(f.L + lr[j], r);
          if (f.A) a = __ldcg(f.A + lr[j]);
        } else {
          r = -1;
        }
      }
      if (f.A) {
        const unsigned peers = __match_any_sync(NSGB_FULL, r);
        const int sum = __reduce_add_sync(peers, a);
        if (r >= 0 && (__ffs(peers) - 1) == lane) atomicAdd(f.A + r, sum);
      }
    }
  }
}

static __global__ void ccl_flatten_roots(Forest f, int max_roots) {
  pdl_wait();
  pdl_release();
  flatten_roots(f, max_roots);
}

__device__ __forceinline__ void set_root_bit(unsigned* bits, int r) {
  const unsigned bit = 1u << (r & 31);
  if (!(__ldcg(&bits[r >> 5]) & bit)) atomicOr(&bits[r >> 5], bit);
}

// Row walk over the rows of all images: g(image, row within the image) for every row this
// block row owns.  A single image strides its rows by gridDim.y.  A batch gives each block row
// a contiguous range of the concatenated rows, so the image is looked up once per block row
// (a binary search over the table) and then followed across image boundaries, instead of
// searching again for every row.
template <class G>
__device__ __forceinline__ void for_batch_rows(const Imgs& I, int total_rows, G&& g) {
  if (!I.d) {
    for (int gr = blockIdx.y; gr < total_rows; gr += gridDim.y) g(I.one, gr);
    return;
  }
  const int per = (total_rows + (int)gridDim.y - 1) / (int)gridDim.y;
  const int r0 = (int)blockIdx.y * per, r1 = min(total_rows, r0 + per);
  if (r0 >= r1) return;
  int ii = img_of(I, r0, RowBase());
  Img m = I.d[ii];
  int next = ii + 1 < I.n ? I.d[ii + 1].row_base : INT_MAX;
  for (int gr = r0; gr < r1; ++gr) {
    while (gr >= next) {
      ++ii;
      m = I.d[ii];
      next = ii + 1 < I.n ? I.d[ii + 1].row_base : INT_MAX;
    }
    g(m, gr - m.row_base);
  }
}

// Row grid over the rows of all images: x = column (blockIdx.x * blockDim.x + threadIdx.x);
// f(image, y, x) runs for every pixel.
template <class F>
__device__ __forceinline__ void for_batch_pixels(const Imgs& I, int total_rows, F&& f) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  for_batch_rows(I, total_rows, [&](const Img& m, int y) {
    if (x < m.W) f(m, y, x);
  });
}

// The same with four consecutive pixels per thread: f(image, y, x, n) for pixels x .. x+n-1
// (n <= 4) of row y; x grid over max_w / 4.
template <class F>
__device__ __forceinline__ void for_batch_quads(const Imgs& I, int total_rows, F&& f) {
  const int x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  for_batch_rows(I, total_rows, [&](const Img& m, int y) {
    if (x < m.W) f(m, y, x, min(4, m.W - x));
  });
}

// Label plane entries of four consecutive pixels (L read-only; -1 from n on): one 16-byte load
// when aligned.
__device__ __forceinline__ void labels4_ro(const int* L, int64_t i, int n, int (&l)[4]) {
  if (n == 4 && ((i & 3) == 0)) {
    const int4 v = __ldg((const int4*)(L + i));
    l[0] = v.x, l[1] = v.y, l[2] = v.z, l[3] = v.w;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) l[k] = k < n ? __ldg(L + i + k) : -1;
  }
}

// Roots of four consecutive pixels (L read-only).
__device__ __forceinline__ void roots4_ro(const int* L, int64_t i, int n, int (&r)[4]) {
  int l[4];
  labels4_ro(L, i, n, l);
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = l[k] < 0 ? -1 : (k > 0 && l[k] == l[k - 1] ? -2 : __ldg(L + l[k]));
#pragma unroll
  for (int k = 1; k < 4; ++k)
    if (r[k] == -2) r[k] = r[k - 1];
}

// Seed pixels set bit root(p) in `bits`.
template <class Seed>
__global__ void ccl_seed_pixels(Imgs I, int total_rows, const int* __restrict__ L, Seed seed,
                                unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  for_batch_pixels(I, total_rows, [&](const Img& m, int y, int x) {
    if (!seed(m, y, x)) return;
    const int r = root_of(L, (int64_t)m.px_base + (int64_t)y * m.W + x);
    if (r >= 0) set_root_bit(bits, r);
  });
}

// Border pixel k of an H x W image (top row, bottom row, left column, right column; 2W + 2H
// positions, corners visited twice).
__device__ __forceinline__ void border_pixel(int k, int H, int W, int& y, int& x) {
  if (k < W) {
    y = 0;
    x = k;
  } else if (k < 2 * W) {
    y = H - 1;
    x = k - W;
  } else if (k < 2 * W + H) {
    y = k - 2 * W;
    x = 0;
  } else {
    y = k - 2 * W - H;
    x = W - 1;
  }
}

// Seed pixels on each image's border only: blockIdx.y = image, x walks its border.
template <class Seed>
__global__ void ccl_seed_border(Imgs I, const int* __restrict__ L, Seed seed, unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  const Img m = img_at(I, blockIdx.y);
  const int H = m.H, W = m.W;
  const int per = 2 * W + 2 * H;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < per; k += gridDim.x * blockDim.x) {
    int y, x;
    border_pixel(k, H, W, y, x);
    if (!seed(m, y, x)) continue;
    const int r = root_of(L, (int64_t)m.px_base + (int64_t)y * W + x);
    if (r >= 0) set_root_bit(bits, r);
  }
}

// The same before the roots are flattened (after ccl_merge): the root is found by walking the
// forest.
template <class Seed>
__global__ void ccl_seed_border_walk(Imgs I, int* L, Seed seed, unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  const Img m = img_at(I, blockIdx.y);
  const int H = m.H, W = m.W;
  const int per = 2 * W + 2 * H;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < per; k += gridDim.x * blockDim.x) {
    int y, x;
    border_pixel(k, H, W, y, x);
    if (!seed(m, y, x)) continue;
    const int r = g_find(L, m.px_base + y * W + x);
    if (r >= 0) set_root_bit(bits, r);
  }
}

// Read-only in the kernels that call it, so the L1-cached path is used: a giant component's
// root word is read by every pixel and would otherwise hammer one L2 line.
__device__ __forceinline__ bool test_bit(const unsigned* bits, int r) {
  return (__ldg(&bits[r >> 5]) >> (r & 31)) & 1u;
}

// Host helpers (ccl.cu).
int flat_grid(int64_t n);
// Grid for kernels that walk a device-side list whose length (unknown on the host) is at most
// max_items.
int list_grid(int64_t max_items);
// Row grids: x covers the widest image (256 columns, or 256 quads of columns, per block), y
// strides the rows (one block row per image row up to the grid limit: batched kernels look
// the image of a row up per row, so they want many short row walks).
inline unsigned row_blocks(int total_rows) { return (unsigned)(total_rows < 65535 ? total_rows : 65535); }
inline dim3 rowcol_grid(int total_rows, int max_w) {
  const unsigned bx = (unsigned)((max_w + 255) / 256);
  return dim3(bx, row_blocks(total_rows));
}
inline dim3 quadrow_grid(int total_rows, int max_w) {
  const unsigned bx = (unsigned)(((max_w + 3) / 4 + 255) / 256);
  return dim3(bx, row_blocks(total_rows));
}

inline unsigned merge_grid(int c_tiles) { return (unsigned)((c_tiles + kMergeTiles - 1) / kMergeTiles); }
inline unsigned local_grid(int c_tiles) { return (unsigned)((c_tiles + kLocalWarps - 1) / kLocalWarps); }

// Up to four word ranges to clear in one launch (n[k] words from p[k]; unused ranges have n 0).
struct ZeroSpans {
  unsigned* p[4];
  int n[4];
  int total() const { return n[0] + n[1] + n[2] + n[3]; }
};

static __global__ void zero_words(ZeroSpans z) {
  pdl_wait();
  pdl_release();
  const int total = z.n[0] + z.n[1] + z.n[2] + z.n[3];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int j = i, r = 0;
    while (j >= z.n[r]) j -= z.n[r++];
    z.p[r][j] = 0u;
  }
}

// Launches `kernel` the ordinary way, or (pdl) as a programmatic dependent of the kernel before
// it on the stream, which every kernel launched here waits for first thing.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s,
                            Args&&... args) {
  if (pdl) return launch_dependent(kernel, grid, block, s, std::forward<Args>(args)...);
  kernel<<<grid, block, 0, s>>>(std::forward<Args>(args)...);
  return cudaGetLastError();
}

// Labels every image of the batch: local pass, edge merge, root flattening.  Afterwards
// root(i) = L[L[i]].  The first launch is an ordinary one (it may follow anything); it clears the
// root count and the caller's ranges 1 to 3 of `more`, so that no memset stands between the
// launches, and every later launch is a programmatic dependent of the one before it.
template <class Cls>
cudaError_t label(const Cls& cls, const Imgs& I, const BatchTotals& t, int conn, const Forest& f, cudaStream_t s,
                  ZeroSpans more = ZeroSpans{{nullptr, nullptr, nullptr, nullptr}, {0, 0, 0, 0}}) {
  ZeroSpans z = more;
  z.p[0] = (unsigned*)f.nroots;
  z.n[0] = 1;
  cudaError_t e = launch_k(false, zero_words, dim3(flat_grid(z.total())), dim3(256), s, z);
  const dim3 lg(local_grid(t.c_tiles)), mg(merge_grid(t.c_tiles));
  if (e != cudaSuccess) return e;
  if (conn == 8) {
    e = launch_dependent(ccl_local<Cls, 8>, lg, dim3(32 * kLocalWarps), s, cls, I, f, t.c_tiles);
    if (e == cudaSuccess) e = launch_dependent(ccl_merge<Cls, 8>, mg, dim3(64 * kMergeTiles), s, cls, I, f, t.c_tiles);
  } else {
    e = launch_dependent(ccl_local<Cls, 4>, lg, dim3(32 * kLocalWarps), s, cls, I, f, t.c_tiles);
    if (e == cudaSuccess) e = launch_dependent(ccl_merge<Cls, 4>, mg, dim3(64 * kMergeTiles), s, cls, I, f, t.c_tiles);
  }
  if (e == cudaSuccess) e = launch_dependent(ccl_flatten_roots, dim3(list_grid(t.px)), dim3(256), s, f, (int)t.px);
  return e;
}

// Enclosure tree of a two-class labelling (kConnFg8Bg4 / kConnFg4Bg8, before flattening):
// with dual connectivities the components of the two classes form a tree by enclosure, the
// image's outside (the components marked in `outside`, those of the outside class that touch
// the border) at its top, and a component's parent is the component of the pixel directly
// above its first pixel in raster order (its root).  Every component below the top joins its
// parent, so each set that results is one component of "class 1 plus the class-2 components
// it encloses" (class 1 with its holes filled).  One thread per listed local root; a global
// root is hooked only by its own thread (its parent's root index is smaller than its own), so
// the test for a global root at the start holds until the thread itself changes it.
static __global__ void ccl_join_parents(Imgs I, Forest f, int max_roots, const unsigned* __restrict__ outside) {
  pdl_wait();
  pdl_release();
  const int n = min(__ldcg(f.nroots), max_roots);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int r = __ldcg(f.roots + k);
    if (ld_relaxed(f.L + r) != r) continue;
    if ((__ldcg(outside + (r >> 5)) >> (r & 31)) & 1u) continue;
    const Img m = img_at(I, img_of(I, r, PxBase()));
    if (r - m.px_base < m.W) continue;  // first row: its parent is the outside
    const int p = g_find(f.L, r - m.W);
    if (p < 0 || ((__ldcg(outside + (p >> 5)) >> (p & 31)) & 1u)) continue;
    g_union(f.L, r, p);
  }
}

// Seed test: pixels of class 2.
template <class Cls>
struct Class2 {
  Cls cls;
  __device__ bool operator()(const Img& m, int y, int x) const { return cls(m, y, x) == 2u; }
};

// Labels both classes of a two-class classifier (class 1 = the foreground, class 2 = the rest)
// with dual connectivities and joins every component below the outside to its parent: the
// sets are then the components of the foreground with its holes filled, each rooted at its
// smallest raster index, and A holds their areas (holes included).  The border components of
// class 2 are marked in `outside` (zeroed first; their roots stay roots and are not part of
// the filled image).  Afterwards root(i) = L[L[i]].
template <class Cls>
cudaError_t label_filled(const Cls& cls, const Imgs& I, const BatchTotals& t, int conn, const Forest& f,
                         unsigned* outside, size_t outside_bytes, cudaStream_t s, bool pdl = false,
                         ZeroSpans more = ZeroSpans{{nullptr, nullptr, nullptr, nullptr}, {0, 0, 0, 0}}) {
  // The first launch follows whatever the caller queued last, so it is an ordinary one; the
  // rest may start while their predecessor drains.  It also clears the caller's ranges 2 and 3
  // of `more` (for the ranking that follows, say).
  ZeroSpans z = more;
  z.p[0] = (unsigned*)f.nroots;
  z.n[0] = 1;
  z.p[1] = outside;
  z.n[1] = (int)(outside_bytes / sizeof(unsigned));
  cudaError_t e = launch_k(false, zero_words, dim3(flat_grid(z.total())), dim3(256), s, z);
  if (e != cudaSuccess) return e;
  if (conn == kConnFg8Bg4) {
    e = launch_k(pdl, ccl_local<Cls, kConnFg8Bg4>, dim3(local_grid(t.c_tiles)), dim3(32 * kLocalWarps), s, cls, I, f, t.c_tiles);
    if (e == cudaSuccess) e = launch_k(pdl, ccl_merge<Cls, kConnFg8Bg4>, dim3(merge_grid(t.c_tiles)), dim3(64 * kMergeTiles), s, cls, I, f, t.c_tiles);
  } else {
    e = launch_k(pdl, ccl_local<Cls, kConnFg4Bg8>, dim3(local_grid(t.c_tiles)), dim3(32 * kLocalWarps), s, cls, I, f, t.c_tiles);
    if (e == cudaSuccess) e = launch_k(pdl, ccl_merge<Cls, kConnFg4Bg8>, dim3(merge_grid(t.c_tiles)), dim3(64 * kMergeTiles), s, cls, I, f, t.c_tiles);
  }
  const int gx = (t.perimeter_max + 255) / 256 > 64 ? 64 : (t.perimeter_max + 255) / 256;
  if (e == cudaSuccess)
    e = launch_k(pdl, ccl_seed_border_walk<Class2<Cls>>, dim3(gx > 0 ? gx : 1, t.n), dim3(256), s, I, f.L,
                 Class2<Cls>{cls}, outside);
  if (e == cudaSuccess)
    e = launch_k(pdl, ccl_join_parents, dim3(list_grid(t.px)), dim3(256), s, I, f, (int)t.px, (const unsigned*)outside);
  if (e == cudaSuccess) e = launch_k(pdl, ccl_flatten_roots, dim3(list_grid(t.px)), dim3(256), s, f, (int)t.px);
  return e;
}

// Raster-order ranks of the global roots, from the list of local roots: rank[r] = number of
// roots of r's image before r (written at roots only).  counts[2*i] = roots of image i,
// counts[2*i+1] = roots whose area (A, if given) lies in [lo, hi).  `bits` (one bit per
// pixel, px/32 + 2 words), `block_tmp` (one int per rank block) and `wpre` (32 ints per rank
// block) are scratch.
// Roots marked in `skip` (optional) are left out: not counted and not ranked.
// With pdl, every launch is a programmatic dependent of the kernel before it (the caller's last
// launch must be a kernel), and `bits` and `counts` are already clear.
cudaError_t rank_roots(const Imgs& I, const BatchTotals& t, const Forest& f, int lo, int hi, int* rank,
                       unsigned* bits, size_t bits_bytes, int* block_tmp, int* wpre, int* counts, cudaStream_t s,
                       const unsigned* skip = nullptr, bool pdl = false);
// The counts of rank_roots alone (no ranks), into `counts` that are already clear.  `bits` receives
// the global roots' bits (scratch, not cleared first).
cudaError_t count_roots(const Imgs& I, const BatchTotals& t, const Forest& f, int lo, int hi, unsigned* bits,
                        int* counts, cudaStream_t s, const unsigned* skip, bool pdl);
constexpr int kBlockPx = 1024;

// The counting half of rank_roots for any bitmap of the images' pixels: per 1024-px block the
// set bits before it in its image (block_tmp, exclusive scan) and per 32-px word the set bits
// before it in its block (wpre).  A set bit's rank is then bit_rank().
cudaError_t rank_bits(const Imgs& I, const BatchTotals& t, const unsigned* bits, int* block_tmp, int* wpre,
                      cudaStream_t s);

// Bits of pixels p .. p+31 (the bitmap has a spare word at the end).
__device__ __forceinline__ unsigned bits_at(const unsigned* bits, int p) {
  const int w = p >> 5, sh = p & 31;
  const unsigned lo = __ldcg(bits + w);
  return sh ? __funnelshift_r(lo, __ldcg(bits + w + 1), sh) : lo;
}

// Rank of pixel p (a set bit) among the set bits of a single image, after rank_bits.
__device__ __forceinline__ int bit_rank(const unsigned* bits, const int* block_tmp, const int* wpre, int p) {
  const int b = p / kBlockPx, j = (p % kBlockPx) >> 5;
  const int w0 = b * kBlockPx + 32 * j;
  int c = __ldcg(block_tmp + b) + __ldcg(wpre + 32 * b + j);
  if (p > w0) c += __popc(bits_at(bits, w0) & ((1u << (p - w0)) - 1u));
  return c;
}

}  // namespace ccl
}  // namespace nsgb
