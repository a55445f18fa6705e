// The operations of the reconstruction / labelling path and their C ABI (include/nsgb.h).
// Each operation is a short sequence of kernels on the caller's stream, using only the
// caller's workspace.  All kernels take an image table (batch.cuh); a single-image call is a
// batch of one whose image is passed by value.  Reference functions are cited at each entry
// point.
#include <cuda_runtime.h>
#include <limits.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include <cmath>
#include <limits>
#include <type_traits>
#include <algorithm>
#include <vector>

#include "../../include/nsgb.h"
#include "batch.cuh"
#include "bbox.cuh"
#include "bitfill.cuh"
#include "ccl.cuh"
#include "common.cuh"
#include "edt.cuh"
#include "fillstart.cuh"
#include "morph.cuh"
#include "recon.cuh"

namespace nsgb {
namespace {

// ------------------------------------------------------------------------------------------
// Pixel access helpers.
template <typename T>
__device__ __forceinline__ T px(const void* base, int64_t pitch, int y, int x) {
  return __ldg((const T*)((const char*)base + (int64_t)y * pitch) + x);
}
template <typename T>
__device__ __forceinline__ T pxcg(const void* base, int64_t pitch, int y, int x) {
  return __ldcg((const T*)((const char*)base + (int64_t)y * pitch) + x);
}
// A plain load, for planes an earlier launch wrote: unlike the one above it can be batched with
// its neighbours by the compiler (32 rows of a labelling tile in flight at once).
template <typename T>
__device__ __forceinline__ T pxw(const void* base, int64_t pitch, int y, int x) {
  return *((const T*)((const char*)base + (int64_t)y * pitch) + x);
}
template <typename T>
__device__ __forceinline__ T* pxp(void* base, int64_t pitch, int y, int x) {
  return (T*)((char*)base + (int64_t)y * pitch) + x;
}

// ------------------------------------------------------------------------------------------
// `x > thr` with thr a double, as OpenCV's `Mat > k` compares (HistologicalEntities.cpp:214),
// without double arithmetic on the device: an integer image compares with floor(thr) (x > thr
// for integer x); a float image with thr converted to float (rounded to nearest), since
// OpenCV's compare converts the scalar to the image's depth.  Both are prepared on the host.
template <typename T>
struct GtThr {
  using K = std::conditional_t<std::is_floating_point<T>::value, float, int>;
  K k;        // integers: the smallest value above the threshold
  bool none;  // integers: nothing is above it
  static GtThr make(double thr) {
    GtThr g;
    g.none = false;
    if constexpr (std::is_floating_point<T>::value) {
      g.k = (float)thr;
    } else {
      const double f = floor(thr);
      g.none = !(f < (double)INT_MAX);  // NaN: nothing is greater
      g.k = g.none ? INT_MAX : f < (double)INT_MIN ? INT_MIN : (int)f + 1;
    }
    return g;
  }
  __device__ __forceinline__ bool operator()(T x) const {
    if constexpr (std::is_floating_point<T>::value) return x > k;
    else return (int)x >= k && !none;
  }
};

// ------------------------------------------------------------------------------------------
// Classifiers (class 0 = background; equal non-zero classes are joined).  They read the
// image's plane (Img::plane) or aux plane.
struct ClsValueU8 {  // bwlabel: the pixel value
  static constexpr ccl::ClassKind kKind = ccl::kAnyClass;
  __device__ uint32_t operator()(const Img& m, int y, int x) const { return px<uint8_t>(m.plane, m.pitch, y, x); }
};
struct ClsNotFlooded {  // a batch's filled image: the pixels the flood from outside did not reach
  static constexpr ccl::ClassKind kKind = ccl::kRowBits;
  const uint32_t* flooded;  // bit plane, rows of bit_words(W) words from Img::b_base
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    const uint32_t w = __ldg(flooded + m.b_base + (int64_t)y * ((m.W + 31) / 32) + (x >> 5));
    return ((w >> (x & 31)) & 1u) ^ 1u;
  }
  // columns x .. x + 31 of row y (x a multiple of 32)
  __device__ uint32_t row_bits(const Img& m, int y, int x) const {
    return ~__ldg(flooded + m.b_base + (int64_t)y * ((m.W + 31) / 32) + (x >> 5));
  }
};
struct ClsDenseU8 {  // the chain's filled image F in the workspace (dense, at px_base)
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  const uint8_t* F;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    return __ldg(F + m.px_base + (int64_t)y * m.W + x) != 0 ? 1u : 0u;
  }
};
template <typename T>
struct ClsNonZero {  // binary reconstruction (mask = aux), bwselect (image = plane)
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  bool use_aux;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    return px<T>(use_aux ? m.aux : m.plane, m.pitch, y, x) != (T)0 ? 1u : 0u;
  }
};
template <typename T>
struct ClsNotMax {  // binary hole filling: pixels that are not foreground (max<T>)
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    return px<T>(m.plane, m.pitch, y, x) != std::numeric_limits<T>::max() ? 1u : 0u;
  }
};
template <typename T>
struct ClsAboveOrNot {  // hole filling and labelling at once: 1 where R > thr, 2 elsewhere
  static constexpr ccl::ClassKind kKind = ccl::kTwoClasses;
  GtThr<T> gt;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    return gt(pxw<T>(m.plane, m.pitch, y, x)) ? 1u : 2u;
  }
};
template <typename T>
struct ClsNotAbove {  // hole filling of (R > thr): the complement class !(R > thr); R = plane
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  GtThr<T> gt;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    return gt(pxw<T>(m.plane, m.pitch, y, x)) ? 0u : 1u;
  }
};

// The red-channel valleys of the nucleus-candidate stage, D = rc - R (OpenCV's saturating u8
// Mat subtraction, HistologicalEntities.cpp:199), from the reconstruction R (plane, written by
// an earlier launch) and the image rc it was taken under (aux).
__device__ __forceinline__ uint8_t valley(const Img& m, int y, int x) {
  const int d = (int)px<uint8_t>(m.aux, m.pitch, y, x) - (int)pxw<uint8_t>(m.plane, m.pitch, y, x);
  return (uint8_t)(d > 0 ? d : 0);
}
struct ClsValleyAboveOrNot {  // hole filling and labelling of (D > g1) at once: 1 where D > g1, 2 elsewhere
  static constexpr ccl::ClassKind kKind = ccl::kTwoClasses;
  GtThr<uint8_t> gt;
  __device__ uint32_t operator()(const Img& m, int y, int x) const { return gt(valley(m, y, x)) ? 1u : 2u; }
};
struct ClsValleyAbove {  // bwselect's image D > g2
  static constexpr ccl::ClassKind kKind = ccl::kOneClass;
  GtThr<uint8_t> gt;
  __device__ uint32_t operator()(const Img& m, int y, int x) const { return gt(valley(m, y, x)) ? 1u : 0u; }
};

// Seeds (pixels that flag their component's root).
template <class Cls>
struct SeedBorder {
  Cls cls;
  __device__ bool operator()(const Img& m, int y, int x) const { return cls(m, y, x) != 0u; }
};
template <typename T>
struct SeedBoth {  // a != 0 and b != 0, with a = plane or aux as selected
  bool a_is_plane;
  __device__ bool operator()(const Img& m, int y, int x) const {
    const void* a = a_is_plane ? m.plane : m.aux;
    const void* b = a_is_plane ? m.aux : m.plane;
    return pxcg<T>(a, m.pitch, y, x) != (T)0 && px<T>(b, m.pitch, y, x) != (T)0;
  }
};

// bwselect's seeds in the nucleus-candidate stage: D > g2 on a pixel of a filled component
// (forest LF, areas A) whose area lies in [lo, hi) -- bw2 & bw1_t without writing bw1_t.  A seed
// marks its root in the forest L2 of D > g2.  Four pixels per thread; rc and R come as one 32-bit
// load each where rows allow it (`words`), and few quads hold a pixel above g2 (byte loads and
// the filled component's lookups one pixel after another took 69 us at 4096^2, this 49).
struct CandidateSeeds {
  GtThr<uint8_t> gt;
  const int* LF;
  const int* A;
  int lo, hi;
  const unsigned* outside;  // roots of LF that are not part of the filled image
  bool words;
};
__global__ void candidate_seeds_kernel(Imgs I, int total_rows, const int* __restrict__ L2, CandidateSeeds c,
                                       unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    const uint8_t* rc = (const uint8_t*)m.aux + (int64_t)y * m.pitch + x;
    const uint8_t* rec = (const uint8_t*)m.plane + (int64_t)y * m.pitch + x;
    uint32_t a = 0, b = 0;
    if (c.words && n == 4) {
      a = *(const uint32_t*)rc;
      b = *(const uint32_t*)rec;
    } else {
      for (int k = 0; k < n; ++k) {
        a |= (uint32_t)rc[k] << (8 * k);
        b |= (uint32_t)rec[k] << (8 * k);
      }
    }
    bool sd[4], any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int d = (int)((a >> (8 * k)) & 0xFFu) - (int)((b >> (8 * k)) & 0xFFu);
      sd[k] = k < n && c.gt((uint8_t)(d > 0 ? d : 0));
      any = any || sd[k];
    }
    if (!any) return;
    const int64_t gi = (int64_t)m.px_base + (int64_t)y * m.W + x;
    int rf[4], r[4];
    ccl::roots4_ro(c.LF, gi, n, rf);
    ccl::roots4_ro(L2, gi, n, r);
    bool kept = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == 0 || rf[k] != rf[k - 1]) {
        const int area = rf[k] < 0 || ccl::test_bit(c.outside, rf[k]) ? -1 : __ldg(c.A + rf[k]);
        kept = area >= 0 && area >= c.lo && area < c.hi;
      }
      sd[k] = sd[k] && kept;
      if (sd[k] && r[k] >= 0 && !(k > 0 && sd[k - 1] && r[k - 1] == r[k])) ccl::set_root_bit(bits, r[k]);
    }
  });
}

// ------------------------------------------------------------------------------------------
// Output kernels (row grids over all images; a pixel's root is L[L[i]]).

// Binary hole filling: 0 where the non-foreground pixel's component touches the border.
// Writes the workspace plane F (dense, if given) and the caller's output (single image:
// `out` / `pitch_out`; batch: Img::fill, dense).
// Stores of four consecutive outputs (one vector store when aligned).
__device__ __forceinline__ void store4_u8(uint8_t* p, int n, const uint8_t (&v)[4]) {
  if (n == 4 && (((uintptr_t)p & 3) == 0)) {
    *(uchar4*)p = make_uchar4(v[0], v[1], v[2], v[3]);
  } else {
    for (int k = 0; k < n; ++k) p[k] = v[k];
  }
}
__device__ __forceinline__ void store4_i32(int32_t* p, int n, const int (&v)[4]) {
  if (n == 4 && (((uintptr_t)p & 15) == 0)) {
    *(int4*)p = make_int4(v[0], v[1], v[2], v[3]);
  } else {
    for (int k = 0; k < n; ++k) p[k] = v[k];
  }
}

template <typename TO>
__global__ void fill_out_kernel(Imgs I, int total_rows, const int* __restrict__ L, const unsigned* __restrict__ bits,
                                uint8_t* F, TO* out, int64_t pitch_out, TO fg) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    const int64_t gi = (int64_t)m.px_base + (int64_t)y * m.W + x;
    int r[4];
    ccl::roots4_ro(L, gi, n, r);
    uint8_t f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      f[k] = (k > 0 && r[k] == r[k - 1]) ? f[k - 1] : ((r[k] >= 0 && ccl::test_bit(bits, r[k])) ? 0 : (uint8_t)fg);
    if (F) store4_u8(F + gi, n, f);
    TO* o = nullptr;
    if (!I.d) o = out ? pxp<TO>(out, pitch_out, y, x) : nullptr;
    else if (m.fill) o = (TO*)m.fill + (int64_t)y * m.W + x;
    if (!o) return;
    if constexpr (sizeof(TO) == 1) {
      store4_u8((uint8_t*)o, n, f);
    } else {
      for (int k = 0; k < n; ++k) o[k] = f[k] ? fg : (TO)0;
    }
  });
}

// Bit planes for the chain's hole fill (bitfill.cu): open = 1 where the reconstruction is not
// above the threshold (the class the fill works on), flooded = 0.  One lane per 32-pixel word of
// the planes of all images (a flat walk, so narrow images leave no lane idle).  Where every
// lane's word starts on a 16-byte boundary the lanes load their own words with vector loads;
// otherwise (rows of an odd width start anywhere) the warp loads each lane's word in turn, one
// pixel per lane, and forms it with a ballot: every load then reads consecutive bytes, where
// per-lane scalar loads would touch 32 sectors per instruction.
struct BBase { __device__ int operator()(const Img& m) const { return m.b_base; } };

template <typename T>
__global__ void pack_open_kernel(Imgs I, int total_words, GtThr<T> gt, uint32_t* __restrict__ open,
                                 uint32_t* __restrict__ flooded) {
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x + threadIdx.x - lane; base < total_words; base += stride) {
    const int wi = base + lane;
    const T* row = nullptr;
    int n = 0;
    if (wi < total_words) {
      const Img& m = I.d ? I.d[img_of(I, wi, BBase())] : I.one;
      const int nw = bit_words(m.W);
      const int rel = wi - m.b_base;
      const int y = rel / nw, k = rel - y * nw;
      row = (const T*)((const char*)m.plane + (int64_t)y * m.pitch) + 32 * k;
      n = min(32, m.W - 32 * k);
    }
    uint32_t bits = 0;
    if (__all_sync(NSGB_FULL, n == 0 || (n == 32 && ((uintptr_t)row & 15) == 0))) {
      if (n == 32) {
        constexpr int V = 16 / sizeof(T);
#pragma unroll
        for (int q = 0; q < 32 / V; ++q) {
          const uint4 v = __ldg((const uint4*)row + q);
          T e[V];
          memcpy(e, &v, 16);
#pragma unroll
          for (int j = 0; j < V; ++j) bits |= (gt(e[j]) ? 0u : 1u) << (q * V + j);
        }
      }
    } else {
#pragma unroll 4
      for (int src = 0; src < 32; ++src) {
        const T* r = (const T*)__shfl_sync(NSGB_FULL, (unsigned long long)row, src);
        const int ns = __shfl_sync(NSGB_FULL, n, src);
        const uint32_t b = __ballot_sync(NSGB_FULL, lane < ns && !gt(__ldg(r + lane)));
        if (lane == src) bits = b;
      }
    }
    if (wi < total_words) {
      open[wi] = bits;
      flooded[wi] = 0u;
    }
  }
}

// Binary reconstruction output, in place on the marker (= plane).
template <typename T>
__global__ void binrecon_out_kernel(Imgs I, int total_rows, const int* __restrict__ L,
                                    const unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_pixels(I, total_rows, [&](const Img& m, int y, int x) {
    T* p = pxp<T>(m.plane, m.pitch, y, x);
    if (*p != (T)0) return;
    const int r = ccl::root_of_ro(L, (int64_t)m.px_base + (int64_t)y * m.W + x);
    if (r >= 0 && ccl::test_bit(bits, r)) *p = std::numeric_limits<T>::max();
  });
}

template <typename T>
__global__ void bwselect_out_kernel(Imgs I, int total_rows, void* out, const int* __restrict__ L,
                                    const unsigned* __restrict__ bits) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_pixels(I, total_rows, [&](const Img& m, int y, int x) {
    const T v = px<T>(m.plane, m.pitch, y, x);
    const int r = ccl::root_of_ro(L, (int64_t)m.px_base + (int64_t)y * m.W + x);
    *pxp<T>(out, m.pitch, y, x) = (v != (T)0 && r >= 0 && ccl::test_bit(bits, r)) ? v : (T)0;
  });
}

// Nucleus candidates: 255 on a component of (D > g2) that holds a seed, where rbc is 0
// (bwselect(bw2, bw1_t, 8) & (rbc == 0), HistologicalEntities.cpp:268-271).  L2 is the forest
// of D > g2 (root -1 off it), `bits` its seeded roots.
__global__ void candidates_out_kernel(Imgs I, int total_rows, const int* __restrict__ L2,
                                      const unsigned* __restrict__ bits, const uint8_t* __restrict__ rbc,
                                      uint8_t* out) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    int r[4];
    ccl::roots4_ro(L2, (int64_t)m.px_base + (int64_t)y * m.W + x, n, r);
    const uint8_t* q = rbc + (int64_t)y * m.pitch + x;
    bool sel[4];
    uint8_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sel[k] = (k > 0 && r[k] == r[k - 1]) ? sel[k - 1] : (r[k] >= 0 && ccl::test_bit(bits, r[k]));
      o[k] = (k < n && sel[k] && __ldg(q + k) == 0) ? 255 : 0;
    }
    store4_u8(pxp<uint8_t>(out, m.pitch, y, x), n, o);
  });
}

// Labels out: relabel ? (bg 0, root's rank + 1) : the root's raster index in its image / -1.
// Optional area-filter outputs from the same pass.  rank / A are read-only here: L1-cached
// loads, because a giant component's root is read by every one of its pixels.
// RELABEL: raster rank labels (else root indices); AREA: area-filter outputs (A non-null).
// FILLED: the labelled pixels are the filled image (255, 0 elsewhere); with `outside` (the forest
// of ccl::label_filled) the roots it marks are background too.
struct LabelQuad {
  int lab[4], kept[4];
  uint8_t flat[4], filled[4];
};
template <bool RELABEL, bool AREA, bool FILLED>
__device__ __forceinline__ void label_quad(int (&r)[4], int px_base, const int* __restrict__ rank,
                                           const int* __restrict__ A, int lo, int hi,
                                           const unsigned* __restrict__ outside, LabelQuad& q) {
  if (FILLED) {
    bool out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      out[k] = (k > 0 && r[k] == r[k - 1]) ? out[k - 1] : (r[k] >= 0 && outside && ccl::test_bit(outside, r[k]));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (out[k]) r[k] = -1;
      q.filled[k] = r[k] >= 0 ? 255 : 0;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool same = k > 0 && r[k] == r[k - 1];
    q.lab[k] = same ? q.lab[k - 1]
                    : (RELABEL ? (r[k] < 0 ? 0 : __ldg(&rank[r[k]]) + 1) : (r[k] < 0 ? -1 : r[k] - px_base));
    bool keep = false;
    if (AREA) {
      if (same) {
        keep = q.flat[k - 1] != 0;
      } else {
        const int a = r[k] >= 0 ? __ldg(&A[r[k]]) : 0;
        keep = r[k] >= 0 && a >= lo && a < hi;
      }
    }
    q.flat[k] = keep ? 255 : 0;
    q.kept[k] = keep ? r[k] - px_base : -1;
  }
}

// Single image: explicit output pointers / pitches (`filled` optional); a table of one: Img's.
template <bool RELABEL, bool AREA, bool FILLED = false>
__global__ void label_out_kernel(Imgs I, int total_rows, const int* __restrict__ L, const int* __restrict__ rank,
                                 int32_t* labels, int64_t pitch_labels, const int* __restrict__ A, int lo,
                                 int hi, int32_t* kept_labels, int64_t pitch_kept, uint8_t* flat, int64_t pitch_flat,
                                 const unsigned* __restrict__ outside = nullptr, uint8_t* filled = nullptr,
                                 int64_t pitch_filled = 0) {
  pdl_wait();
  pdl_release();
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    int r[4];
    LabelQuad q;
    ccl::roots4_ro(L, (int64_t)m.px_base + (int64_t)y * m.W + x, n, r);
    label_quad<RELABEL, AREA, FILLED>(r, m.px_base, rank, A, lo, hi, outside, q);
    if (!I.d) {
      if (FILLED && filled) store4_u8(pxp<uint8_t>(filled, pitch_filled, y, x), n, q.filled);
      if (labels) store4_i32(pxp<int32_t>(labels, pitch_labels, y, x), n, q.lab);
      if (AREA && kept_labels) store4_i32(pxp<int32_t>(kept_labels, pitch_kept, y, x), n, q.kept);
      if (AREA && flat) store4_u8(pxp<uint8_t>(flat, pitch_flat, y, x), n, q.flat);
    } else {
      const int64_t li = (int64_t)y * m.W + x;
      if (FILLED && m.fill) store4_u8(m.fill + li, n, q.filled);
      if (m.labels) store4_i32(m.labels + li, n, q.lab);
      if (AREA && m.area) store4_u8(m.area + li, n, q.flat);
    }
  });
}

// The same for a batch, whose outputs are dense: an image is a line of pixels, and every quad of
// it is aligned in the label plane (px_base is a multiple of 4, or the quads are read one by one:
// see batch_totals) and in outputs that start aligned,
// whatever the width -- row by row an odd width left three rows of four to scalar accesses (47
// Mpixel of uneven u8 tiles: 211 us row by row, 98 us along the line).  A CTA takes kLineBlocks
// consecutive rank blocks of 1024 pixels and looks its image up once.
constexpr int kLineBlocks = 4;
template <bool RELABEL, bool AREA, bool FILLED>
__global__ void __launch_bounds__(ccl::kBlockPx / 4) label_line_kernel(Imgs I, int nblocks, const int* __restrict__ L,
                                                                       const int* __restrict__ rank,
                                                                       const int* __restrict__ A, int lo, int hi) {
  pdl_wait();
  pdl_release();
  const int b0 = blockIdx.x * kLineBlocks, b1 = min(nblocks, b0 + kLineBlocks);
  int ii = img_of(I, b0, BlkBase());
  for (int b = b0; b < b1; ++b) {
    while (ii + 1 < I.n && b >= I.d[ii + 1].blk_base) ++ii;
    const Img& m = I.d[ii];
    const int px_base = m.px_base;
    const int64_t at = (int64_t)(b - m.blk_base) * ccl::kBlockPx + 4 * threadIdx.x;
    const int64_t left = (int64_t)m.H * m.W - at;
    if (left <= 0) continue;
    const int n = (int)min((int64_t)4, left);
    int r[4];
    LabelQuad q;
    ccl::roots4_ro(L, px_base + at, n, r);
    label_quad<RELABEL, AREA, FILLED>(r, px_base, rank, A, lo, hi, nullptr, q);
    if (FILLED && m.fill) store4_u8(m.fill + at, n, q.filled);
    if (m.labels) store4_i32(m.labels + at, n, q.lab);
    if (AREA && m.area) store4_u8(m.area + at, n, q.flat);
  }
}

// Area of arbitrary int32 labels in [-1, n): dense histogram (background -1 skipped).
__global__ void label_hist_kernel(Imgs I, int total_rows, int* __restrict__ A, int* status) {
  ccl::for_batch_pixels(I, total_rows, [&](const Img& m, int y, int x) {
    const int64_t n = (int64_t)m.H * m.W;
    const int l = px<int32_t>(m.plane, m.pitch, y, x);
    if (l == -1) return;
    if (l < -1 || (int64_t)l >= n) {
      set_status(status, NSGB_ERR_BAD_ARG);
      return;
    }
    atomicAdd(&A[l], 1);
  });
}

__global__ void labeled_area_out_kernel(Imgs I, int total_rows, const int* __restrict__ A, int lo, int hi,
                                        int32_t* kept_labels, int64_t pitch_kept, uint8_t* flat, int64_t pitch_flat) {
  ccl::for_batch_pixels(I, total_rows, [&](const Img& m, int y, int x) {
    const int64_t n = (int64_t)m.H * m.W;
    const int l = px<int32_t>(m.plane, m.pitch, y, x);
    const int a = (l >= 0 && (int64_t)l < n) ? __ldg(&A[l]) : 0;
    const bool keep = l >= 0 && (int64_t)l < n && a >= lo && a < hi;
    if (kept_labels) *pxp<int32_t>(kept_labels, pitch_kept, y, x) = keep ? l : -1;
    if (flat) *pxp<uint8_t>(flat, pitch_flat, y, x) = keep ? 255 : 0;
  });
}

__global__ void count_labels_in_range_kernel(const int* __restrict__ A, int64_t n, int lo, int hi, int* out) {
  int c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int a = __ldcg(&A[i]);
    if (a > 0 && a >= lo && a < hi) ++c;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(NSGB_FULL, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ------------------------------------------------------------------------------------------
// Elementwise kernels on one image (row / column grids).
#define NSGB_FOR_PIXELS                                   \
  const int x = blockIdx.x * blockDim.x + threadIdx.x;    \
  if (x >= W) return;                                     \
  for (int y = blockIdx.y; y < H; y += gridDim.y)

template <typename T>
struct alignas(4 * sizeof(T)) Vec4 {
  T v[4];
};

// Four pixels per thread (x grid over W / 4); VEC: rows and bases allow one vector load and
// one 32-bit store per thread.
#define NSGB_FOR_QUADS                                        \
  const int x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);  \
  if (x >= W) return;                                         \
  for (int y = blockIdx.y; y < H; y += gridDim.y)

template <typename T, bool VEC>
__global__ void threshold_kernel(const T* in, int64_t pitch_in, uint8_t* out, int64_t pitch_out, int H, int W,
                                 GtThr<T> gt) {
  NSGB_FOR_QUADS {
    const T* r = (const T*)((const char*)in + (int64_t)y * pitch_in) + x;
    uint8_t* o = out + (int64_t)y * pitch_out + x;
    if (VEC && x + 4 <= W) {
      const Vec4<T> v = *(const Vec4<T>*)r;
      uchar4 q;
      q.x = gt(v.v[0]) ? 255 : 0;
      q.y = gt(v.v[1]) ? 255 : 0;
      q.z = gt(v.v[2]) ? 255 : 0;
      q.w = gt(v.v[3]) ? 255 : 0;
      *(uchar4*)o = q;
    } else {
      for (int k = 0; k < 4 && x + k < W; ++k) o[k] = gt(r[k]) ? 255 : 0;
    }
  }
}

// 8- and 16-bit images whose rows allow it: 16 bytes of pixels per thread (four pixels per thread
// took 205 us at 16384^2 u8, this 103).
template <typename T>
__global__ void threshold_wide_kernel(const T* in, int64_t pitch_in, uint8_t* out, int64_t pitch_out, int H, int W,
                                      GtThr<T> gt) {
  constexpr int V = 16 / sizeof(T);
  const int x = V * (blockIdx.x * blockDim.x + threadIdx.x);
  if (x >= W) return;
  for (int y = blockIdx.y; y < H; y += gridDim.y) {
    const T* r = (const T*)((const char*)in + (int64_t)y * pitch_in) + x;
    uint8_t* o = out + (int64_t)y * pitch_out + x;
    if (x + V <= W) {
      const uint4 v = *(const uint4*)r;
      T e[V];
      memcpy(e, &v, 16);
      uint32_t q[V / 4];
#pragma unroll
      for (int k = 0; k < V / 4; ++k)
        q[k] = (gt(e[4 * k]) ? 0xFFu : 0u) | (gt(e[4 * k + 1]) ? 0xFF00u : 0u) | (gt(e[4 * k + 2]) ? 0xFF0000u : 0u) |
               (gt(e[4 * k + 3]) ? 0xFF000000u : 0u);
      if constexpr (V == 16) *(uint4*)o = make_uint4(q[0], q[1], q[2], q[3]);
      else *(uint2*)o = make_uint2(q[0], q[1]);
    } else {
      for (int k = 0; k < V && x + k < W; ++k) o[k] = gt(r[k]) ? 255 : 0;
    }
  }
}

template <typename T>
__device__ __forceinline__ T invert_value(T v) {
  if constexpr (std::numeric_limits<T>::is_integer) {
    if constexpr (std::numeric_limits<T>::is_signed) {
      return v == std::numeric_limits<T>::min() ? std::numeric_limits<T>::max() : (T)(-v);
    } else {
      return (T)(std::numeric_limits<T>::max() - v);
    }
  } else {
    return (T)0 - v;  // OpenCV's `-img` is `0 - img`: +0.0 for both zeros
  }
}

// -0.0 -> +0.0 over a float plane.  The reference's float imhmin and imfillHoles end with
// PixelOperations::invert (`0 - x`, never -0.0); the order-reversed reconstruction here flips
// the sign bit instead, so their outputs pass through this once.
// VEC: rows allow one 16-byte load per thread; the store is rare.
template <bool VEC>
__global__ void canon_zero_f32_kernel(float* out, int64_t pitch, int H, int W) {
  NSGB_FOR_QUADS {
    unsigned* o = (unsigned*)((char*)out + (int64_t)y * pitch) + x;
    if (VEC && x + 4 <= W) {
      const uint4 v = *(const uint4*)o;
      if (v.x != 0x80000000u && v.y != 0x80000000u && v.z != 0x80000000u && v.w != 0x80000000u) continue;
    }
    for (int k = 0; k < 4 && x + k < W; ++k)
      if (o[k] == 0x80000000u) o[k] = 0u;
  }
}

template <typename T, bool VEC>
__global__ void invert_kernel(const T* in, T* out, int64_t pitch, int H, int W) {
  NSGB_FOR_QUADS {
    const T* r = (const T*)((const char*)in + (int64_t)y * pitch) + x;
    T* o = (T*)((char*)out + (int64_t)y * pitch) + x;
    if (VEC && x + 4 <= W) {
      Vec4<T> v = *(const Vec4<T>*)r;
#pragma unroll
      for (int k = 0; k < 4; ++k) v.v[k] = invert_value(v.v[k]);
      *(Vec4<T>*)o = v;
    } else {
      for (int k = 0; k < 4 && x + k < W; ++k) o[k] = invert_value(r[k]);
    }
  }
}

inline dim3 quad_grid(int64_t rows, int64_t cols) { return ccl::quadrow_grid((int)rows, (int)cols); }

void canon_zero(void* out, int64_t rows, int64_t cols, int64_t pitch, cudaStream_t s) {
  if ((uintptr_t)out % 16 == 0 && pitch % 16 == 0)
    canon_zero_f32_kernel<true><<<quad_grid(rows, cols), 256, 0, s>>>((float*)out, pitch, (int)rows, (int)cols);
  else
    canon_zero_f32_kernel<false><<<quad_grid(rows, cols), 256, 0, s>>>((float*)out, pitch, (int)rows, (int)cols);
}

// h-minima marker: image + h, saturating for integers (h truncated), h rounded to float for float.
// Four pixels per thread, one vector load and store where the rows allow it (a load and a store
// per pixel took 49 us at 4096^2 f32).
template <typename T>
using HminH = std::conditional_t<std::is_floating_point<T>::value, T, int64_t>;
// (Within 62 bits: a conversion beyond the type is undefined, and the sum with a pixel has to fit.  NaN is no h.)
template <typename T>
HminH<T> hmin_h(double h) {
  if constexpr (std::is_floating_point<T>::value) return (T)h;
  else return h != h ? 0 : (int64_t)std::min(std::max(h, -0x1p62), 0x1p62);
}
template <typename T>
__device__ __forceinline__ T hmin_value(T v, HminH<T> h) {
  if constexpr (std::numeric_limits<T>::is_integer) {
    const int64_t s = (int64_t)v + h;
    return (T)(s > (int64_t)std::numeric_limits<T>::max() ? (int64_t)std::numeric_limits<T>::max() : s);
  } else {
    return v + h;
  }
}
template <typename T, bool VEC>
__global__ void hmin_marker_kernel(const T* image, T* out, int64_t pitch, int H, int W, HminH<T> h) {
  NSGB_FOR_QUADS {
    const T* r = (const T*)((const char*)image + (int64_t)y * pitch) + x;
    T* o = (T*)((char*)out + (int64_t)y * pitch) + x;
    if (VEC && x + 4 <= W) {
      Vec4<T> v = *(const Vec4<T>*)r;
#pragma unroll
      for (int k = 0; k < 4; ++k) v.v[k] = hmin_value(v.v[k], h);
      *(Vec4<T>*)o = v;
    } else {
      for (int k = 0; k < 4 && x + k < W; ++k) o[k] = hmin_value(r[k], h);
    }
  }
}

template <typename T>
__global__ void fill_const_kernel(T* out, int64_t pitch, int H, int W, T v) {
  NSGB_FOR_PIXELS { *pxp<T>(out, pitch, y, x) = v; }
}

// ------------------------------------------------------------------------------------------
// Plans and workspace.

struct Plan {
  Imgs I;
  BatchTotals t;
};

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Fills the labelling / rank / row fields of `m` and advances the running totals.
void add_image(Img& m, BatchTotals& t) {
  m.c_tiles_x = (m.W + ccl::kTile - 1) / ccl::kTile;
  const int c_tiles_y = (m.H + ccl::kTile - 1) / ccl::kTile;
  m.r_tile_base = t.r_tiles;
  m.r_stile_base = t.r_stiles;
  m.r_even_base = t.r_even;
  for (int c = 0; c < 3; ++c) m.r_col_base[c] = t.r_col[c];
  m.c_tile_base = t.c_tiles;
  if (!t.tight) t.px = (t.px + 3) & ~(int64_t)3;  // four pixels of an image's label plane are one aligned load
  m.px_base = (int)t.px;
  m.blk_base = t.blocks;
  m.row_base = t.rows;
  m.b_base = (int)t.b_words;
  m.f_tile_base = t.f_tiles;
  const int64_t npx = (int64_t)m.H * m.W;
  t.b_words += (int64_t)m.H * bit_words(m.W);
  t.f_tiles += flood_tiles_x(m.W) * flood_tiles_y(m.H);
  t.r_tiles += m.r_tiles_x * m.r_tiles_y;
  if (m.r_tw > 0) t.r_stiles += ((m.H + 47) / 32) * ((m.W + m.r_tw / 2 + m.r_tw - 1) / m.r_tw);
  t.r_even += even_tiles(m.r_tiles_x, m.r_tiles_y);
  for (int c = 0; c < 3; ++c) t.r_col[c] += colour_tiles(m.r_tiles_x, m.r_tiles_y, c);
  t.c_tiles += m.c_tiles_x * c_tiles_y;
  t.px += npx;
  t.blocks += (int)((npx + ccl::kBlockPx - 1) / ccl::kBlockPx);
  t.rows += m.H;
  if (m.W > t.max_w) t.max_w = m.W;
  if (2 * (m.H + m.W) > t.perimeter_max) t.perimeter_max = 2 * (m.H + m.W);
  t.n += 1;
}

Plan single_plan(int dtype, void* plane, const void* aux, int64_t H, int64_t W, int64_t pitch) {
  Plan P = {};
  P.I.n = 1;
  P.I.d = nullptr;
  P.I.one = recon_image(dtype, plane, aux, H, W, pitch);
  add_image(P.I.one, P.t);
  return P;
}

struct WsSizes {
  size_t recon, L, A, R, roots, bits, tmp, wpre, F, table, maps, total;
};

WsSizes ws_sizes(const BatchTotals& t) {
  WsSizes z;
  z.recon = align256(recon_workspace_bytes_tiles(t.r_tiles > 0 ? t.r_tiles : 1));
  z.L = align256(sizeof(int) * (size_t)t.px);
  z.A = z.L;
  z.R = z.L;
  z.roots = z.L;
  z.bits = align256(sizeof(unsigned) * (size_t)(t.px / 32 + 2));
  z.tmp = align256(sizeof(int) * (size_t)(2 * (int64_t)t.blocks + 2 * (int64_t)t.n + 8));
  z.wpre = align256(sizeof(int) * 32 * (size_t)t.blocks);
  z.F = align256((size_t)t.px);
  z.table = t.n > 1 ? align256(sizeof(Img) * (size_t)t.n) : 0;
  z.maps = t.n > 1 ? align256(sizeof(int) * ((size_t)t.r_tiles + (size_t)t.c_tiles)) : 0;
  z.total = z.recon + z.L + z.A + z.R + z.roots + z.bits + z.tmp + z.wpre + z.F + z.table + z.maps;
  return z;
}

struct Ws {
  int* status;  // == start of the recon region
  void* recon;
  int* L;
  int* A;
  int* R;        // root ranks (at roots)
  int* roots;    // list of local roots
  unsigned* bits;
  int* tmp;      // 2 ints per rank block
  int* counts;   // 2 per image
  int* nroots;   // [1]
  int* wpre;     // 32 per rank block
  uint8_t* F;
  Img* table;
  int* r_img;  // batches: image of every reconstruction tile
  int* c_img;  // batches: image of every labelling tile
  size_t bits_bytes;
  ccl::Forest forest(bool areas) const { return ccl::Forest{L, areas ? A : nullptr, roots, nroots}; }
};

Ws carve(void* ws, const BatchTotals& t) {
  const WsSizes z = ws_sizes(t);
  char* p = (char*)ws;
  Ws w;
  w.status = (int*)p;
  w.recon = p;
  p += z.recon;
  w.L = (int*)p;
  p += z.L;
  w.A = (int*)p;
  p += z.A;
  w.R = (int*)p;
  p += z.R;
  w.roots = (int*)p;
  p += z.roots;
  w.bits = (unsigned*)p;
  w.bits_bytes = sizeof(unsigned) * (size_t)(t.px / 32 + 2);
  p += z.bits;
  w.tmp = (int*)p;
  w.counts = w.tmp + 2 * (int64_t)t.blocks;
  w.nroots = w.counts + 2 * (int64_t)t.n;
  p += z.tmp;
  w.wpre = (int*)p;
  p += z.wpre;
  w.F = (uint8_t*)p;
  p += z.F;
  w.table = t.n > 1 ? (Img*)p : nullptr;
  p += z.table;
  w.r_img = t.n > 1 ? (int*)p : nullptr;
  w.c_img = t.n > 1 ? w.r_img + t.r_tiles : nullptr;
  return w;
}

inline int grid1d(int64_t n) { return ccl::flat_grid(n); }
inline dim3 rc(int64_t rows, int64_t cols) { return ccl::rowcol_grid((int)rows, (int)cols); }
inline dim3 qr(int64_t rows, int64_t cols) { return ccl::quadrow_grid((int)rows, (int)cols); }
inline dim3 qrb(const BatchTotals& t) { return ccl::quadrow_grid(t.rows, t.max_w); }

// Ranges that the labelling's first launch clears for a call: the status word, the bitmap, and
// (optional) the counts.
ccl::ZeroSpans call_spans(const Ws& w, bool bits, int counts) {
  return ccl::ZeroSpans{{nullptr, (unsigned*)w.status, w.bits, (unsigned*)w.counts},
                        {0, 1, bits ? (int)(w.bits_bytes / sizeof(unsigned)) : 0, counts}};
}

// Records the caller's optional timing event around the reconstruction kernel.  While the
// stream is being captured into a CUDA graph the record becomes an external event-record node,
// so the event is recorded at every replay (a plain record in a capture only orders streams).
cudaError_t record(const nsgb_opts* o, bool begin, cudaStream_t s) {
  if (!o) return cudaSuccess;
  void* ev = begin ? o->recon_event_begin : o->recon_event_end;
  if (!ev) return cudaSuccess;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) return e;
  return cap == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags((cudaEvent_t)ev, s, cudaEventRecordExternal)
                                              : cudaEventRecord((cudaEvent_t)ev, s);
}

// Reconstruction of the whole plan bracketed by the optional timing events.
cudaError_t recon_timed(const nsgb_opts* o, int dtype, const Plan& P, int conn, bool erode, bool ring, void* ws,
                        cudaStream_t s, int resweeps = 0) {
  cudaError_t e = record(o, true, s);
  if (e != cudaSuccess) return e;
  e = recon_launch_batch(dtype, P.I, P.t.r_tiles, conn, erode, ring, ws, s, o ? o->max_visits_per_tile : 0,
                         o ? o->max_visit_iters : 0, resweeps, o ? o->queue_poll_limit : 0, o ? o->recon_passes : 0,
                         P.t.r_stiles, o ? o->recon_order : 0, (long long)P.t.px, o ? o->recon_ctas_per_sm : 0);
  if (e != cudaSuccess) return e;
  return record(o, false, s);
}

template <typename F>
void dispatch_all(int dtype, F&& f) {
  switch (dtype) {
    case NSGB_U8: f((uint8_t*)nullptr); break;
    case NSGB_U16: f((uint16_t*)nullptr); break;
    case NSGB_I32: f((int32_t*)nullptr); break;
    case NSGB_F32: f((float*)nullptr); break;
    default: break;
  }
}

template <typename F>
cudaError_t dispatch_int(int dtype, F&& f) {
  switch (dtype) {
    case NSGB_U8: return f((uint8_t*)nullptr);
    case NSGB_U16: return f((uint16_t*)nullptr);
    case NSGB_I32: return f((int32_t*)nullptr);
    default: return cudaErrorInvalidValue;
  }
}

// Image table of `n` equally sized images `stride` bytes apart (image 0 = proto).
__global__ void stack_table_kernel(Img proto, int n, int64_t stride, BatchTotals one, Img* table) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Img m = proto;
  m.plane = (void*)((uintptr_t)proto.plane + (uintptr_t)(i * stride));
  m.aux = (const void*)((uintptr_t)proto.aux + (uintptr_t)(i * stride));
  m.r_tile_base = i * one.r_tiles;
  m.r_stile_base = i * one.r_stiles;
  m.r_even_base = i * even_tiles(proto.r_tiles_x, proto.r_tiles_y);
  for (int c = 0; c < 3; ++c) m.r_col_base[c] = i * colour_tiles(proto.r_tiles_x, proto.r_tiles_y, c);
  m.c_tile_base = i * one.c_tiles;
  m.px_base = (int)(i * one.px);
  m.blk_base = i * one.blocks;
  m.row_base = i * one.rows;
  m.b_base = (int)(i * one.b_words);
  m.f_tile_base = i * one.f_tiles;
  table[i] = m;
}

// Totals of `n` stacked copies of one image's plan.
BatchTotals stacked_totals(const BatchTotals& one, int64_t n) {
  BatchTotals t = one;
  t.n = (int)n;
  t.px = one.px * n;
  t.r_tiles = (int)(one.r_tiles * n);
  t.r_stiles = (int)(one.r_stiles * n);
  t.r_even = (int)(one.r_even * n);
  for (int c = 0; c < 3; ++c) t.r_col[c] = (int)(one.r_col[c] * n);
  t.c_tiles = (int)(one.c_tiles * n);
  t.blocks = (int)(one.blocks * n);
  t.rows = (int)(one.rows * n);
  t.b_words = one.b_words * n;
  t.f_tiles = (int)(one.f_tiles * n);
  return t;
}

// ------------------------------------------------------------------------------------------
// The single-tile / batched chain on a prepared plan: (a) reconstruction in place,
// (b)+(c) threshold fused into the binary hole fill, (d)+(e) one labelling of the filled image
// for both the raster relabel and the areas.  Counts land in w.counts (2 per image).
cudaError_t chain_impl(int dtype, const Plan& P, const Ws& w, int recon_conn, double thr, int fill_conn,
                       int label_conn, int area_min, int area_max, uint8_t* fill_out, int32_t* labels_out,
                       uint8_t* area_out, const nsgb_opts* opts, cudaStream_t s) {
  const BatchTotals& t = P.t;
  cudaError_t e = recon_timed(opts, dtype, P, recon_conn, false, dtype == NSGB_I32, w.recon, s);
  const bool dual = (fill_conn == 4 && label_conn == 8) || (fill_conn == 8 && label_conn == 4);
  if (e == cudaSuccess && dual && !(P.I.d && t.n > 1)) {
    // (b)-(e) on one image with one labelling.  With dual connectivities (the not-above class
    // flooded 4-connected, the filled image labelled 8-connected, or the other way round) the
    // components of R > thr and of its complement form a tree by enclosure, and a component of
    // the filled image is a top-level component of R > thr with everything it encloses: both
    // classes are labelled in one forest, each component joined to its parent (the component
    // above its first pixel) unless that is a complement component touching the border.  The
    // bitmap of those outside components lives in F, which this path does not otherwise use.
    unsigned* outside = (unsigned*)w.F;
    const int code = label_conn == 8 ? ccl::kConnFg8Bg4 : ccl::kConnFg4Bg8;
    e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
      using T = std::remove_pointer_t<decltype(tag)>;
      // the ranking's bitmap and counts are cleared by the labelling's first launch
      const ccl::ZeroSpans rank_zero{{nullptr, nullptr, w.bits, (unsigned*)w.counts},
                                     {0, 0, (int)(w.bits_bytes / sizeof(unsigned)), 2 * t.n}};
      return ccl::label_filled(ClsAboveOrNot<T>{GtThr<T>::make(thr)}, P.I, t, code, w.forest(true), outside,
                               w.bits_bytes, s, true, rank_zero);
    });
    // From the labelling on, every launch is a programmatic dependent of the one before it.
    if (e == cudaSuccess)
      e = ccl::rank_roots(P.I, t, w.forest(true), area_min, area_max, w.R, w.bits, w.bits_bytes, w.tmp, w.wpre,
                          w.counts, s, outside, true);
    if (e == cudaSuccess) {
      const int64_t W1 = P.I.d ? 0 : P.I.one.W;
      e = launch_dependent(label_out_kernel<true, true, true>, qrb(t), dim3(256), s, P.I, t.rows, (const int*)w.L,
                           (const int*)w.R, labels_out, W1 * 4, (const int*)w.A, area_min, area_max,
                           (int32_t*)nullptr, (int64_t)0, area_out, W1, (const unsigned*)outside, fill_out, W1);
    }
    return e;
  }
  if (e == cudaSuccess && P.I.d && t.n > 1) {
    // (b)-(e) on a batch: the pixels not above the threshold as a bit plane, flooded from
    // outside each image (bitfill.cu); the filled image is what the flood does not reach, and
    // it is labelled straight from the flooded plane, the label output writing it out.  The
    // planes L and R hold the open and flooded bit planes until the labelling (L) and the rank
    // (R) overwrite them.  A flood is a chain of dependent tile visits from the border inwards;
    // many images flood at once, so the batch hides that latency, and it then costs a fraction
    // of the labelling (pack and flood touch 1 bit per pixel where a labelling writes an int).
    uint32_t* open = (uint32_t*)w.L;
    uint32_t* flooded = (uint32_t*)w.R;
    e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
      using T = std::remove_pointer_t<decltype(tag)>;
      pack_open_kernel<T><<<ccl::flat_grid(t.b_words), 256, 0, s>>>(P.I, (int)t.b_words, GtThr<T>::make(thr), open,
                                                                   flooded);
      return cudaGetLastError();
    });
    if (e == cudaSuccess)
      e = flood_launch(P.I, t.f_tiles, open, flooded, fill_conn, w.recon, s, opts ? opts->queue_poll_limit : 0);
    if (e == cudaSuccess) {
      // (the flooded plane lies in R, which the ranking overwrites after the labelling; the bitmap
      // and the counts are cleared by the labelling's first launch)
      ccl::ZeroSpans z = call_spans(w, true, 2 * t.n);
      z.n[1] = 0;  // the status holds the reconstruction's
      e = ccl::label(ClsNotFlooded{flooded}, P.I, t, label_conn, w.forest(true), s, z);
    }
    if (e == cudaSuccess)
      e = ccl::rank_roots(P.I, t, w.forest(true), area_min, area_max, w.R, w.bits, w.bits_bytes, w.tmp, w.wpre,
                          w.counts, s, nullptr, true);
    if (e == cudaSuccess)
      e = launch_dependent(label_line_kernel<true, true, true>, dim3((t.blocks + kLineBlocks - 1) / kLineBlocks),
                           dim3(ccl::kBlockPx / 4), s, P.I, t.blocks, (const int*)w.L, (const int*)w.R,
                           (const int*)w.A, area_min, area_max);
    return e;
  }
  if (e == cudaSuccess) {
    // (b)+(c) on one image: the threshold fused into the labelling's classifier, components
    // touching the border seeded.  (One image's flood is a chain of dependent tile visits that
    // the labelling does not have: 0.58 against 0.49 ms for the 4096^2 chain.)
    e = cudaMemsetAsync(w.bits, 0, w.bits_bytes, s);
    if (e == cudaSuccess) {
      e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
        using T = std::remove_pointer_t<decltype(tag)>;
        ClsNotAbove<T> cls{GtThr<T>::make(thr)};
        cudaError_t r = ccl::label(cls, P.I, t, fill_conn, w.forest(false), s);
        if (r != cudaSuccess) return r;
        const int gx = grid1d(t.perimeter_max) > 64 ? 64 : grid1d(t.perimeter_max);
        ccl::ccl_seed_border<SeedBorder<ClsNotAbove<T>>><<<dim3(gx, t.n), 256, 0, s>>>(
            P.I, w.L, SeedBorder<ClsNotAbove<T>>{cls}, w.bits);
        fill_out_kernel<uint8_t><<<qrb(t), 256, 0, s>>>(P.I, t.rows, w.L, w.bits, w.F, fill_out,
                                                        P.I.d ? 0 : (int64_t)P.I.one.W, (uint8_t)255);
        return cudaGetLastError();
      });
    }
  }
  if (e == cudaSuccess) e = ccl::label(ClsDenseU8{w.F}, P.I, t, label_conn, w.forest(true), s);
  if (e == cudaSuccess) e = ccl::rank_roots(P.I, t, w.forest(true), area_min, area_max, w.R, w.bits, w.bits_bytes, w.tmp, w.wpre, w.counts, s);
  if (e == cudaSuccess) {
    const int64_t W1 = P.I.d ? 0 : P.I.one.W;
    label_out_kernel<true, true><<<qrb(t), 256, 0, s>>>(P.I, t.rows, w.L, w.R, labels_out, W1 * 4, w.A, area_min,
                                                        area_max, nullptr, 0, area_out, W1);
    e = cudaGetLastError();
  }
  return e;
}

// Quads of an image's rows start on 4-byte boundaries in both planes (u8).
bool words_ok(const Img& m) {
  return ((uintptr_t)m.plane % 4) == 0 && ((uintptr_t)m.aux % 4) == 0 && m.pitch % 4 == 0;
}

// The nucleus-candidate stage on one image (plane = rc_open, reconstructed in place; aux = rc):
// (a) R = recon(rc_open, rc, 8); (b) bw1 = imfillHoles(D > g1, 4) and (c) bw1's 8-connected
// components with their areas, from one labelling of D > g1 and its complement (the threshold
// in the classifier), the kept ones counted (w.counts[1]); (d) bwselect(D > g2, bw1_t, 8): D > g2 labelled into a second
// forest (the rank array R, unused here), its roots seeded straight from bw1's forest and
// areas, so bw1_t is never written; (e) the output with rbc == 0 folded in.
cudaError_t candidates_impl(const Plan& P, const Ws& w, double g1, double g2, int lo, int hi, const uint8_t* rbc,
                            uint8_t* out, const nsgb_opts* opts, cudaStream_t s) {
  const BatchTotals& t = P.t;
  const GtThr<uint8_t> gt1 = GtThr<uint8_t>::make(g1);
  const GtThr<uint8_t> gt2 = GtThr<uint8_t>::make(g2);
  cudaError_t e = recon_timed(opts, NSGB_U8, P, 8, false, false, w.recon, s);
  // (b)+(c) as one labelling of D > g1 (8-connected) and its complement (4-connected), each
  // component joined to the one enclosing it (ccl::label_filled); the complement components
  // that touch the border are marked in F (used as a bitmap here) and are not part of bw1.
  unsigned* outside = (unsigned*)w.F;
  if (e == cudaSuccess)
    e = ccl::label_filled(ClsValleyAboveOrNot{gt1}, P.I, t, ccl::kConnFg8Bg4, w.forest(true), outside,
                          w.bits_bytes, s, true, ccl::ZeroSpans{{nullptr, nullptr, (unsigned*)w.counts, nullptr}, {0, 0, 2 * t.n, 0}});
  if (e == cudaSuccess)
    e = ccl::count_roots(P.I, t, w.forest(true), lo, hi, w.bits, w.counts, s, outside, true);
  const ccl::Forest sel{w.R, nullptr, w.roots, w.nroots};
  ccl::ZeroSpans z = call_spans(w, true, 0);
  z.n[1] = 0;  // the status holds the reconstruction's
  if (e == cudaSuccess) e = ccl::label(ClsValleyAbove{gt2}, P.I, t, 8, sel, s, z);
  if (e == cudaSuccess)
    e = launch_dependent(candidate_seeds_kernel, qrb(t), dim3(256), s, P.I, t.rows, (const int*)w.R,
                         CandidateSeeds{gt2, w.L, w.A, lo, hi, outside, words_ok(P.I.one)}, w.bits);
  if (e == cudaSuccess)
    e = launch_dependent(candidates_out_kernel, qrb(t), dim3(256), s, P.I, t.rows, (const int*)w.R,
                         (const unsigned*)w.bits, rbc, out);
  return e;
}

// The image of every reconstruction tile and of every labelling tile: blockIdx.y walks the images.
__global__ void batch_maps_kernel(const Img* __restrict__ table, int n, int* __restrict__ r_img, int* __restrict__ c_img) {
  for (int i = blockIdx.y; i < n; i += gridDim.y) {
    const Img& m = table[i];
    const int nr = m.r_tiles_x * m.r_tiles_y, nc = m.c_tiles_x * ((m.H + ccl::kTile - 1) / ccl::kTile);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nr; k += gridDim.x * blockDim.x) r_img[m.r_tile_base + k] = i;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) c_img[m.c_tile_base + k] = i;
  }
}

}  // namespace
}  // namespace nsgb

// ============================================================================================
// C ABI
using namespace nsgb;

namespace {

bool want_sync(const nsgb_opts* o) { return o == nullptr || o->sync != 0; }

nsgb_status cuda_status(cudaError_t e) { return e == cudaSuccess ? NSGB_OK : NSGB_ERR_CUDA; }

// Finishes a call: reports launch errors; with sync, waits and reports the device status.  With
// `n` > 0 the counts (n words of the workspace, which may start with the status) are read too, sync or not.  Status
// and counts come in one strided copy where the distance allows it: each copy to pageable memory
// is a round trip of its own (about 8 us).
nsgb_status finish(cudaError_t e, const void* ws, cudaStream_t s, const nsgb_opts* o, const int* counts = nullptr,
                   int n = 0, int32_t* to = nullptr) {
  if (e != cudaSuccess) return NSGB_ERR_CUDA;
  e = cudaGetLastError();
  if (e != cudaSuccess) return NSGB_ERR_CUDA;
  if (n == 0 && !want_sync(o)) return NSGB_OK;
  constexpr int kRow = 32;
  const int64_t apart = n > 0 ? (const char*)counts - (const char*)ws : 0;
  int32_t both[2][kRow] = {};
  if (n > 0 && n <= kRow && apart >= (int64_t)sizeof(int) * kRow && apart < (int64_t)INT_MAX) {
    e = cudaMemcpy2DAsync(both, sizeof(both[0]), ws, (size_t)apart, sizeof(int) * (size_t)n, 2, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) memcpy(to, both[1], sizeof(int) * (size_t)n);
  } else {
    if (n > 0) e = cudaMemcpyAsync(to, counts, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && (n == 0 || apart != 0))
      e = cudaMemcpyAsync(&both[0][0], ws, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (n > 0 && apart == 0) both[0][0] = to[0];
  }
  if (e != cudaSuccess) return NSGB_ERR_CUDA;
  return want_sync(o) ? (nsgb_status)both[0][0] : NSGB_OK;
}

nsgb_status check_ws_bytes(void* ws, size_t ws_bytes, size_t need) {
  if (!ws) return NSGB_ERR_WORKSPACE;
  if (ws_bytes < need) return NSGB_ERR_WORKSPACE;
  if ((uintptr_t)ws % 256 != 0) return NSGB_ERR_WORKSPACE;
  return NSGB_OK;
}

nsgb_status check_ws(void* ws, size_t ws_bytes, int op, int dtype, int64_t rows, int64_t cols) {
  return check_ws_bytes(ws, ws_bytes, nsgb_workspace_size(op, dtype, rows, cols));
}

}  // namespace

extern "C" {

size_t nsgb_workspace_size(int op, int dtype, int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0 || op < 0 || op > NSGB_OP_DISTANCE) return 0;
  if (op == NSGB_OP_BWLABEL || op == NSGB_OP_BWAREAOPEN || op == NSGB_OP_NUCLEUS_CANDIDATES ||
      op == NSGB_OP_MORPH_OPEN || op == NSGB_OP_DISTANCE)
    dtype = NSGB_U8;
  if (dtype < 0 || dtype > 3) return 0;
  if (op == NSGB_OP_IMRECONSTRUCT || op == NSGB_OP_HMIN) return align256(recon_workspace_bytes(dtype, rows, cols));
  if (op == NSGB_OP_BOUNDING_BOX) return align256(bbox_workspace_bytes(rows * cols));
  if (op == NSGB_OP_MORPH_OPEN) return align256(morph_open_workspace_bytes(rows, cols));
  if (op == NSGB_OP_DISTANCE) return align256(edt_workspace_bytes(rows, cols));
  const Plan P = single_plan(dtype, nullptr, nullptr, rows, cols, cols * elem_size(dtype));
  return ws_sizes(P.t).total;
}

const char* nsgb_status_string(int status) {
  switch (status) {
    case NSGB_OK: return "ok";
    case NSGB_ERR_BAD_ARG: return "bad argument";
    case NSGB_ERR_UNSUPPORTED_DTYPE: return "unsupported dtype for this operation";
    case NSGB_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
    case NSGB_ERR_NOT_CONVERGED: return "iteration budget exhausted before convergence";
    case NSGB_ERR_TIMEOUT: return "a bounded device-side wait timed out";
    case NSGB_ERR_CUDA: return "CUDA runtime error";
    case NSGB_ERR_QUEUE_OVERFLOW: return "device work list overflow";
    default: return "unknown status";
  }
}

nsgb_status nsgb_device_status(const void* ws, nsgb_stream_t stream) {
  if (!ws) return NSGB_ERR_WORKSPACE;
  int v = 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(&v, ws, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return NSGB_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return NSGB_ERR_CUDA;
  return (nsgb_status)v;
}

nsgb_status nsgb_imreconstruct(int dtype, void* marker, const void* mask, int64_t rows, int64_t cols, int64_t pitch,
                               int conn, int erode, void* ws, size_t ws_bytes, nsgb_stream_t stream,
                               const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!marker || !mask || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_IMRECONSTRUCT, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const bool ring = !erode && (dtype == NSGB_I32 || dtype == NSGB_F32);
  const Plan P = single_plan(dtype, marker, mask, rows, cols, pitch);
  cudaError_t e = recon_timed(opts, dtype, P, conn, erode != 0, ring, ws, s);
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_imreconstruct_binary(int dtype, void* marker, const void* mask, int64_t rows, int64_t cols,
                                      int64_t pitch, int conn, void* ws, size_t ws_bytes, nsgb_stream_t stream,
                                      const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (dtype == NSGB_F32) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!marker || !mask || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_IMRECONSTRUCT_BINARY, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(dtype, marker, mask, rows, cols, pitch);
  Ws w = carve(ws, P.t);
  cudaError_t e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
    using T = std::remove_pointer_t<decltype(tag)>;
    cudaError_t r = ccl::label(ClsNonZero<T>{true}, P.I, P.t, conn, w.forest(false), s, call_spans(w, true, 0));
    if (r == cudaSuccess)
      r = launch_dependent(ccl::ccl_seed_pixels<SeedBoth<T>>, rc(rows, cols), dim3(256), s, P.I, P.t.rows,
                           (const int*)w.L, SeedBoth<T>{true}, w.bits);
    if (r == cudaSuccess)
      r = launch_dependent(binrecon_out_kernel<T>, rc(rows, cols), dim3(256), s, P.I, P.t.rows, (const int*)w.L,
                           (const unsigned*)w.bits);
    return r;
  });
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_imfill_holes(int dtype, const void* image, void* out, int64_t rows, int64_t cols, int64_t pitch,
                              int binary, int conn, void* ws, size_t ws_bytes, nsgb_stream_t stream,
                              const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!image || !out || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  if (binary && dtype == NSGB_F32) return NSGB_ERR_UNSUPPORTED_DTYPE;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_FILL_HOLES, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const int H = (int)rows, W = (int)cols;
  const Plan P = single_plan(dtype, (void*)image, nullptr, rows, cols, pitch);
  Ws w = carve(ws, P.t);
  cudaError_t e = cudaSuccess;
  if (binary) {
    if (dtype == NSGB_I32) {
      // min<int> is non-zero, so the reference's binary reconstruction has no background to
      // grow into and every pixel comes back as invert(min<int>) = INT_MAX.
      e = cudaMemsetAsync(w.status, 0, sizeof(int), s);
      if (e != cudaSuccess) return NSGB_ERR_CUDA;
      fill_const_kernel<int32_t><<<rc(rows, cols), 256, 0, s>>>((int32_t*)out, pitch, H, W, INT_MAX);
      return finish(cudaGetLastError(), ws, s, opts);
    }
    e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
      using T = std::remove_pointer_t<decltype(tag)>;
      ClsNotMax<T> cls;
      cudaError_t r = ccl::label(cls, P.I, P.t, conn, w.forest(false), s, call_spans(w, true, 0));
      if (r == cudaSuccess)
        r = launch_dependent(ccl::ccl_seed_border<SeedBorder<ClsNotMax<T>>>, dim3(grid1d(2 * (rows + cols)), 1),
                             dim3(256), s, P.I, (const int*)w.L, SeedBorder<ClsNotMax<T>>{cls}, w.bits);
      if (r == cudaSuccess)
        r = launch_dependent(fill_out_kernel<T>, qr(rows, cols), dim3(256), s, P.I, P.t.rows, (const int*)w.L,
                             (const unsigned*)w.bits, (uint8_t*)nullptr, (T*)out, pitch, std::numeric_limits<T>::max());
      return r;
    });
    return finish(e, ws, s, opts);
  }
  // Grayscale: erosion reconstruction of (image on the border, max inside) above the image.
  if (out == image) return NSGB_ERR_BAD_ARG;
  e = fill_start_launch(dtype, P.I, P.t.c_tiles, w.forest(false), w.bits, w.bits_bytes, w.F, out, conn, s);
  if (e != cudaSuccess) return NSGB_ERR_CUDA;
  const Plan R = single_plan(dtype, out, image, rows, cols, pitch);
  // front from the border: re-sweep a tile up to four times when a neighbour changed while it
  // ran (16384^2 fills, 8-connected: 11.76 -> 11.53 ms u8, 18.48 -> 17.93 ms i32 against two)
  e = recon_timed(opts, dtype, R, conn, true, false, ws, s, 4);
  if (e == cudaSuccess && dtype == NSGB_F32) {
    canon_zero(out, rows, cols, pitch, s);
    e = cudaGetLastError();
  }
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_imhmin(int dtype, const void* image, void* out, int64_t rows, int64_t cols, int64_t pitch, double h,
                        int conn, void* ws, size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz || dtype == NSGB_I32) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!image || !out || out == image || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) ||
      !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_HMIN, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const int H = (int)rows, W = (int)cols;
  const bool vec = ((uintptr_t)image % (4 * esz)) == 0 && ((uintptr_t)out % (4 * esz)) == 0 && pitch % (4 * esz) == 0;
  dispatch_all(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const auto hh = hmin_h<T>(h);
    if (vec) hmin_marker_kernel<T, true><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)image, (T*)out, pitch, H, W, hh);
    else hmin_marker_kernel<T, false><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)image, (T*)out, pitch, H, W, hh);
  });
  // invert(recon(invert(I) - h, invert(I))): the order-reversed reconstruction with the
  // reference's 0-valued padding ring taken in the inverted domain.
  const Plan P = single_plan(dtype, out, image, rows, cols, pitch);
  cudaError_t e = recon_timed(opts, dtype, P, conn, true, true, ws, s);
  if (e == cudaSuccess && dtype == NSGB_F32) {
    canon_zero(out, rows, cols, pitch, s);
    e = cudaGetLastError();
  }
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_bwselect(int dtype, const void* image, const void* seeds, void* out, int64_t rows, int64_t cols,
                          int64_t pitch, int conn, void* ws, size_t ws_bytes, nsgb_stream_t stream,
                          const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz || dtype == NSGB_F32) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!image || !seeds || !out || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_BWSELECT, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(dtype, (void*)image, seeds, rows, cols, pitch);
  Ws w = carve(ws, P.t);
  cudaError_t e = dispatch_int(dtype, [&](auto* tag) -> cudaError_t {
    using T = std::remove_pointer_t<decltype(tag)>;
    cudaError_t r = ccl::label(ClsNonZero<T>{false}, P.I, P.t, conn, w.forest(false), s, call_spans(w, true, 0));
    // seeds (aux) != 0 and image (plane) != 0
    if (r == cudaSuccess)
      r = launch_dependent(ccl::ccl_seed_pixels<SeedBoth<T>>, rc(rows, cols), dim3(256), s, P.I, P.t.rows,
                           (const int*)w.L, SeedBoth<T>{false}, w.bits);
    if (r == cudaSuccess)
      r = launch_dependent(bwselect_out_kernel<T>, rc(rows, cols), dim3(256), s, P.I, P.t.rows, out, (const int*)w.L,
                           (const unsigned*)w.bits);
    return r;
  });
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_bwlabel(const uint8_t* bin, int32_t* labels, int64_t rows, int64_t cols, int64_t pitch_in,
                         int64_t pitch_labels, int conn, int relabel, int32_t* count, void* ws, size_t ws_bytes,
                         nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!bin || !labels || !valid_dims(rows, cols) || !valid_pitch(pitch_in, cols, 1) ||
      !valid_pitch(pitch_labels, cols, 4) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_BWLABEL, NSGB_U8, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(NSGB_U8, (void*)bin, nullptr, rows, cols, pitch_in);
  Ws w = carve(ws, P.t);
  cudaError_t e = ccl::label(ClsValueU8{}, P.I, P.t, conn, w.forest(false), s, call_spans(w, true, 2));
  if (e == cudaSuccess)
    e = ccl::rank_roots(P.I, P.t, w.forest(false), 0, 0, w.R, w.bits, w.bits_bytes, w.tmp, w.wpre, w.counts, s, nullptr,
                        true);
  if (e == cudaSuccess)
    e = launch_dependent(relabel ? label_out_kernel<true, false> : label_out_kernel<false, false>, qr(rows, cols),
                         dim3(256), s, P.I, P.t.rows, (const int*)w.L, (const int*)w.R, labels, pitch_labels,
                         (const int*)nullptr, 0, 0, (int32_t*)nullptr, (int64_t)0, (uint8_t*)nullptr, (int64_t)0,
                         (const unsigned*)nullptr, (uint8_t*)nullptr, (int64_t)0);
  return finish(e, ws, s, opts, w.counts, count ? 1 : 0, count);
}

nsgb_status nsgb_bwareaopen(const void* in, int labeled, int32_t* labels_out, uint8_t* flat_out, int64_t rows,
                            int64_t cols, int64_t pitch_in, int64_t pitch_labels, int64_t pitch_flat, int32_t min_size,
                            int32_t max_size, int conn, int32_t* count, void* ws, size_t ws_bytes,
                            nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!in || !valid_dims(rows, cols) || !valid_pitch(pitch_in, cols, labeled ? 4 : 1) || !valid_conn(conn))
    return NSGB_ERR_BAD_ARG;
  if (labels_out && !valid_pitch(pitch_labels, cols, 4)) return NSGB_ERR_BAD_ARG;
  if (flat_out && !valid_pitch(pitch_flat, cols, 1)) return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_BWAREAOPEN, NSGB_U8, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t n = rows * cols;
  const Plan P = single_plan(NSGB_U8, (void*)in, nullptr, rows, cols, pitch_in);
  Ws w = carve(ws, P.t);
  cudaError_t e = cudaSuccess;
  if (!labeled) {
    e = ccl::label(ClsValueU8{}, P.I, P.t, conn, w.forest(true), s, call_spans(w, true, 2));
    if (e == cudaSuccess)
      e = ccl::rank_roots(P.I, P.t, w.forest(true), min_size, max_size, w.R, w.bits, w.bits_bytes, w.tmp, w.wpre, w.counts,
                          s, nullptr, true);
    if (e == cudaSuccess)
      e = launch_dependent(label_out_kernel<false, true>, qr(rows, cols), dim3(256), s, P.I, P.t.rows, (const int*)w.L,
                           (const int*)w.R, (int32_t*)nullptr, (int64_t)0, (const int*)w.A, min_size, max_size, labels_out,
                           pitch_labels, flat_out, pitch_flat, (const unsigned*)nullptr, (uint8_t*)nullptr, (int64_t)0);
    return finish(e, ws, s, opts, w.counts + 1, count ? 1 : 0, count);
  }
  e = cudaMemsetAsync(w.status, 0, sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.A, 0, sizeof(int) * (size_t)n, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.counts, 0, 2 * sizeof(int), s);
  if (e == cudaSuccess) {
    label_hist_kernel<<<rc(rows, cols), 256, 0, s>>>(P.I, P.t.rows, w.A, w.status);
    count_labels_in_range_kernel<<<grid1d(n), 256, 0, s>>>(w.A, n, min_size, max_size, w.counts + 1);
    labeled_area_out_kernel<<<rc(rows, cols), 256, 0, s>>>(P.I, P.t.rows, w.A, min_size, max_size, labels_out,
                                                            pitch_labels, flat_out, pitch_flat);
    e = cudaGetLastError();
  }
  return finish(e, ws, s, opts, w.counts + 1, count ? 1 : 0, count);
}

nsgb_status nsgb_bounding_boxes(const int32_t* labels, int64_t rows, int64_t cols, int64_t pitch, int32_t bgval,
                                int32_t* boxes, int64_t capacity, int32_t* count, int32_t* count_dev, void* ws,
                                size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!labels || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, 4) || capacity < 0 || (capacity > 0 && !boxes))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_BOUNDING_BOX, NSGB_I32, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(NSGB_I32, (void*)labels, nullptr, rows, cols, pitch);
  cudaError_t e = bbox_launch(P.I, P.t, bgval, ws, boxes, capacity, count_dev, s);
  // the count sits in the header, two words behind the status
  int32_t head[3] = {};
  const nsgb_status r = finish(e, ws, s, opts, (const int*)ws, count ? 3 : 0, head);
  if (count && r != NSGB_ERR_CUDA) *count = head[2];
  return r;
}

nsgb_status nsgb_morph_open(const uint8_t* in, uint8_t* out, int64_t rows, int64_t cols, int64_t pitch_in,
                            int64_t pitch_out, const uint8_t* kernel, int k, void* ws, size_t ws_bytes,
                            nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!in || !out || !valid_dims(rows, cols) || !valid_pitch(pitch_in, cols, 1) || !valid_pitch(pitch_out, cols, 1))
    return NSGB_ERR_BAD_ARG;
  MorphElement e;
  if (!morph_element(kernel, k, &e)) return NSGB_ERR_BAD_ARG;
  const char *a0 = (const char*)in, *a1 = a0 + (rows - 1) * pitch_in + cols;
  const char *b0 = (const char*)out, *b1 = b0 + (rows - 1) * pitch_out + cols;
  if (a0 < b1 && b0 < a1) return NSGB_ERR_BAD_ARG;  // out overlaps in
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_MORPH_OPEN, NSGB_U8, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e2 = cudaMemsetAsync(ws, 0, sizeof(int), s);
  if (e2 == cudaSuccess)
    e2 = morph_open_launch(in, pitch_in, out, pitch_out, (int)rows, (int)cols, e, (uint8_t*)ws + 256, s);
  return finish(e2, ws, s, opts);
}

nsgb_status nsgb_distance_transform(const uint8_t* mask, float* out, int64_t rows, int64_t cols, int64_t pitch_in,
                                    int64_t pitch_out, int basins, void* ws, size_t ws_bytes, nsgb_stream_t stream,
                                    const nsgb_opts* opts) {
  if (!mask || !out || !valid_dims(rows, cols) || !valid_pitch(pitch_in, cols, 1) || !valid_pitch(pitch_out, cols, 4) ||
      rows > 65535LL * 128)
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_DISTANCE, NSGB_U8, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(ws, 0, sizeof(int), s);
  if (e == cudaSuccess) e = edt_launch(mask, pitch_in, out, pitch_out, (int)rows, (int)cols, basins != 0, ws, s);
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_nucleus_candidates(uint8_t* rc_open, const uint8_t* rc, const uint8_t* rbc, uint8_t* seg_out,
                                    int64_t rows, int64_t cols, int64_t pitch, double g1, double g2,
                                    int32_t area_min, int32_t area_max, int32_t* n_kept, int32_t* n_kept_dev,
                                    void* ws, size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!rc_open || !rc || !rbc || !seg_out || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, 1))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_NUCLEUS_CANDIDATES, NSGB_U8, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(NSGB_U8, rc_open, rc, rows, cols, pitch);
  Ws w = carve(ws, P.t);
  cudaError_t e = candidates_impl(P, w, g1, g2, area_min, area_max, rbc, seg_out, opts, s);
  if (e == cudaSuccess && n_kept_dev)
    e = cudaMemcpyAsync(n_kept_dev, w.counts + 1, sizeof(int32_t), cudaMemcpyDeviceToDevice, s);
  return finish(e, ws, s, opts, w.counts + 1, n_kept ? 1 : 0, n_kept);
}

nsgb_status nsgb_threshold(int dtype, const void* in, uint8_t* out, int64_t rows, int64_t cols, int64_t pitch_in,
                           int64_t pitch_out, double thr, nsgb_stream_t stream) {
  const int esz = elem_size(dtype);
  if (!esz) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!in || !out || !valid_dims(rows, cols) || !valid_pitch(pitch_in, cols, esz) || !valid_pitch(pitch_out, cols, 1))
    return NSGB_ERR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int H = (int)rows, W = (int)cols;
  const bool vec = ((uintptr_t)in % (4 * esz)) == 0 && pitch_in % (4 * esz) == 0 && ((uintptr_t)out % 4) == 0 &&
                   pitch_out % 4 == 0;
  dispatch_all(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const GtThr<T> gt = GtThr<T>::make(thr);
    if constexpr (sizeof(T) <= 2) {
      constexpr int V = 16 / sizeof(T);
      if ((uintptr_t)in % 16 == 0 && pitch_in % 16 == 0 && (uintptr_t)out % V == 0 && pitch_out % V == 0) {
        const dim3 grid((unsigned)((cols + 256 * V - 1) / (256 * V)), ccl::row_blocks(H));
        threshold_wide_kernel<T><<<grid, 256, 0, s>>>((const T*)in, pitch_in, out, pitch_out, H, W, gt);
        return;
      }
    }
    if (vec) threshold_kernel<T, true><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)in, pitch_in, out, pitch_out, H, W, gt);
    else threshold_kernel<T, false><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)in, pitch_in, out, pitch_out, H, W, gt);
  });
  return cuda_status(cudaGetLastError());
}

nsgb_status nsgb_invert(int dtype, const void* in, void* out, int64_t rows, int64_t cols, int64_t pitch,
                        nsgb_stream_t stream) {
  const int esz = elem_size(dtype);
  if (!esz) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!in || !out || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz)) return NSGB_ERR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int H = (int)rows, W = (int)cols;
  const bool vec = ((uintptr_t)in % (4 * esz)) == 0 && ((uintptr_t)out % (4 * esz)) == 0 && pitch % (4 * esz) == 0;
  dispatch_all(dtype, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if (vec) invert_kernel<T, true><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)in, (T*)out, pitch, H, W);
    else invert_kernel<T, false><<<quad_grid(rows, cols), 256, 0, s>>>((const T*)in, (T*)out, pitch, H, W);
  });
  return cuda_status(cudaGetLastError());
}

nsgb_status nsgb_chain(int dtype, void* marker, const void* mask, int64_t rows, int64_t cols, int64_t pitch,
                       int recon_conn, double thr, int fill_conn, int label_conn, int32_t area_min, int32_t area_max,
                       uint8_t* fill_out, int32_t* labels_out, uint8_t* area_out, int32_t* n_labels, int32_t* n_kept,
                       void* ws, size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  const int esz = elem_size(dtype);
  if (!esz || dtype == NSGB_F32) return NSGB_ERR_UNSUPPORTED_DTYPE;
  if (!marker || !mask || !valid_dims(rows, cols) || !valid_pitch(pitch, cols, esz) || !valid_conn(recon_conn) ||
      !valid_conn(fill_conn) || !valid_conn(label_conn))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws(ws, ws_bytes, NSGB_OP_CHAIN, dtype, rows, cols);
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P = single_plan(dtype, marker, mask, rows, cols, pitch);
  Ws w = carve(ws, P.t);
  cudaError_t e = chain_impl(dtype, P, w, recon_conn, thr, fill_conn, label_conn, area_min, area_max, fill_out,
                             labels_out, area_out, opts, s);
  int32_t c[2] = {0, 0};
  const nsgb_status r = finish(e, ws, s, opts, w.counts, n_labels || n_kept ? 2 : 0, c);
  if (r != NSGB_ERR_CUDA) {
    if (n_labels) *n_labels = c[0];
    if (n_kept) *n_kept = c[1];
  }
  return r;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Batches.  nsgb_batch_prepare writes the image table into the workspace once and fills the
// caller's nsgb_batch (host copy of the totals); nsgb_chain_batch / nsgb_imreconstruct_batch
// then only enqueue kernels and memsets (plus small count reads when asked for).

namespace {

// `tight`: without alignment of the images in the label planes.  A batch takes it when only the
// padding would put it over the limit of 2^31 - 1 pixels (kernels check the alignment they use).
bool batch_totals(int dtype, const nsgb_tile* tiles, int n, std::vector<Img>* imgs, BatchTotals* t,
                  bool tight = false) {
  *t = BatchTotals{};
  t->tight = tight;
  if (imgs) imgs->clear();
  const int esz = elem_size(dtype);
  if (!esz || !tiles || n <= 0) return false;
  for (int i = 0; i < n; ++i) {
    const nsgb_tile& tl = tiles[i];
    if (!tl.marker || !tl.mask || !valid_dims(tl.rows, tl.cols) || !valid_pitch(tl.pitch, tl.cols, esz))
      return false;
    Img m = recon_image(dtype, tl.marker, tl.mask, tl.rows, tl.cols, tl.pitch);
    add_image(m, *t);
    m.fill = tl.fill_out;
    m.labels = tl.labels_out;
    m.area = tl.area_out;
    if (t->px >= (int64_t)INT_MAX) return !tight && batch_totals(dtype, tiles, n, imgs, t, true);
    if (imgs) imgs->push_back(m);
  }
  return true;
}

// Batch workspaces always carry the device table, even for one image.
BatchTotals table_totals(BatchTotals t) {
  if (t.n == 1) t.n = 2;
  return t;
}

nsgb_status batch_plan(const nsgb_batch* b, Plan* P, Ws* w) {
  if (!b || !b->ws) return NSGB_ERR_BAD_ARG;
  BatchTotals t{};
  t.n = b->n;
  t.px = b->total_px;
  t.r_tiles = b->recon_tiles;
  t.c_tiles = b->label_tiles;
  t.blocks = b->rank_blocks;
  t.rows = b->total_rows;
  t.max_w = b->max_cols;
  t.perimeter_max = b->max_perimeter;
  t.f_tiles = b->flood_tiles;
  t.b_words = b->bit_words;
  if (t.n <= 0) return NSGB_ERR_BAD_ARG;
  if (b->ws_bytes < ws_sizes(table_totals(t)).total) return NSGB_ERR_WORKSPACE;
  *w = carve(b->ws, table_totals(t));
  P->t = t;
  P->I = Imgs{};
  P->I.n = t.n;
  P->I.d = w->table;
  P->I.r_img = w->r_img;
  P->I.c_img = w->c_img;
  return NSGB_OK;
}

}  // namespace

extern "C" {

size_t nsgb_batch_workspace_size(int dtype, const nsgb_tile* tiles, int n_tiles) {
  BatchTotals t{};
  if (!batch_totals(dtype, tiles, n_tiles, nullptr, &t)) return 0;
  return ws_sizes(table_totals(t)).total;
}

nsgb_status nsgb_batch_prepare(int dtype, const nsgb_tile* tiles, int n_tiles, void* ws, size_t ws_bytes,
                               nsgb_batch* batch) {
  if (!batch) return NSGB_ERR_BAD_ARG;
  std::vector<Img> imgs;
  BatchTotals t{};
  if (!batch_totals(dtype, tiles, n_tiles, &imgs, &t)) return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws_bytes(ws, ws_bytes, nsgb_batch_workspace_size(dtype, tiles, n_tiles));
  if (st != NSGB_OK) return st;
  Ws w = carve(ws, table_totals(t));
  // Synchronous copy: the host array goes away when this returns.  The tile maps (image of every
  // reconstruction tile, then of every labelling tile) are written on the device from the table.
  if (cudaMemcpy(w.table, imgs.data(), sizeof(Img) * imgs.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return NSGB_ERR_CUDA;
  batch_maps_kernel<<<dim3(8, (unsigned)std::min(t.n, 65535)), 256>>>(w.table, t.n, w.r_img, w.c_img);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(0) != cudaSuccess) return NSGB_ERR_CUDA;
  memset(batch, 0, sizeof(*batch));
  batch->dtype = dtype;
  batch->n = t.n;
  batch->total_px = t.px;
  batch->recon_tiles = t.r_tiles;
  batch->label_tiles = t.c_tiles;
  batch->rank_blocks = t.blocks;
  batch->total_rows = t.rows;
  batch->max_cols = t.max_w;
  batch->max_perimeter = t.perimeter_max;
  batch->flood_tiles = t.f_tiles;
  batch->bit_words = (int)t.b_words;
  batch->ws = ws;
  batch->ws_bytes = ws_bytes;
  return NSGB_OK;
}

nsgb_status nsgb_chain_batch(const nsgb_batch* batch, int recon_conn, double thr, int fill_conn, int label_conn,
                             int32_t area_min, int32_t area_max, int32_t* n_labels, int32_t* n_kept,
                             nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!valid_conn(recon_conn) || !valid_conn(fill_conn) || !valid_conn(label_conn)) return NSGB_ERR_BAD_ARG;
  Plan P;
  Ws w;
  nsgb_status st = batch_plan(batch, &P, &w);
  if (st != NSGB_OK) return st;
  if (batch->dtype == NSGB_F32 || !elem_size(batch->dtype)) return NSGB_ERR_UNSUPPORTED_DTYPE;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = chain_impl(batch->dtype, P, w, recon_conn, thr, fill_conn, label_conn, area_min, area_max,
                             nullptr, nullptr, nullptr, opts, s);
  std::vector<int32_t> c(n_labels || n_kept ? 2 * (size_t)P.t.n : 0);
  const nsgb_status r = finish(e, w.status, s, opts, w.counts, (int)c.size(), c.data());
  for (int i = 0; i < P.t.n && r != NSGB_ERR_CUDA; ++i) {
    if (n_labels) n_labels[i] = c[2 * i];
    if (n_kept) n_kept[i] = c[2 * i + 1];
  }
  return r;
}

nsgb_status nsgb_batch_counts_async(const nsgb_batch* batch, int32_t* counts, nsgb_stream_t stream) {
  Plan P;
  Ws w;
  if (!counts) return NSGB_ERR_BAD_ARG;
  nsgb_status st = batch_plan(batch, &P, &w);
  if (st != NSGB_OK) return st;
  return cuda_status(cudaMemcpyAsync(counts, w.counts, 2 * sizeof(int32_t) * (size_t)P.t.n, cudaMemcpyDefault,
                                     (cudaStream_t)stream));
}

nsgb_status nsgb_imreconstruct_batch(const nsgb_batch* batch, int conn, int erode, nsgb_stream_t stream,
                                     const nsgb_opts* opts) {
  if (!valid_conn(conn)) return NSGB_ERR_BAD_ARG;
  Plan P;
  Ws w;
  nsgb_status st = batch_plan(batch, &P, &w);
  if (st != NSGB_OK) return st;
  if (!elem_size(batch->dtype)) return NSGB_ERR_UNSUPPORTED_DTYPE;
  cudaStream_t s = (cudaStream_t)stream;
  const bool ring = !erode && (batch->dtype == NSGB_I32 || batch->dtype == NSGB_F32);
  cudaError_t e = recon_timed(opts, batch->dtype, P, conn, erode != 0, ring, w.recon, s);
  return finish(e, w.status, s, opts);
}

}  // extern "C"

// ============================================================================================
// Differentiable float32 reconstruction by dilation (an extension: the reference has no
// gradient).  The result only ever copies input values, so each R(p) has one source pixel:
// mask(q) (clamped at q), marker(q), or the zero ring the reference pads around the image
// (MorphologicOperations.cpp:671-674, which can only win on a border pixel, as 0).  A source
// and the pixels that took its value form a plateau (connected, equal R), so the forward
// labels the plateaus of R with the union-find labeller and gives each the best source it
// contains (mask before marker before ring, then the smallest raster index):
//   prov = ~q (mask q), q (marker q), INT32_MIN (ring); q = y * cols + x within the image.
// The adjoint scatters the upstream gradient along prov with exact 128-bit fixed-point sums
// (resolution 2^-96) and rounds each sum to float once.
namespace nsgb {
namespace {

constexpr int kKeyNone = 0x7F7F7F7F;  // memset byte 0x7F: no source seen yet

// Plateau class: all 32 bits of R (+0 and -0 merged), plus one so that no value is background.
struct ClsPlateau {
  static constexpr ccl::ClassKind kKind = ccl::kAnyClass;
  using class_t = uint32_t;
  __device__ uint32_t operator()(const Img& m, int y, int x) const {
    uint32_t v = __float_as_uint(pxw<float>(m.plane, m.pitch, y, x));
    if ((v << 1) == 0u) v = 0u;
    return v + 1u;
  }
};

__device__ __forceinline__ const void* shifted(const void* p, int64_t off) {
  return (const void*)((uintptr_t)p + (uintptr_t)off);
}

// Source key of pixel (y, x) with result r: mask q < marker n + q < ring 2n; kKeyNone if it is no
// source.
__device__ __forceinline__ int source_key(const Img& m, float r, float mask, float marker, int y, int x) {
  const int n = m.H * m.W, q = y * m.W + x;
  if (r == mask) return q;
  if (r == marker) return n + q;
  if (r == 0.0f && (y == 0 || y == m.H - 1 || x == 0 || x == m.W - 1)) return 2 * n;
  return kKeyNone;
}

// Four consecutive floats of a row.
__device__ __forceinline__ void load4(const float* p, int n, bool quads, float (&v)[4]) {
  if (quads && n == 4) {
    const float4 q = *(const float4*)p;
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = p[min(k, n - 1)];
  }
}

// Four pixels per thread; equal roots among them (one plateau) are merged before the atomic.
// plane = R, aux = mask, the marker sits `marker_off` bytes from R in every image.  The three planes
// and the labels come as 16-byte loads where rows allow it (`quads`), all issued together (one
// float after another, each waiting for the one before: 510 us at 16 x 2048^2, this 389).
__global__ void source_best_kernel(Imgs I, int total_rows, int64_t marker_off, const int* __restrict__ L,
                                   int* __restrict__ best, bool quads) {
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    const int64_t at = (int64_t)y * m.pitch + (int64_t)x * 4;
    float rv[4], mask[4], marker[4];
    load4((const float*)((const char*)m.plane + at), n, quads, rv);
    load4((const float*)((const char*)m.aux + at), n, quads, mask);
    load4((const float*)((const char*)shifted(m.plane, marker_off) + at), n, quads, marker);
    int key[4], r[4];
    ccl::roots4_ro(L, (int64_t)m.px_base + (int64_t)y * m.W + x, n, r);
#pragma unroll
    for (int k = 0; k < 4; ++k) key[k] = k < n ? source_key(m, rv[k], mask[k], marker[k], y, x + k) : kKeyNone;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (key[k] == kKeyNone) continue;
      if (k < 3 && r[k + 1] == r[k]) {  // pass the smaller key on to the next pixel of the plateau
        key[k + 1] = min(key[k + 1], key[k]);
        continue;
      }
      if (key[k] < __ldcg(&best[r[k]])) atomicMin(&best[r[k]], key[k]);
    }
  });
}

__global__ void prov_out_kernel(Imgs I, int total_rows, const int* __restrict__ L, const int* __restrict__ best,
                                int64_t prov_off, int* status) {
  ccl::for_batch_quads(I, total_rows, [&](const Img& m, int y, int x, int n) {
    int r[4], p[4];
    ccl::roots4_ro(L, (int64_t)m.px_base + (int64_t)y * m.W + x, n, r);
    const int np = m.H * m.W;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= n) {
        p[k] = INT_MIN;
        continue;
      }
      const int key = (k > 0 && r[k] == r[k - 1]) ? -1 : __ldg(&best[r[k]]);
      if (key < 0) {
        p[k] = p[k - 1];
      } else if (key < np) {
        p[k] = ~key;
      } else if (key < 2 * np) {
        p[k] = key - np;
      } else {
        p[k] = INT_MIN;
        if (key != 2 * np) set_status(status, NSGB_ERR_BAD_ARG);  // a plateau without a source: NaN input
      }
    }
    store4_i32(pxp<int32_t>((void*)shifted(m.plane, prov_off), m.pitch, y, x), n, p);
  });
}

// Exact fixed point for the adjoint: a value is held as a 128-bit two's-complement integer S
// (lo, hi words) standing for S * 2^-96.  Every float32 g with 2^-73 <= |g| < 2^31 converts
// exactly (its last mantissa bit is worth at least 2^-96); smaller magnitudes round to the
// nearest multiple of 2^-96 (ties to even).  Sums of such values are exact as long as they
// stay below 2^31 in magnitude, and the order in which atomics land does not matter.
struct Fix128 {
  unsigned long long lo;
  long long hi;
};

// Returns false for |g| >= 2^31, inf and NaN.
__device__ __forceinline__ bool fix_from_float(float g, Fix128& out) {
  const uint32_t b = __float_as_uint(g);
  const uint32_t ex = (b >> 23) & 0xFFu;
  uint32_t man = b & 0x7FFFFFu;
  if (ex >= 127u + 31u) return false;
  int sh;  // value = man * 2^sh
  if (ex == 0) {
    sh = -149;
  } else {
    man |= 0x800000u;
    sh = (int)ex - 150;
  }
  // fixed = man * 2^(sh + 96)
  unsigned long long lo = 0, hi = 0;
  const int s = sh + 96;
  if (s >= 0) {  // s <= 157 - 150 + 96 = 103, man < 2^24: fits in 127 bits
    if (s < 64) {
      lo = (unsigned long long)man << s;
      hi = s == 0 ? 0ull : (unsigned long long)man >> (64 - s);
    } else {
      hi = (unsigned long long)man << (s - 64);
    }
  } else if (-s < 32) {  // round man * 2^s (ties to even)
    const int r = -s;
    const uint32_t q = man >> r, rem = man & ((1u << r) - 1u), half = 1u << (r - 1);
    lo = q + ((rem > half || (rem == half && (q & 1u))) ? 1u : 0u);
  }
  if (b >> 31) {  // negate: two's complement over 128 bits
    lo = ~lo + 1ull;
    hi = ~hi + (lo == 0ull ? 1ull : 0ull);
  }
  out.lo = lo;
  out.hi = (long long)hi;
  return true;
}

__device__ __forceinline__ Fix128 fix_add(const Fix128& a, const Fix128& b) {
  Fix128 r;
  r.lo = a.lo + b.lo;
  r.hi = a.hi + b.hi + (r.lo < a.lo ? 1ll : 0ll);
  return r;
}

// S * 2^-96 rounded to the nearest float (ties to even).  |S| < 2^127, so the result is a
// normal float or zero (the smallest non-zero magnitude, 2^-96, is far above 2^-126).
__device__ __forceinline__ float fix_to_float(unsigned long long lo, long long hi) {
  const bool neg = hi < 0;
  unsigned long long ml = lo, mh = (unsigned long long)hi;
  if (neg) {
    ml = ~ml + 1ull;
    mh = ~mh + (ml == 0ull ? 1ull : 0ull);
  }
  if ((ml | mh) == 0ull) return 0.0f;
  const int lead = mh ? 127 - __clzll((long long)mh) : 63 - __clzll((long long)ml);  // top set bit
  // 24 significant bits: m = floor(M / 2^(lead - 23)), remainder decides the rounding
  uint32_t m;
  bool above_half = false, exactly_half = false;
  if (lead <= 23) {
    m = (uint32_t)(ml << (23 - lead));
  } else {
    const int r = lead - 23;  // bits dropped, 1..104
    // m = bits [r, r + 24) of (mh:ml)
    unsigned long long q;
    if (r >= 64) q = mh >> (r - 64);
    else q = (ml >> r) | (r == 0 ? 0ull : (mh << (64 - r)));
    m = (uint32_t)q;
    // the dropped bits: half = bit r - 1, sticky = bits below it
    const int hb = r - 1;
    const bool hbit = hb >= 64 ? ((mh >> (hb - 64)) & 1ull) : ((ml >> hb) & 1ull);
    bool sticky;
    if (hb >= 64) sticky = ml != 0ull || (hb > 64 && (mh & ((1ull << (hb - 64)) - 1ull)) != 0ull);
    else sticky = hb > 0 && (ml & ((1ull << hb) - 1ull)) != 0ull;
    above_half = hbit && sticky;
    exactly_half = hbit && !sticky;
  }
  int e = lead - 96;  // value = m * 2^(e - 23)
  if (above_half || (exactly_half && (m & 1u))) {
    ++m;
    if (m == (1u << 24)) {
      m >>= 1;
      ++e;
    }
  }
  const uint32_t bits = ((uint32_t)(e + 127) << 23) | (m & 0x7FFFFFu) | (neg ? 0x80000000u : 0u);
  return __uint_as_float(bits);
}

// The adjoint: grad(q) = exact sum of the gradients of the pixels whose source is q, rounded once.
// Sources are near their pixels (a plateau grows a few pixels around its source), so the sums are
// formed per 32 x 32 tile in shared memory by the CTA that owns the sources, and only pixels whose
// source lies in another tile go through 128-bit accumulators in the workspace:
//   (1) grad_touch: the accumulators such pixels use are zeroed and marked in a bitmap (a small image has
//       all of them zeroed by the first launch instead, and (2) does the marking);
//   (2) grad_far: such pixels add to them (two 64-bit atomics each, runs of one row summed first);
//   (3) grad_tiles: every tile sums its own pixels, adds the marked accumulators, rounds, writes;
//   (4) grad_wide_tiles: the same for tiles whose gradients span too many bits for (3).
// An accumulator for every pixel, zeroed, added to and read back (64 bytes of traffic a pixel
// against the 16 that come in and go out), took 2.1 ms at 16 x 2048^2; this takes 0.9 ms.
struct GradArgs {
  const float* g;
  const int32_t* prov;
  float *dmarker, *dmask;
  int64_t pitch, stride;  // bytes, of all planes
  int H, W, n;            // images of H x W
  int tiles_x, tiles_y;
  unsigned div_mul;  // y = umulhi(q, div_mul) >> div_shift for q = y * W + x < 2^31 (W > 1)
  int div_shift;
  unsigned long long *acc[2];  // two words per pixel: marker sources, mask sources
  unsigned* far_bits[2];       // sources with pixels in other tiles
  int* wide;                   // [0] tiles left to grad_wide_tiles, then their indices
  int* status;
};

template <typename T>
__device__ __forceinline__ T* grad_row(const GradArgs& a, T* base, int img, int y) {
  return (T*)((char*)base + img * a.stride + (int64_t)y * a.pitch);
}

// Source of a pixel: class 0 (marker q) or 1 (mask q), -1 for none (ring, or out of range: reported).
struct GradSource {
  int cls, q, y, x;
};
__device__ __forceinline__ GradSource grad_source(const GradArgs& a, int32_t p) {
  GradSource s = {-1, 0, 0, 0};
  if (p == INT_MIN) return s;
  s.q = p >= 0 ? p : ~p;
  if ((int64_t)s.q >= (int64_t)a.H * a.W) return s;
  s.cls = p >= 0 ? 0 : 1;
  s.y = a.W > 1 ? (int)(__umulhi((unsigned)s.q, a.div_mul) >> a.div_shift) : s.q;
  s.x = s.q - s.y * a.W;
  return s;
}

constexpr int kGradTile = 32;
__device__ __forceinline__ bool other_tile(const GradSource& s, int y, int x) {
  return ((s.y ^ y) | (s.x ^ x)) >= kGradTile;
}

// Four pixels per thread (grid: columns, rows, images).
template <bool VEC>
__global__ void __launch_bounds__(128) grad_touch_kernel(GradArgs a) {
  const int x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (x >= a.W) return;
  for (int img = blockIdx.z; img < a.n; img += gridDim.z) {
    for (int y = blockIdx.y; y < a.H; y += gridDim.y) {
      const int32_t* row = grad_row(a, a.prov, img, y) + x;
      int32_t p[4];
      if (VEC && x + 4 <= a.W) {
        const int4 v = __ldg((const int4*)row);
        p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) p[k] = x + k < a.W ? __ldg(row + k) : INT_MIN;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const GradSource s = grad_source(a, p[k]);
        if (s.cls < 0 || !other_tile(s, y, x + k) || (k > 0 && p[k] == p[k - 1] && (x + k) % kGradTile)) continue;
        const int64_t gq = (int64_t)img * a.H * a.W + s.q;
        const unsigned bit = 1u << (gq & 31);
        unsigned* word = a.far_bits[s.cls] + (gq >> 5);
        if (__ldcg(word) & bit) continue;  // set after its accumulator was zeroed, or about to be
        *(ulonglong2*)(a.acc[s.cls] + 2 * gq) = make_ulonglong2(0ull, 0ull);
        atomicOr(word, bit);
      }
    }
  }
}

// Lanes of a warp hold consecutive pixels of one row, which mostly share a source: a segmented
// warp scan sums runs of equal targets first, so only the last lane of each run issues the atomics
// (low word, then the high word with the low word's carry).  Four rows per thread, their sources
// loaded together; a warp without a far pixel in a row skips the row.
constexpr int kFarRows = 4;
template <bool MARK>
__global__ void __launch_bounds__(128) grad_far_kernel(GradArgs a) {
  pdl_wait();
  pdl_release();
  const int lane = threadIdx.x & 31;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  for (int img = blockIdx.z; img < a.n; img += gridDim.z) {
    for (int y0 = blockIdx.y * kFarRows; y0 < a.H; y0 += gridDim.y * kFarRows) {  // uniform per block
      int32_t p[kFarRows];
#pragma unroll
      for (int r = 0; r < kFarRows; ++r)
        p[r] = x < a.W && y0 + r < a.H ? __ldg(grad_row(a, a.prov, img, y0 + r) + x) : INT_MIN;
#pragma unroll 1
      for (int r = 0; r < kFarRows; ++r) {
        const int y = y0 + r;
        const int32_t pr = r == 0 ? p[0] : r == 1 ? p[1] : r == 2 ? p[2] : p[3];
        const GradSource s = grad_source(a, pr);
        const bool far = s.cls >= 0 && other_tile(s, y, x);
        if (!__any_sync(NSGB_FULL, far)) continue;
        long long key = -1;
        Fix128 v = {0ull, 0ll};
        if (far && fix_from_float(__ldg(grad_row(a, a.g, img, y) + x), v))
          key = ((int64_t)img * a.H * a.W + s.q) | ((long long)s.cls << 40);
        else
          v = Fix128{0ull, 0ll};
        const long long kprev = __shfl_up_sync(NSGB_FULL, key, 1);
        const long long knext = __shfl_down_sync(NSGB_FULL, key, 1);
        bool head = lane == 0 || kprev != key || key < 0;
#pragma unroll 1
        for (int o = 1; o < 32 && !__all_sync(NSGB_FULL, head); o <<= 1) {
          Fix128 v2;
          v2.lo = __shfl_up_sync(NSGB_FULL, v.lo, o);
          v2.hi = __shfl_up_sync(NSGB_FULL, v.hi, o);
          const bool h2 = __shfl_up_sync(NSGB_FULL, head, o);
          if (lane >= o && !head) {
            v = fix_add(v, v2);
            head = h2;
          }
        }
        const bool tail = lane == 31 || knext != key;
        if (tail && key >= 0) {
          const int64_t gq = key & ((1ll << 40) - 1);
          unsigned long long* q = a.acc[key >> 40] + 2 * gq;
          if (MARK) atomicOr(a.far_bits[key >> 40] + (gq >> 5), 1u << (gq & 31));
          const unsigned long long old = atomicAdd(q, v.lo);
          const unsigned long long carry = old + v.lo < old ? 1ull : 0ull;
          atomicAdd(q + 1, (unsigned long long)v.hi + carry);
        }
      }
    }
  }
}

// A tile's pixels: position, source and gradient (kept in registers by both tile kernels).
constexpr int kGradPx = kGradTile * kGradTile;
constexpr int kGradThreads = 256;
constexpr int kGradRows = kGradTile / (kGradThreads / 32);  // rows per thread
struct GradTileAt {
  int img, x0, y0;
  int64_t px0;
};
__device__ __forceinline__ GradTileAt grad_tile_at(const GradArgs& a, int b) {
  const int per = a.tiles_x * a.tiles_y;
  GradTileAt t;
  t.img = b / per;
  const int lt = b - t.img * per, ty = lt / a.tiles_x;
  t.x0 = (lt - ty * a.tiles_x) * kGradTile;
  t.y0 = ty * kGradTile;
  t.px0 = (int64_t)t.img * a.H * a.W;
  return t;
}
__device__ __forceinline__ bool far_marked(const GradArgs& a, int c, int64_t gq) {
  return (__ldg(a.far_bits[c] + (gq >> 5)) >> (gq & 31)) & 1u;
}
__device__ __forceinline__ Fix128 far_sum(const GradArgs& a, int c, int64_t gq) {
  const ulonglong2 v = __ldcg((const ulonglong2*)(a.acc[c] + 2 * gq));
  return Fix128{v.x, (long long)v.y};
}

// When the tile's non-zero gradients lie within 30 binary orders of magnitude, counted from 2^-73 at
// least (where the last of 24 bits is the resolution, 2^-96), each is an integer of 53 bits at most in units
// of the smallest one's last bit or of the resolution, to which it is rounded as in the wide sums, and the
// sum of all 1024 fits 63 bits.  It is added to three signed 32-bit limbs of 21 bits (1024 pixels cannot
// overflow one) without returning atomics or carries, and the total converts to float with one
// rounding (the scale is a power of two).  Tiles outside that range are listed for grad_wide_tiles.
constexpr int kSpan = 29;
struct alignas(16) GradLimbs {  // cleared 16 bytes at a time
  int v[2][3][kGradPx];
};
static_assert(alignof(GradLimbs) >= alignof(uint4) && sizeof(GradLimbs) % sizeof(uint4) == 0, "cleared as uint4");
constexpr int kUnitEx = 127 - 73;  // exponent whose last bit is the resolution
__global__ void __launch_bounds__(kGradThreads) grad_tiles_kernel(GradArgs a) {
  __shared__ GradLimbs limbs;
  int (&limb)[2][3][kGradPx] = limbs.v;
  __shared__ uint16_t list[2 * kGradPx];  // class * kGradPx + pixel: sums with a far part
  __shared__ int listed, s_lo[kGradThreads / 32], s_hi[kGradThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GradTileAt T = grad_tile_at(a, blockIdx.x);
  const int x = T.x0 + lane, yw = T.y0 + warp * kGradRows;
  const int64_t at = T.img * a.stride + (int64_t)yw * a.pitch + (int64_t)x * 4;  // first row, bytes
  const int rows_in = x < a.W ? min(kGradRows, a.H - yw) : 0;
  int32_t p[kGradRows];
  uint32_t g[kGradRows];
  int lo = 255, hi = 0;  // exponents of the non-zero gradients
#pragma unroll
  for (int k = 0; k < kGradRows; ++k) {
    p[k] = k < rows_in ? __ldg((const int32_t*)((const char*)a.prov + at + k * a.pitch)) : INT_MIN;
    g[k] = k < rows_in ? __ldg((const uint32_t*)((const char*)a.g + at + k * a.pitch)) : 0u;
  }
  for (int i = threadIdx.x; i < 2 * 3 * kGradPx / 4; i += kGradThreads)
    ((uint4*)&limbs)[i] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int k = 0; k < kGradRows; ++k) {
    const int ex = (g[k] >> 23) & 0xFF;
    if (g[k] << 1) lo = min(lo, ex), hi = max(hi, ex);
  }
  lo = __reduce_min_sync(NSGB_FULL, lo);
  hi = __reduce_max_sync(NSGB_FULL, hi);
  if (lane == 0) s_lo[warp] = lo, s_hi[warp] = hi;
  if (threadIdx.x == 0) listed = 0;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kGradThreads / 32; ++w) lo = min(lo, s_lo[w]), hi = max(hi, s_hi[w]);
  const bool below = lo < kUnitEx;  // the same for the whole tile
  lo = max(lo, kUnitEx);
  if (hi >= 127 + 31 || hi - lo > kSpan) {
    if (threadIdx.x == 0) a.wide[1 + atomicAdd(a.wide, 1)] = blockIdx.x;
    return;
  }
#pragma unroll
  for (int k = 0; k < kGradRows; ++k) {
    if (p[k] == INT_MIN) continue;
    const GradSource s = grad_source(a, p[k]);
    if (s.cls < 0) {
      set_status(a.status, NSGB_ERR_BAD_ARG);
      continue;
    }
    if (other_tile(s, yw + k, x) || (g[k] << 1) == 0u) continue;
    const int i = (s.y & (kGradTile - 1)) * kGradTile + (s.x & (kGradTile - 1));
    const int ex = (g[k] >> 23) & 0xFF;
    unsigned long long v = (g[k] & 0x7FFFFFu) | 0x800000u;
    if (!below || ex >= lo) {
      v <<= ex - lo;
    } else {  // below the resolution (lo = kUnitEx): nearest, ties to even; far below it nothing is left
      const int r = lo - ex;
      const unsigned m = (unsigned)v, rem = r < 32 ? m & ((1u << r) - 1u) : 0u, half = 1u << (min(r, 32) - 1);
      const unsigned q = r < 32 ? m >> r : 0u;
      v = q + ((rem > half || (rem == half && (q & 1u))) ? 1u : 0u);
    }
    const int sign = (int)g[k] >> 31;  // 0 or -1
    constexpr int kMask = (1 << 21) - 1;
    const int l0 = (int)v & kMask, l1 = (int)(v >> 21) & kMask, l2 = (int)(v >> 42);
    if (l0) atomicAdd(&limb[s.cls][0][i], (l0 ^ sign) - sign);
    if (l1) atomicAdd(&limb[s.cls][1][i], (l1 ^ sign) - sign);
    if (l2) atomicAdd(&limb[s.cls][2][i], (l2 ^ sign) - sign);
  }
  __syncthreads();
  const float scale = __uint_as_float((unsigned)(min(lo, 254) - 23) << 23);  // 2^(lo - 150)
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    char* const out = (char*)(c ? a.dmask : a.dmarker) + at;
    const unsigned* const bits = a.far_bits[c];
#pragma unroll
    for (int k = 0; k < kGradRows; ++k) {
      const int i = (warp * kGradRows + k) * kGradTile + lane;
      // the far bits of the tile's 32 pixels of this row (the bitmap has a spare word at its end)
      const int64_t gq = T.px0 + (int64_t)min(yw + k, a.H - 1) * a.W + T.x0;
      const unsigned* word = bits + (gq >> 5);
      const unsigned row_far = __funnelshift_r(__ldg(word), __ldg(word + 1), (unsigned)gq & 31u);
      const bool far = k < rows_in && ((row_far >> lane) & 1u);
      if (k < rows_in) {
        const long long sum = limb[c][0][i] + ((long long)limb[c][1][i] << 21) + ((long long)limb[c][2][i] << 42);
        if (!far) *(float*)(out + k * a.pitch) = __ll2float_rn(sum) * scale;
      }
      const unsigned m = __ballot_sync(NSGB_FULL, far);
      if (m) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&listed, __popc(m));
        base = __shfl_sync(NSGB_FULL, base, 0);
        if (far) list[base + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(c * kGradPx + i);
      }
    }
  }
  __syncthreads();
  const int up = hi ? lo - kUnitEx : 0;  // the tile's unit is 2^(up - 96), 0 <= up <= 103
  for (int j = threadIdx.x; j < listed; j += kGradThreads) {
    const int c = list[j] / kGradPx, i = list[j] & (kGradPx - 1);
    const int y = T.y0 + i / kGradTile, xi = T.x0 + (i & (kGradTile - 1));
    const long long sum = limb[c][0][i] + ((long long)limb[c][1][i] << 21) + ((long long)limb[c][2][i] << 42);
    Fix128 v;
    if (up < 64) {
      v.lo = (unsigned long long)sum << up;
      v.hi = up ? sum >> (64 - up) : sum >> 63;
    } else {
      v.lo = 0ull;
      v.hi = (long long)((unsigned long long)sum << (up - 64));
    }
    v = fix_add(v, far_sum(a, c, T.px0 + (int64_t)y * a.W + xi));
    grad_row(a, c ? a.dmask : a.dmarker, T.img, y)[xi] = fix_to_float(v.lo, v.hi);
  }
}

// The listed tiles, any finite gradients below 2^31.  Contributions are counted first.  The one gradient of
// a source that gets no other stays as it is; the sources that get several (512 at most) have six signed
// 32-bit limbs of 21 bits (a gradient's 24 bits touch three at most, and 1024 pixels cannot overflow the
// lower five).  Sources with limbs or marked in the bitmap are listed and converted densely; the others are
// their gradient.
// Bound: latency at up to 48 warps an SM.  (A compare-and-swap per gradient for its source's slot, and limbs
// for all 2048 sources -- 61 KB, three CTAs an SM -- took 82 us at 4 x 1024^2 with all tiles listed, this 68.)
constexpr int kLimbs = 6, kLimbBits = 21, kMulti = kGradPx / 2;
struct alignas(16) GradTile {  // counts and limbs are cleared 16 bytes at a time
  int count[2 * kGradPx];      // class * kGradPx + pixel: gradients, or -1 - index of the limbs
  int limb[kLimbs][kMulti];
  uint32_t one[2 * kGradPx];   // the gradient where there is one
  uint16_t list[2 * kGradPx];
  int listed, multi;
};
static_assert(alignof(GradTile) >= alignof(uint4) && offsetof(GradTile, limb) % sizeof(uint4) == 0, "cleared as uint4");
constexpr int kWideCtasPerSm = 6;  // shared memory

__device__ __forceinline__ void limb_add(int (*limb)[kMulti], int i, float g) {
  const uint32_t b = __float_as_uint(g), ex = (b >> 23) & 0xFFu;
  uint32_t man = b & 0x7FFFFFu;
  int s = ex == 0 ? -149 + 96 : (int)ex - 150 + 96;  // g = +-man * 2^(s - 96)
  if (ex != 0) man |= 0x800000u;
  if (s < 0) {  // round to the resolution, ties to even
    const int r = -s;
    if (r >= 32) return;
    const uint32_t q = man >> r, rem = man & ((1u << r) - 1u), half = 1u << (r - 1);
    man = q + ((rem > half || (rem == half && (q & 1u))) ? 1u : 0u);
    s = 0;
  }
  const int k = s / kLimbBits;
  unsigned long long v = (unsigned long long)man << (s - k * kLimbBits);
  const bool neg = (b >> 31) != 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    // the last limb takes all that is left (s <= 103: bits 105 .. 126), modulo 2^32: the sum of a
    // source is below 2^127, so the last limb's final value fits
    const bool last = k + j == kLimbs - 1;
    const int l = last ? (int)v : (int)(v & ((1u << kLimbBits) - 1u));
    v = last ? 0ull : v >> kLimbBits;
    if (l) atomicAdd(&limb[k + j][i], neg ? -l : l);
  }
}

__device__ __forceinline__ void grad_wide_tile(const GradArgs& a, GradTile& S, int tile) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kRows = kGradRows;
  const GradTileAt T = grad_tile_at(a, tile);
  const int img = T.img, y0 = T.y0, x = T.x0 + lane;
  const int64_t px0 = T.px0;
  int32_t p[kRows];
  float g[kRows];
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const int y = y0 + warp * kRows + k;
    const bool in = y < a.H && x < a.W;
    p[k] = in ? __ldg(grad_row(a, a.prov, img, y) + x) : INT_MIN;
    g[k] = in ? __ldg(grad_row(a, a.g, img, y) + x) : 0.f;
  }
  for (int i = threadIdx.x; i < 2 * kGradPx / 4; i += kGradThreads) ((uint4*)S.count)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = threadIdx.x; i < kLimbs * kMulti / 4; i += kGradThreads) ((uint4*)S.limb)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x == 0) S.listed = S.multi = 0;
  __syncthreads();
  int src[kRows];  // class * kGradPx + pixel of the tile's own sources, else -1
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    src[k] = -1;
    if (p[k] == INT_MIN) continue;
    const GradSource s = grad_source(a, p[k]);
    const uint32_t mag = __float_as_uint(g[k]) & 0x7FFFFFFFu;
    if (s.cls < 0 || mag >= (127u + 31u) << 23) {  // |g| >= 2^31, inf, NaN
      set_status(a.status, NSGB_ERR_BAD_ARG);
      continue;
    }
    if (mag == 0u || other_tile(s, y0 + warp * kRows + k, x)) continue;
    src[k] = s.cls * kGradPx + (s.y & (kGradTile - 1)) * kGradTile + (s.x & (kGradTile - 1));
    atomicAdd(&S.count[src[k]], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kGradPx; i += kGradThreads) {  // whole warps
    const bool many = S.count[i] > 1;
    const unsigned m = __ballot_sync(NSGB_FULL, many);
    if (!m) continue;
    int base = 0;
    if (lane == 0) base = atomicAdd(&S.multi, __popc(m));
    base = __shfl_sync(NSGB_FULL, base, 0);
    if (many) S.count[i] = -1 - (base + __popc(m & ((1u << lane) - 1u)));
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    if (src[k] < 0) continue;
    const int n = S.count[src[k]];
    if (n > 0) S.one[src[k]] = __float_as_uint(g[k]);
    else limb_add(S.limb, -1 - n, g[k]);
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float* const out = c ? a.dmask : a.dmarker;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int i = c * kGradPx + (warp * kRows + k) * kGradTile + lane;
      const int y = y0 + warp * kRows + k;
      const bool in = y < a.H && x < a.W;
      bool more = false;
      if (in) {
        const int n = S.count[i];
        const uint32_t one = n > 0 ? S.one[i] : 0u;
        // a gradient below 2^-73 still has to be rounded to the resolution
        more = n < 0 || far_marked(a, c, px0 + (int64_t)y * a.W + x) ||
               (n > 0 && (one & 0x7FFFFFFFu) < (uint32_t)kUnitEx << 23);
        if (!more) grad_row(a, out, img, y)[x] = __uint_as_float(one);
      }
      const unsigned m = __ballot_sync(NSGB_FULL, more);
      if (m) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&S.listed, __popc(m));
        base = __shfl_sync(NSGB_FULL, base, 0);
        if (more) S.list[base + __popc(m & ((1u << lane) - 1u))] = (uint16_t)i;
      }
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < S.listed; j += kGradThreads) {
    const int c = S.list[j] / kGradPx, i = S.list[j] & (kGradPx - 1), n = S.count[S.list[j]];
    const int y = y0 + i / kGradTile, xi = T.x0 + (i & (kGradTile - 1));
    Fix128 v = {0ull, 0ll};
    if (n < 0) {
      __int128 sum = 0;
#pragma unroll
      for (int l = kLimbs - 1; l >= 0; --l) sum = sum * (1 << kLimbBits) + S.limb[l][-1 - n];
      v = Fix128{(unsigned long long)sum, (long long)(sum >> 64)};
    } else if (n > 0) {
      fix_from_float(__uint_as_float(S.one[S.list[j]]), v);
    }
    const int64_t gq = px0 + (int64_t)y * a.W + xi;
    if (far_marked(a, c, gq)) v = fix_add(v, far_sum(a, c, gq));
    grad_row(a, c ? a.dmask : a.dmarker, img, y)[xi] = fix_to_float(v.lo, v.hi);
  }
}

__global__ void __launch_bounds__(kGradThreads, kWideCtasPerSm) grad_wide_tiles_kernel(GradArgs a) {
  __shared__ GradTile tile;
  const int n = __ldcg(a.wide);
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    grad_wide_tile(a, tile, __ldcg(a.wide + 1 + j));
    __syncthreads();
  }
}

bool f32_dims_ok(int64_t batch, int64_t rows, int64_t cols, int64_t pitch, int64_t stride) {
  if (batch <= 0 || rows <= 0 || cols <= 0 || rows >= INT_MAX || cols >= INT_MAX) return false;
  if (pitch < cols * 4 || pitch % 4) return false;
  const int64_t n = rows * cols;
  if (2 * n >= kKeyNone || n * batch >= (int64_t)INT_MAX || rows * batch >= (int64_t)INT_MAX) return false;
  if (batch > 1 && (stride < rows * pitch || stride % 4)) return false;
  return true;
}

size_t f32_fwd_bytes(int64_t batch, int64_t rows, int64_t cols) {
  const Plan P1 = single_plan(NSGB_F32, nullptr, nullptr, rows, cols, cols * 4);
  return ws_sizes(stacked_totals(P1.t, batch)).total;
}

// Up to this many pixels clearing all accumulators (32 bytes a pixel) is quicker than a launch that finds the
// ones to clear (200 x 333: 2 against 5 us).
constexpr size_t kGradSmallPx = 1 << 18;

int64_t grad_tiles(int64_t batch, int64_t rows, int64_t cols) {
  return batch * ((rows + kGradTile - 1) / kGradTile) * ((cols + kGradTile - 1) / kGradTile);
}

size_t f32_bwd_bytes(int64_t batch, int64_t rows, int64_t cols) {
  // status, the accumulators and bitmaps of marker and mask sources, the list of wide tiles
  const size_t px = (size_t)(batch * rows * cols);
  return 256 + 2 * align256(16 * px) + 2 * align256(sizeof(unsigned) * (px / 32 + 2)) +
         align256(sizeof(int) * (size_t)(grad_tiles(batch, rows, cols) + 1));
}

// Plan over the stacked images; with more than one image the table is built on the device.
cudaError_t stacked_plan(void* plane, const void* aux, int64_t batch, int64_t rows, int64_t cols, int64_t pitch,
                         int64_t stride, Img* table, Plan* P, cudaStream_t s) {
  const Plan P1 = single_plan(NSGB_F32, plane, aux, rows, cols, pitch);
  P->t = stacked_totals(P1.t, batch);
  P->I = P1.I;
  P->I.n = (int)batch;
  if (batch == 1) return cudaSuccess;
  Img proto = P1.I.one;
  proto.aligned = proto.aligned && (stride % 4 == 0);
  P->I.one = proto;
  P->I.d = table;
  P->I.r_per = P1.t.r_tiles;
  P->I.c_per = P1.t.c_tiles;
  stack_table_kernel<<<(unsigned)((batch + 127) / 128), 128, 0, s>>>(proto, (int)batch, stride, P1.t, table);
  return cudaGetLastError();
}

}  // namespace
}  // namespace nsgb

extern "C" {

size_t nsgb_recon_f32_workspace_size(int64_t batch, int64_t rows, int64_t cols, int backward) {
  if (!f32_dims_ok(batch, rows, cols, cols * 4, rows * cols * 4)) return 0;
  return backward ? f32_bwd_bytes(batch, rows, cols) : f32_fwd_bytes(batch, rows, cols);
}

nsgb_status nsgb_recon_f32_fwd(const float* marker, const float* mask, float* out, int32_t* prov, int64_t batch,
                               int64_t rows, int64_t cols, int64_t pitch, int64_t image_stride, int conn, void* ws,
                               size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!marker || !mask || !out || !prov || (const void*)out == (const void*)marker || !valid_conn(conn) ||
      !f32_dims_ok(batch, rows, cols, pitch, image_stride))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws_bytes(ws, ws_bytes, f32_fwd_bytes(batch, rows, cols));
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const Plan P1 = single_plan(NSGB_F32, out, mask, rows, cols, pitch);
  const Ws w = carve(ws, stacked_totals(P1.t, batch));
  Plan P;
  cudaError_t e = stacked_plan(out, mask, batch, rows, cols, pitch, image_stride, w.table, &P, s);
  // out = marker, image by image (one 2-D copy when the stack is contiguous)
  const bool dense = batch == 1 || image_stride == rows * pitch;
  for (int64_t b = 0; e == cudaSuccess && b < (dense ? 1 : batch); ++b)
    e = cudaMemcpy2DAsync((char*)out + b * image_stride, pitch, (const char*)marker + b * image_stride, pitch,
                          (size_t)cols * 4, (size_t)(dense ? rows * batch : rows), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = recon_timed(opts, NSGB_F32, P, conn, false, true, w.recon, s);
  if (e == cudaSuccess) e = ccl::label(ClsPlateau{}, P.I, P.t, conn, w.forest(false), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.A, 0x7F, sizeof(int) * (size_t)P.t.px, s);
  if (e == cudaSuccess) {
    const int64_t moff = (int64_t)((uintptr_t)marker - (uintptr_t)out);
    const int64_t poff = (int64_t)((uintptr_t)prov - (uintptr_t)out);
    const bool quads = (((uintptr_t)out | (uintptr_t)mask | (uintptr_t)marker) % 16) == 0 && pitch % 16 == 0 &&
                       (batch == 1 || image_stride % 16 == 0);
    source_best_kernel<<<qrb(P.t), 256, 0, s>>>(P.I, P.t.rows, moff, w.L, w.A, quads);
    prov_out_kernel<<<qrb(P.t), 256, 0, s>>>(P.I, P.t.rows, w.L, w.A, poff, w.status);
    e = cudaGetLastError();
  }
  return finish(e, ws, s, opts);
}

nsgb_status nsgb_recon_f32_bwd(const float* grad_out, const int32_t* prov, float* grad_marker, float* grad_mask,
                               int64_t batch, int64_t rows, int64_t cols, int64_t pitch, int64_t image_stride,
                               void* ws, size_t ws_bytes, nsgb_stream_t stream, const nsgb_opts* opts) {
  if (!grad_out || !prov || !grad_marker || !grad_mask || !f32_dims_ok(batch, rows, cols, pitch, image_stride))
    return NSGB_ERR_BAD_ARG;
  nsgb_status st = check_ws_bytes(ws, ws_bytes, f32_bwd_bytes(batch, rows, cols));
  if (st != NSGB_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t px = (size_t)(batch * rows * cols);
  const size_t acc_bytes = align256(16 * px), bit_bytes = align256(sizeof(unsigned) * (px / 32 + 2));
  char* p = (char*)ws;
  GradArgs a = {};
  a.g = grad_out;
  a.prov = prov;
  a.dmarker = grad_marker;
  a.dmask = grad_mask;
  a.pitch = pitch;
  a.stride = batch > 1 ? image_stride : 0;
  a.H = (int)rows;
  a.W = (int)cols;
  a.n = (int)batch;
  a.tiles_x = (a.W + kGradTile - 1) / kGradTile;
  a.tiles_y = (a.H + kGradTile - 1) / kGradTile;
  // floor(q / W) for q < 2^31: with 2^l >= W the multiplier exceeds 2^(31 + l) / W by at most 1,
  // which moves the quotient by q / 2^(31 + l) < 1 / W
  int l = 0;
  while ((1ll << l) < cols) ++l;
  a.div_shift = l - 1;
  a.div_mul = cols > 1 ? (unsigned)((1ull << (31 + l)) / (unsigned long long)cols + 1ull) : 0u;
  a.status = (int*)p;
  a.acc[0] = (unsigned long long*)(p + 256);
  a.acc[1] = (unsigned long long*)(p + 256 + acc_bytes);
  a.far_bits[0] = (unsigned*)(p + 256 + 2 * acc_bytes);
  a.far_bits[1] = (unsigned*)(p + 256 + 2 * acc_bytes + bit_bytes);
  a.wide = (int*)(p + 256 + 2 * acc_bytes + 2 * bit_bytes);
  const bool vec = ((uintptr_t)prov % 16) == 0 && pitch % 16 == 0 && a.stride % 16 == 0;
  const bool small = px <= kGradSmallPx;
  // The first launch clears the status, the bitmaps, the count of wide tiles behind them and, for a small
  // image, the accumulators in front of them.
  unsigned* const first = small ? (unsigned*)a.acc[0] : a.far_bits[0];
  const ccl::ZeroSpans z{{(unsigned*)a.status, first, nullptr, nullptr}, {1, (int)((unsigned*)a.wide - first) + 1, 0, 0}};
  cudaError_t e = ccl::launch_k(false, ccl::zero_words, dim3(grid1d(z.total())), dim3(256), s, z);
  const unsigned gy = (unsigned)std::min<int64_t>(rows, 65535), gz = (unsigned)std::min<int64_t>(batch, 65535);
  const dim3 quads((a.W + 511) / 512, gy, gz);
  const dim3 rows4((a.W + 127) / 128, (unsigned)std::min<int64_t>((rows + kFarRows - 1) / kFarRows, 65535), gz);
  const int64_t tiles = grad_tiles(batch, rows, cols);
  // (ordinary launches: the wait of a dependent one costs many short CTAs 20 us each at 16 x 2048^2)
  if (e == cudaSuccess && !small) {
    if (vec) grad_touch_kernel<true><<<quads, 128, 0, s>>>(a);
    else grad_touch_kernel<false><<<quads, 128, 0, s>>>(a);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = launch_dependent(small ? grad_far_kernel<true> : grad_far_kernel<false>, rows4, dim3(128), s, a);
  if (e == cudaSuccess) {
    grad_tiles_kernel<<<(unsigned)tiles, kGradThreads, 0, s>>>(a);
    grad_wide_tiles_kernel<<<(unsigned)std::min<int64_t>(tiles, kWideCtasPerSm * 152), kGradThreads, 0, s>>>(a);
    e = cudaGetLastError();
  }
  return finish(e, ws, s, opts);
}

}  // extern "C"
