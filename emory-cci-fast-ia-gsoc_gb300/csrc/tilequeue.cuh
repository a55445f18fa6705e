// Tile work queue of the reconstruction kernel (recon.cu): per-tile states, a bounded
// multi-producer / multi-consumer ring with per-slot sequence numbers (Vyukov's queue),
// neighbour marking, and the initial orders.
// Every wait is bounded; a wait that runs out sets the status word.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace nsgb {
namespace tq {

enum TileState : int { kIdle = 0, kQueued = 1, kRunning = 2, kRunningDirty = 3 };


struct alignas(8) Slot {
  int val;
  unsigned seq;
};

// One 64-bit word, changed by one atomic: `pending` in the low half, the ticket counter above it.
// `pending` is never negative and at most twice the number of tiles (a tile given up by `and ~2` can be
// marked and counted again before its own release is counted), far below 2^32: nothing carries into
// the upper half.
struct alignas(8) Tally {
  int pending;
  unsigned tail;
};

struct Ctl {
  int* state;         // [ntiles] TileState
  Slot* slots;        // [cap] work ring
  unsigned* head;     // consumer ticket counter
  Tally* tally;       // producer ticket counter and count of queued + running tiles
  int* done;          // set once pending reaches zero
  int* status;
  int* stats;         // [0] visits, [1] sweeps, [2] re-runs
  unsigned long long* visit_count;  // budget counter
  unsigned long long* prof;         // [8] phase cycle counters (profiling builds only)
  unsigned cap;       // ring capacity (power of two >= ntiles)
  long long max_visits;
  long long spin_limit;  // polls before a queue wait gives up (kSpinLimit unless overridden)
  int budget_step;
};

// A slot is read and written as one 64-bit word (tile, sequence number), so a consumer gets the
// tile with the poll that finds it and neither side needs a fence: the word itself carries all
// that is passed on here (the pixels are ordered by the tile states below).  Polls are relaxed: an
// acquire load also drops the SM's L1 contents, under the warps that are still sweeping.
__device__ __forceinline__ Slot ld_slot(const Slot* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  Slot s;
  s.val = (int)(unsigned)v;
  s.seq = (unsigned)(v >> 32);
  return s;
}
__device__ __forceinline__ void st_slot(Slot* p, int val, unsigned seq) {
  const unsigned long long v = ((unsigned long long)seq << 32) | (unsigned)val;
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Producer side of the ring (Vyukov's bounded queue) with ticket `p`: wait until its slot is free
// for this lap, then fill it.
__device__ __forceinline__ bool queue_put(const Ctl& c, unsigned p, int t) {
  Slot* sl = &c.slots[p & (c.cap - 1)];
  long long spins = 0;
  while (ld_slot(sl).seq != p) {
    if (++spins > c.spin_limit || ld_relaxed(c.status) != 0) {
      set_status(c.status, kDevTimeout);
      return false;
    }
    __nanosleep(64);
  }
  st_slot(sl, t, p + 1u);
  return true;
}

// Consumer side: claim a ticket and wait for its item; returns -1 once no tile is queued or
// running any more (the done flag: nothing can be pushed again) or after an error.  A waiting
// warp polls its own slot; the done flag only every second wait and the status word every 64th,
// so that idle warps do not flood the L2 lines that the working warps' atomics use.
__device__ __forceinline__ int queue_pop(const Ctl& c) {
  const unsigned tk = atomicAdd(c.head, 1u);
  Slot* sl = &c.slots[tk & (c.cap - 1)];
  long long spins = 0;
  unsigned ns = 64;
  for (;;) {
    const Slot got = ld_slot(sl);
    if (got.seq == tk + 1u) {
      st_slot(sl, -1, tk + c.cap);
      return got.val;
    }
    ++spins;
    if ((spins & 1) == 0 && ld_relaxed(c.done) != 0) return -1;
    if ((spins & 63) == 0 && ld_relaxed(c.status) != 0) return -1;
    if (spins > c.spin_limit) {
      set_status(c.status, kDevTimeout);
      return -1;
    }
    __nanosleep(ns);
    if (ns < 512) ns <<= 1;
  }
}

// Tile states and the memory order of tile visits.  Every change of a tile's state is an atomic
// read-modify-write, so all of them are totally ordered per tile.  A visit takes its tile with an
// acquire exchange (QUEUED -> RUNNING) before it reads any pixel.  After its stores a warp issues
// one fence and then marks neighbours with `or 1` (IDLE -> QUEUED, RUNNING -> RUNNING_DIRTY, the
// others unchanged) and gives up its own tile with `and ~2` (RUNNING -> IDLE, RUNNING_DIRTY ->
// QUEUED); the fence makes each of them a release.  For a visit V of tile t and a marker U of t,
// either U's `or` comes before V's exchange in t's order -- then V's acquire reads from U's
// release (or a later read-modify-write of the same sequence) and V's loads see U's stores -- or
// after it, and then U sees RUNNING and the visit is run again.
__device__ __forceinline__ int atom_or(int* p, int v) {
  int old;
  asm volatile("atom.relaxed.gpu.global.or.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int atom_and(int* p, int v) {
  int old;
  asm volatile("atom.relaxed.gpu.global.and.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int atom_exch_acquire(int* p, int v) {
  int old;
  asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// The end of a visit of tile t by one warp, after its stores and a warp barrier: lanes with `mark`
// (lanes 0 .. 8) mark tile nt, whose values may have become stale, lane 9 gives up t.  A marked
// tile that was idle, and t itself if it was marked while it ran, go to the queue.
//
// The marks and the release are one round of atomics behind one fence (the order between them does
// not matter: each only publishes the stores before the fence).  One 64-bit atomic then takes
// the ring tickets of the tiles to queue and moves `pending` by those tiles less the one given up,
// so the count never reaches 0 early: a tile cannot be popped before its ticket is known.  (Release
// atomics and stores one after another, each with a fence of its own -- marks, count, ticket, slot,
// release, count -- were 10% of the kernel's warp time in fence waits and five more round trips.)
__device__ __forceinline__ void mark_and_release(const Ctl& c, bool mark, int nt, int t, int lane) {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  int old = -1;
  if (mark) old = atom_or(&c.state[nt], 1);
  else if (lane == 9) old = atom_and(&c.state[t], ~2);
  const unsigned woken = __ballot_sync(NSGB_FULL, mark && old == kIdle);
  const bool dirty = __shfl_sync(NSGB_FULL, old, 9) == kRunningDirty;
  const unsigned put = woken | (dirty ? 1u << 9 : 0u);
  const int more = __popc(woken) - (dirty ? 0 : 1);
  unsigned ticket = 0;
  if (lane == 9) {
    if (put != 0u || more != 0) {
      const unsigned long long step = ((unsigned long long)__popc(put) << 32) + (unsigned long long)(long long)more;
      const unsigned long long was = atomicAdd((unsigned long long*)c.tally, step);
      ticket = (unsigned)(was >> 32);
      if ((int)(unsigned)was + more == 0) atomicExch(c.done, 1);
    }
    if (dirty) atomicAdd(&c.stats[2], 1);
  }
  if (put != 0u) {  // the same for all lanes
    ticket = __shfl_sync(NSGB_FULL, ticket, 9) + __popc(put & ((1u << lane) - 1u));
    if ((put >> lane) & 1u) queue_put(c, ticket, lane == 9 ? t : nt);
  }
  __syncwarp();
}

// The same steps one after another, each release with its own fence, by the lanes that have
// something to do.  The reconstruction of 32-bit pixels, and every re-sweeping visit (which may
// take its tile back instead), ends this way: with mark_and_release() the compiler emits the 32-bit
// kernel at 61 instead of 42 KB, and the instruction fetches of lone working warps cost more than
// the fences (4096^2 f32 h-minima 242 -> 312 us, 20 batched i32 tiles 1855 -> 2000 us; against u8
// 264 -> 245 us, 15 batched u8 tiles 530 -> 487 us).
__device__ __forceinline__ int atom_or_release(int* p, int v) {
  int old;
  asm volatile("atom.release.gpu.global.or.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int atom_exch_acq_rel(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int atom_cas_acq_rel(int* p, int cmp, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "l"(p), "r"(cmp), "r"(v) : "memory");
  return old;
}
// Queues tile t, counting it as pending (`more` = 1) or not (it is already counted).
__device__ __forceinline__ void queue_push(const Ctl& c, int t, int more) {
  const unsigned long long was =
      atomicAdd((unsigned long long*)c.tally, (1ull << 32) + (unsigned long long)(unsigned)more);
  queue_put(c, (unsigned)(was >> 32), t);
}
__device__ __forceinline__ void mark_tile(const Ctl& c, int nt) {
  if (atom_or_release(&c.state[nt], 1) == kIdle) queue_push(c, nt, 1);
}
__device__ __forceinline__ void pending_release(const Ctl& c) {
  const unsigned long long was = atomicAdd((unsigned long long*)c.tally, ~0ull);
  if ((unsigned)was == 1u) atomicExch(c.done, 1);
}

// Initial queue order.  order 0: raster.  order 1: checkerboard, even tiles first.  order 2:
// four colours by (row parity, column parity) in the sequence (0,0), (1,1), (0,1), (1,0), so
// that no two tiles of one colour touch, not even diagonally.  Tiles taken from the queue at
// the same time are then rarely neighbours, and later colours read finished neighbours.
__device__ __forceinline__ int initial_tile(int i, int ntiles, int tiles_x, int order) {
  const int tiles_y = ntiles / tiles_x;
  if (order == 1) {
    // tiles (ty, tx) with (ty + tx) even first, then the odd ones, each in raster order; row ty
    // holds ceil(tiles_x / 2) of its first colour and floor(tiles_x / 2) of the other
    const int hi = (tiles_x + 1) / 2, lo = tiles_x / 2;
    const int even_total = ((tiles_y + 1) / 2) * hi + (tiles_y / 2) * lo;
    int k = i, parity = 0;
    if (k >= even_total) {
      k -= even_total;
      parity = 1;
    }
    // rows alternate between `a` tiles (ty even for parity 0) and `b` tiles
    const int a = parity ? lo : hi, b = parity ? hi : lo;
    const int pair = a + b;
    int ty = pair ? 2 * (k / pair) : 0;
    k = pair ? k % pair : k;
    if (k >= a) {
      k -= a;
      ++ty;
    }
    const int first = ((ty & 1) ^ parity) ? 1 : 0;
    return ty * tiles_x + first + 2 * k;
  }
  if (order == 2) {
    const int seq_py[4] = {0, 1, 0, 1}, seq_px[4] = {0, 1, 1, 0};
    int k = i;
    for (int c = 0; c < 4; ++c) {
      const int py = seq_py[c], px = seq_px[c];
      const int ny = (tiles_y - py + 1) / 2, nx = (tiles_x - px + 1) / 2;
      if (k < ny * nx) return (py + 2 * (k / nx)) * tiles_x + px + 2 * (k % nx);
      k -= ny * nx;
    }
  }
  return i;
}

inline unsigned ring_cap(int64_t ntiles) {
  unsigned c = 32;
  while ((int64_t)c < ntiles) c <<= 1;
  return c;
}


}  // namespace tq
}  // namespace nsgb
