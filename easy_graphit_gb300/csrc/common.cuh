// Device-side building blocks of the engine: graph and frontier views passed
// to kernels by value, the enqueue primitives of runtime/infra_gpu/
// vertex_frontier.h:176-216 and support.h:14-54 re-done for sm_103a, and a
// bounded grid barrier for persistent kernels.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "gg_internal.h"

namespace cg = cooperative_groups;

namespace gg {

// Error bits of the per-graph device status word.
enum : int32_t {
  DEV_ERR_OVERFLOW = 1,  // a sparse queue ran past its capacity
  DEV_ERR_TIMEOUT = 2,   // a grid barrier wait gave up
};

// --------------------------------------------------------------- graph view
// CSR (or CSC for a transposed graph) plus optional COO sources and dst-block
// buckets, as in graphit_runtime::GraphT (graph.h:17-88).
struct DGraph {
  int32_t V;
  int32_t E;
  const int32_t *__restrict__ off;     // V+1
  const int32_t *__restrict__ dst;     // E
  const int32_t *__restrict__ w;       // E
  const int32_t *__restrict__ src;     // E (COO row of each edge), may be null
  const int32_t *__restrict__ bucket;  // nbuckets+1 bucket starts (blocked graphs)
  int32_t nbuckets;
};

// Which vertices an LB kernel enumerates: q[0..n) or 0..n when q is null.
struct Enum {
  const int32_t *__restrict__ q;
  const int32_t *__restrict__ n_dev;  // device count (read when n < 0)
  int32_t n;
  __device__ __forceinline__ int32_t count() const {
    return n >= 0 ? n : *(volatile const int32_t *)n_dev;
  }
  // L2-coherent load: persistent kernels refill the queue they enumerate.
  __device__ __forceinline__ int32_t at(int32_t i) const { return q ? __ldcg(q + i) : i; }
};

// Membership test against an input frontier (bitmap / boolmap), or "all".
enum : int32_t { IN_ALL = 0, IN_BITMAP = 1, IN_BOOLMAP = 2 };
struct DIn {
  int32_t mode;
  const uint32_t *__restrict__ bm;
  const uint8_t *__restrict__ by;
  __device__ __forceinline__ bool has(int32_t v) const {
    if (mode == IN_ALL) return true;
    if (mode == IN_BITMAP) return (bm[v >> 5] >> (v & 31)) & 1u;
    return by[v] != 0;
  }
};

// Warp-aggregated counter increment (support.h:14-25 atomicAggInc), using a
// coalesced group so it is safe under independent thread scheduling.
__device__ __forceinline__ int32_t agg_inc(int32_t *ctr) {
  cg::coalesced_group g = cg::coalesced_threads();
  int32_t base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(ctr, (int32_t)g.size());
  base = g.shfl(base, 0);
  return base + (int32_t)g.thread_rank();
}

// writeMin / writeMax / CAS of support.h:26-54: an early-out read, then the
// atomic; true when this call changed the value.
__device__ __forceinline__ bool write_min(int32_t *p, int32_t v) {
  if (*(volatile int32_t *)p <= v) return false;
  return atomicMin(p, v) > v;
}
__device__ __forceinline__ bool write_max(int32_t *p, int32_t v) {
  if (*(volatile int32_t *)p >= v) return false;
  return atomicMax(p, v) < v;
}
__device__ __forceinline__ bool cas(int32_t *p, int32_t expect, int32_t v) {
  if (*(volatile int32_t *)p != expect) return false;
  return atomicCAS(p, expect, v) == expect;
}

// A CTA's appends to a sparse queue, staged in shared memory and sent with one
// reservation (stage_flush).  A queue has one count for the whole GPU: a level
// that finds 10^6 vertices in groups of two to four lanes makes 10^5 atomics on
// that one word, which the L2 takes one after another (the widest level of a BFS
// on the directed R-MAT 22, 1.1 M vertices found, with a stage of 1,024 entries,
// half of them appended directly: 101 us pulled and 772 pushed; with 2,048 70 and
// 448).  Appends past its end go to the queue directly; the count is read first, or
// whoever walks a hub alone would pay for two atomics an append (BFS on a star of a
// million leaves, a thread per vertex 1,287 -> 1,170 ms, a warp per vertex 48.7 -> 44.9).
constexpr int32_t kStageCap = 2048;
struct alignas(16) Stage {  // `cap` entries follow it in shared memory
  int32_t n, cap, base, pad_;
  __device__ __forceinline__ int32_t *buf() { return reinterpret_cast<int32_t *>(this + 1); }
  __device__ __forceinline__ void init(int32_t entries) {
    n = 0;
    cap = entries;
  }
  // Stages v; false when the stage is full.
  __device__ __forceinline__ bool add(int32_t v) {
    if (*(volatile int32_t *)&n >= cap) return false;
    const int32_t at = agg_inc(&n);
    if (at >= cap) return false;
    buf()[at] = v;
    return true;
  }
};
// Entries of each of a kernel's several stages: four a thread, at least 512.  With
// 2,048 whatever the CTA, the many small CTAs of an SM leave little of it to the L1
// (SSSP, a thread per vertex, 0.5 M vertices of degree 40: CTAs of 128 3.9 -> 1.8 ms,
// of 64 2.8 -> 1.9).
__host__ __device__ constexpr int32_t stage_cap(int32_t cta) {
  return cta <= 128 ? 512 : (cta < 512 ? 4 * cta : kStageCap);
}
// The i-th of them in dynamic shared memory behind `used` bytes, and the bytes of all.
__device__ __forceinline__ Stage *stage_at(void *smem, int32_t used, int32_t cap, int i) {
  return reinterpret_cast<Stage *>(static_cast<char *>(smem) + (used + 15) / 16 * 16 + i * (16 + 4 * cap));
}
inline size_t with_stages(size_t used, int32_t cap, int n) { return (used + 15) / 16 * 16 + n * (16 + 4 * (size_t)cap); }

struct StageMem {  // one of kStageCap entries in static shared memory
  Stage s;
  int32_t buf[kStageCap];
};

// Output frontier writer: the enqueue_* family of gpu_intrinsics.h:95-110.
enum : int32_t {
  OUT_NONE = 0,
  OUT_SPARSE = 1,        // enqueue_sparse (duplicates allowed)
  OUT_SPARSE_DEDUP = 2,  // enqueue_sparse_no_dupes (writeMax epoch counter)
  OUT_BITMAP = 3,        // enqueue_bitmap (atomicOr + count of new bits)
  OUT_BOOLMAP = 4,       // enqueue_boolmap (byte set + count of new bytes)
};
struct DOut {
  int32_t mode;
  int32_t *__restrict__ q;
  int32_t *cnt;
  int64_t cap;
  uint32_t *bm;
  uint8_t *by;
  int32_t *dedup;
  int32_t epoch;
  int32_t *err;
  Stage *stage;  // shared memory, or null: append directly
  bool few;      // no list is longer than kStage1 edges

  __device__ __forceinline__ void sparse(int32_t v) const {
    if (stage && stage->add(v)) return;
    const int32_t pos = agg_inc(cnt);
    if (pos < cap)
      q[pos] = v;
    else
      atomicOr(err, DEV_ERR_OVERFLOW);
  }
  __device__ __forceinline__ void push(int32_t v) const {
    switch (mode) {
      case OUT_SPARSE:
        sparse(v);
        break;
      case OUT_SPARSE_DEDUP:
        if (write_max(dedup + v, epoch)) sparse(v);
        break;
      case OUT_BITMAP: {
        const uint32_t bit = 1u << (v & 31);
        uint32_t *word = bm + (v >> 5);
        if (!(*(volatile uint32_t *)word & bit) && !(atomicOr(word, bit) & bit)) agg_inc(cnt);
        break;
      }
      case OUT_BOOLMAP: {
        // The reference sets the byte without an atomic and may count a vertex
        // twice (vertex_frontier.h:195-201); an OR on the containing word keeps
        // the count exact.
        if (by[v]) break;
        const uint32_t sh = 8u * (v & 3);
        uint32_t *word = reinterpret_cast<uint32_t *>(by + (v & ~3));
        if (!((atomicOr(word, 1u << sh) >> sh) & 0xffu)) agg_inc(cnt);
        break;
      }
      default:
        break;
    }
  }
};

// Sends what a CTA staged for `out` and empties the stage; the whole CTA calls
// it.  Appends after it need a barrier first (every caller ends its step at one).
__device__ __forceinline__ void stage_flush(Stage *st, int32_t *q, int32_t *cnt, int64_t cap, int32_t *err) {
  __syncthreads();
  const int32_t n = min(st->n, st->cap);
  if (n == 0) return;
  if (threadIdx.x == 0) st->base = atomicAdd(cnt, n);
  __syncthreads();
  const int32_t base = st->base;
  for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
    if (base + i < cap)
      q[base + i] = st->buf()[i];
    else
      atomicOr(err, DEV_ERR_OVERFLOW);
  }
  if (threadIdx.x == 0) st->n = 0;
}
__device__ __forceinline__ void stage_flush(const DOut &out) {
  stage_flush(out.stage, out.q, out.cnt, out.cap, out.err);
}
// The same in the middle of a step, when fewer than `room` entries are left.  The
// whole CTA calls it behind a barrier, with another one before its next append.
__device__ __forceinline__ void stage_make_room(const DOut &out, int32_t room) {
  if (out.stage && out.stage->n > out.stage->cap - room) {
    stage_flush(out);
    __syncthreads();
  }
}

// Appends v to a pile, through a CTA's stage when there is one.
__device__ __forceinline__ void pile_append(Stage *st, int32_t *pile, int32_t *cnt, int32_t cap, int32_t v,
                                            int32_t *err) {
  if (st && st->add(v)) return;
  const int32_t pos = agg_inc(cnt);
  if (pos < cap)
    pile[pos] = v;
  else
    atomicOr(err, DEV_ERR_OVERFLOW);
}

// Raises v's stamp to `tag` and returns what it was: v is this caller's to append
// when that was below the tag.
__device__ __forceinline__ uint32_t stamp_claim(int32_t *stamp, int32_t v, uint32_t tag) {
  return atomicMax(reinterpret_cast<uint32_t *>(stamp) + v, tag);
}
// The same without the answer, and without waiting for one: an atomicMax whose result
// is not used was waited for in three of the four fused SSSP loops (mesh session on a
// 200^2 grid, delta 32: 8.2 ms against 7.2).
__device__ __forceinline__ void stamp_raise(int32_t *stamp, int32_t v, uint32_t tag) {
  asm volatile("red.relaxed.gpu.global.max.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(stamp + v)), "r"(tag)
               : "memory");
}

// Far piles of the single-source delta-stepping queue (bucket_queue.cuh).  A
// relaxation that lowers P[v] to p at or above the window's cutoff parks v on
// the low pile (p below the horizon) or the high pile.  stamp[v] holds the tag
// of the pile generation that already lists v, so each vertex is listed at most
// once per pile: the claim that raises the stamp to the tag decides who appends
// (the order of tags is in bucket_queue.cuh).  With stamp == nullptr nothing is
// parked (a plain edgeset.apply of the relax UDF).
struct DFar {
  int32_t *stamp;           // [V]
  int32_t *lo, *lo_cnt;     // low pile of the current generation and its count
  int32_t *hi, *hi_cnt;     // high pile of the current generation and its count
  uint32_t lo_tag, hi_tag;
  int32_t horizon;          // p < horizon -> low pile
  int32_t cap;              // entries a pile can hold (V)
  int32_t *err;
  Stage *lo_stage, *hi_stage;  // shared memory, or null: append directly
  // Mark of this step's frontier, or 0: improvements below the cutoff queue their
  // vertex every time.  With it a vertex is queued once a step, and a park that
  // another thread of the step decided on an older distance is refused.
  uint32_t near_tag;
  // The same for a thread that walks a hub alone: near_tag, or 0 in a step whose
  // queue holds what its threads find unclaimed too (BqArgs::alone_max).
  uint32_t near_alone;

  __device__ __forceinline__ uint32_t tag_of(int32_t p) const { return p < horizon ? lo_tag : hi_tag; }
  __device__ __forceinline__ void park(int32_t v, int32_t p) const {
    if (stamp_claim(stamp, v, tag_of(p)) < tag_of(p)) append(v, p);
  }
  __device__ __forceinline__ void append(int32_t v, int32_t p) const {
    if (p < horizon)
      pile_append(lo_stage, lo, lo_cnt, cap, v, err);
    else
      pile_append(hi_stage, hi, hi_cnt, cap, v, err);
  }
  // Sends what the CTA staged (all of it, or when less than half is left); the whole
  // CTA calls it, as stage_flush and stage_make_room.
  __device__ __forceinline__ void flush() const {
    if (!lo_stage) return;
    stage_flush(lo_stage, lo, lo_cnt, cap, err);
    stage_flush(hi_stage, hi, hi_cnt, cap, err);
  }
  __device__ __forceinline__ void make_room() const {  // at half a stage
    if (!lo_stage || (lo_stage->n <= lo_stage->cap / 2 && hi_stage->n <= hi_stage->cap / 2)) return;
    flush();
    __syncthreads();
  }
};

// --------------------------------------------------------------- barriers
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier for persistent (cooperatively launched) kernels.  bar is
// one 64-bit arrival count (two words, cleared before the launch) that only
// grows: a block's own arrival tells it which barrier this is, and the wait is
// for the count to reach the end of that barrier.  The wait is bounded by
// timeout_ns; on expiry DEV_ERR_TIMEOUT is raised in *err and the function
// returns false so the caller can leave its loop.  Replaces
// cooperative_groups::this_grid().sync() (gpu_intrinsics.h:113-117), whose wait
// has no limit.
//
// A barrier is a chain of dependent L2 round trips (0.65 us each here with
// gpu-scope ordering), not of bandwidth: with a generation word it took four
// (read it, arrive, publish it, see it), 2.5 us at 304 blocks and 3.1 us at
// 608; arriving and polling one count takes two, 1.5 us and 2.2 us.  64 bits,
// because a loop of a 1.5 us barrier passes 2^32 arrivals within seconds.  The
// wait reads without acquire semantics and one fence follows it: an acquiring
// read drops the L1 of its SM, and with most blocks waiting it did so under the
// ones still at work (BFS on a symmetrized R-MAT 20, a thread per vertex: 91 ms,
// 81 without).
//
// `behind` runs on one thread behind the barrier, before its block goes on: loops
// fetch the words that every thread needs (counts, the stop word) there and hand
// them on in shared memory.  Read by every warp of the GPU they are 10^4 requests a
// word for one line of the L2, answered one after another (BFS on a 1024^2 grid,
// 2,046 levels of about 1,000 vertices: 24.3 ms with three words read by every warp,
// 20.0 with two, 12.6 with one thread a block reading them).
__device__ __forceinline__ uint64_t ld_acquire64(const uint32_t *p) {
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t ld_relaxed64(const uint32_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
template <class Behind>
__device__ __forceinline__ bool grid_barrier_then(uint32_t *bar, uint32_t nblocks, int32_t *err,
                                                  uint64_t timeout_ns, const Behind &behind) {
  __syncthreads();
  __shared__ int ok_s;
  if (threadIdx.x == 0) {
    ok_s = 1;
    uint64_t old;
    asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(old) : "l"(bar) : "memory");
    const uint64_t end = (old / nblocks + 1) * nblocks;
    if (old + 1 != end) {
      const uint64_t t0 = globaltimer_ns();
      uint32_t spins = 0;
      while (ld_relaxed64(bar) < end) {
        if ((++spins & 255u) == 0) {
          if (*(volatile int32_t *)err & DEV_ERR_TIMEOUT) { ok_s = 0; break; }
          if (globaltimer_ns() - t0 > timeout_ns) {
            atomicOr(err, DEV_ERR_TIMEOUT);
            ok_s = 0;
            break;
          }
        }
      }
    }
    __threadfence();
    behind();
  }
  __syncthreads();
  return ok_s != 0;
}
__device__ __forceinline__ bool grid_barrier(uint32_t *bar, uint32_t nblocks, int32_t *err, uint64_t timeout_ns) {
  return grid_barrier_then(bar, nblocks, err, timeout_ns, [] {});
}

// Waits, without arriving, until every other block has arrived at the next
// grid_barrier (the count, modulo nblocks, is the arrivals of the barrier that is
// open, and this block's is missing: nblocks-1 of them mean all others are inside
// the wait).  The caller then works alone and completes the barrier by calling
// grid_barrier itself.  Bounded like grid_barrier; false after the limit.
__device__ __forceinline__ bool grid_wait_others(const uint32_t *bar, uint32_t nblocks, int32_t *err,
                                                 uint64_t timeout_ns) {
  __shared__ int ok_o;
  if (threadIdx.x == 0) {
    ok_o = 1;
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    const uint64_t all = ld_acquire64(bar) / nblocks * nblocks + nblocks - 1;
    while (ld_acquire64(bar) < all) {
      if ((++spins & 255u) == 0) {
        if (*(volatile int32_t *)err & DEV_ERR_TIMEOUT) { ok_o = 0; break; }
        if (globaltimer_ns() - t0 > timeout_ns) {
          atomicOr(err, DEV_ERR_TIMEOUT);
          ok_o = 0;
          break;
        }
      }
      __nanosleep(32);
    }
  }
  __syncthreads();
  return ok_o != 0;
}

// Wall-clock bound of a persistent loop.  In iteration `iter`, just before its
// closing grid barrier, block 0 checks the clock and, the first time it has
// passed, records DEV_ERR_TIMEOUT and writes iter + 1 into *stop: the number
// of the iteration at whose top every block leaves.  A number rather than a
// flag: a block that reads *stop late at the top of iteration `iter` (block 0
// may already be past that point) sees iter + 1 and goes on, so all blocks
// still leave together at the top of iteration iter + 1.
struct LoopClock {
  uint64_t deadline;
  __device__ __forceinline__ void start(uint64_t limit_ns) { deadline = globaltimer_ns() + limit_ns; }
  __device__ __forceinline__ void tick(int32_t *stop, int32_t iter, int32_t *err) const {
    if (blockIdx.x == 0 && threadIdx.x == 0 && globaltimer_ns() > deadline &&
        atomicCAS(stop, 0, iter + 1) == 0)
      atomicOr(err, DEV_ERR_TIMEOUT);
  }
};
// True at the top of iteration `iter` once a stop has been set for it: for the stop
// word as read behind the closing barrier of the iteration before, or any time since.
__device__ __forceinline__ bool stop_reached(int32_t stop, int32_t iter) { return stop != 0 && iter >= stop; }
__device__ __forceinline__ bool stopped(const int32_t *stop, int32_t iter) {
  return stop_reached(*(volatile const int32_t *)stop, iter);
}
// The same stop for a reason other than the clock (block 0, before the
// iteration's closing barrier): a sparse queue that overflowed.
__device__ __forceinline__ void stop_on_overflow(int32_t *stop, int32_t iter, const int32_t *err) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && (*(volatile const int32_t *)err & DEV_ERR_OVERFLOW))
    atomicCAS(stop, 0, iter + 1);
}

__host__ __device__ __forceinline__ int32_t ceil_div(int64_t a, int64_t b) {
  return (int32_t)((a + b - 1) / b);
}

}  // namespace gg

#define GG_CUDA(call)                                                              \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess)                                                         \
      return gg::set_error(e_ == cudaErrorMemoryAllocation ? GG_ERR_OOM : GG_ERR_CUDA, \
                           "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                           __FILE__, __LINE__);                                    \
  } while (0)

#define GG_TRY(expr)                  \
  do {                                \
    gg_status s_ = (expr);            \
    if (s_ != GG_OK) return s_;       \
  } while (0)
