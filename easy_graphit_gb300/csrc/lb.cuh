// Load-balancing strategies of GraphIt's edgeset.apply
// (src/graphit/operators.cpp:72-492), each written as a device function that
// processes one *virtual CTA* of work.  Kernels (unfused launches, persistent
// fused kernels) loop over virtual CTAs, so every strategy runs unchanged in
// both modes -- the multiplexing the reference does for fused kernels
// (operators.cpp:337-342) is the normal path here.
//
// F is an edge functor (udf.cuh) with
//   bool src_ok(s)  -- source filter, checked before every edge (pull early exit)
//   bool dst_ok(d)  -- destination filter
//   int  apply(s, d, w) -> vertex to enqueue into the output frontier or -1
//   static constexpr bool kWeight -- whether apply reads the edge weight
#pragma once

#include "common.cuh"

namespace gg {

constexpr int kStage1 = 8;  // TWCE stage-1 group width (operators.cpp:201)

template <class F>
__device__ __forceinline__ void do_edge(const DGraph &g, const F &f, const DOut &out, int32_t s,
                                        int32_t k) {
  const int32_t d = __ldg(g.dst + k);
  if (!f.dst_ok(d)) return;
  const int32_t w = F::kWeight ? __ldg(g.w + k) : 0;
  const int32_t t = f.apply(s, d, w);
  if (t >= 0) out.push(t);
}

template <class F, class = void>
struct lb_batch {
  static constexpr bool value = false;
};
template <class F>
struct lb_batch<F, decltype(void(F::kBatch))> {
  static constexpr bool value = F::kBatch;
};

// Whether a functor pulls (EdgeF).
template <class F, class = void>
struct lb_pulls {
  static constexpr bool value = false;
};
template <class F>
struct lb_pulls<F, decltype(void(F::kPulls))> {
  static constexpr bool value = F::kPulls;
};

// Edges [b, e) of source s processed by `width` cooperating threads (rank r).
// A functor with a batched range relax (push, no per-edge source test beyond
// the first) takes the whole range at once, B edges of a thread in flight.
template <int B = 4, class F>
__device__ __forceinline__ void do_range(const DGraph &g, const F &f, const DOut &out, int32_t s,
                                         int32_t b, int32_t e, int32_t r, int32_t width) {
  if constexpr (lb_batch<F>::value) {
    if (b + r < e && f.src_ok(s)) f.template relax_range<B>(g, out, s, b, e, r, width);
    return;
  }
  for (int32_t k = b + r; k < e; k += width) {
    if (!f.src_ok(s)) break;
    do_edge(g, f, out, s, k);
  }
}

// ------------------------------------------------------------ VERTEX_BASED
// Edges a thread that walks a longer list alone has in flight (batched relax): a
// hub's list is a chain of such batches (R-MAT of 250,000 vertices, 4 / 8 / 12 in
// flight: 14.4 / 12.8 / 12.1 ms; 12 takes registers the other steps need).
constexpr int kSerialInFlight = 8;
// One thread per enumerated vertex, serial neighbour loop with the early exit
// of operators.cpp:83-94.  Virtual CTA = blockDim.x vertices.
template <class F>
__device__ __forceinline__ void lb_vertex(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                          const DOut &out, int32_t vcta) {
  const int32_t i = vcta * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t s = en.at(i);
  const int32_t b = __ldg(g.off + s), e = __ldg(g.off + s + 1);
  // a pull appends the thread's own vertex at most
  if (lb_pulls<F>::value || e - b <= 4) {
    do_range(g, f, out, s, b, e, 0, 1);
    return;
  }
  // A hub's thread would fill the stages, then try them for nothing: it appends
  // directly.  The relax has one loop for both (two cost the others registers: directed
  // R-MAT 22, SSSP at delta 32, 66.8 against 67.6 ms); elsewhere a loop of its own, which
  // knows that there is no stage (unfused BFS, symmetrized R-MAT 20: 99.0 -> 95.0).
  const bool hub = e - b > kStageCap / 2;
  if constexpr (lb_batch<F>::value) {
    DOut o = out;
    F h = f;
    if (hub) {
      o.stage = nullptr;
      h.alone();
    }
    do_range<kSerialInFlight>(g, h, o, s, b, e, 0, 1);
  } else if (hub) {
    DOut o = out;
    o.stage = nullptr;
    do_range(g, f, o, s, b, e, 0, 1);
  } else {
    do_range(g, f, out, s, b, e, 0, 1);
  }
}

// ---------------------------------------------------------------------- WM
// Warp-mapped: one warp per enumerated vertex, lanes stride the neighbour list
// (coalesced dst loads).  Virtual CTA = blockDim.x/32 vertices.  No reference
// implementation (schedule.h lists WM, operators.cpp:645-646 rejects it).
template <class F>
__device__ __forceinline__ void lb_wm(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                      const DOut &out, int32_t vcta) {
  const int32_t nw = blockDim.x >> 5;
  const int32_t i = vcta * nw + (threadIdx.x >> 5);
  if (i >= n) return;
  const int32_t s = en.at(i);
  do_range(g, f, out, s, __ldg(g.off + s), __ldg(g.off + s + 1), threadIdx.x & 31, 32);
}

// -------------------------------------------------------------------- TWCE
// Thread/warp/CTA binning inside one CTA (operators.cpp:203-323): 8 threads
// read one vertex; its degree splits into a CTA part (multiples of blockDim),
// a warp part (multiples of 32) and a remainder for the 8-thread group.
// Warp-bin entries are taken round-robin by the warps, CTA-bin entries by the
// whole CTA.  Virtual CTA = blockDim.x/8 vertices.
//
// Two things keep a skewed frontier from leaving the GPU idle behind one CTA:
//  * slices: a frontier with fewer virtual CTAs than there are CTAs gives
//    each virtual CTA `nslices` of them; all bin the same vertices and split
//    every part of their lists between them;
//  * hub list: a CTA part of at least hub.min edges (times the slices) goes to
//    a global list as chunks of kHubChunk CTA widths, which all CTAs drain in a
//    pass of their own (lb_chunk) -- one R-MAT hub is otherwise 10^2 rounds of
//    one CTA while the others wait at the level's end.
// A level-1 frontier of one 180,000-edge hub (R-MAT 22) took 376 us on one CTA.
struct TwceSmem {
  int32_t nw, nc;
  int32_t data[1];  // 6 * (blockDim/8) ints: warp bin (s,b,e), CTA bin (s,b,e)
};
__host__ __device__ inline size_t twce_smem_bytes(int cta) {
  return sizeof(int32_t) * (2 + 6 * (cta / kStage1)) + 16;
}

constexpr int32_t kHubChunk = 4;   // CTA widths per chunk: one round of a 4-edges-in-flight relax
constexpr int32_t kHubWidths = 8;  // CTA widths from which a list is split over the CTAs

struct HubList {
  int32_t *list = nullptr;  // [cap][3]: vertex, first edge, end edge; null: no list
  int32_t *cnt = nullptr;   // chunks appended; may pass cap, the surplus was not written
  int32_t cap = 0;
  int32_t min = 0;          // edges of a CTA part from which it goes to the list
  int32_t slices = INT_MAX; // most slices of a virtual CTA (slice_limit)
};

// Slices that the graph's longest list has work for, 8 edges each (stage 1 gives a
// slice no fewer).  On a mesh that is one: the CTAs that a level of a few vertices
// does not fill stay out of it instead of reading the same vertices (BFS on a 200^2
// grid, fused 2.08 -> 1.98 ms, ETWC 15.7 -> 13.9; ten PageRank iterations on a line of
// 20,000, TWCE 153 -> 100 us).
__host__ __device__ inline int32_t slice_limit(int32_t max_degree) {
  return max_degree <= kStage1 ? 1 : ceil_div(max_degree, kStage1);
}

// Appends the chunks of [b, e) of vertex s; false (and no live chunk) when they
// do not all fit.
__device__ __forceinline__ bool hub_append(const HubList &hub, int32_t s, int32_t b, int32_t e) {
  const int32_t chunk = kHubChunk * (int32_t)blockDim.x;
  const int32_t nch = ceil_div(e - b, chunk);
  const int32_t p = atomicAdd(hub.cnt, nch);
  const bool fits = (int64_t)p + nch <= hub.cap;
  for (int32_t c = 0; c < nch && (int64_t)p + c < hub.cap; ++c) {
    int32_t *d = hub.list + 3 * (int64_t)(p + c);
    d[0] = s;
    d[1] = fits ? b + c * chunk : 0;
    d[2] = fits ? min(b + (c + 1) * chunk, e) : 0;
  }
  return fits;
}

template <class F>
__device__ __forceinline__ void lb_twce(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                          const DOut &out, int32_t vcta, int32_t slice, int32_t nslices,
                                          TwceSmem &sm, const HubList &hub) {
  const int32_t per = blockDim.x / kStage1;
  int32_t *wv = sm.data, *wb = wv + per, *we = wb + per;
  int32_t *cv = we + per, *cb = cv + per, *ce = cb + per;
  if (threadIdx.x == 0) {
    sm.nw = 0;
    sm.nc = 0;
  }
  const int32_t sub = threadIdx.x & (kStage1 - 1);
  const int32_t i = vcta * per + (int32_t)(threadIdx.x / kStage1);
  int32_t s = -1, b = 0, e = 0;
  if (i < n) {
    s = en.at(i);
    b = __ldg(g.off + s);
    e = __ldg(g.off + s + 1);
  }
  __syncthreads();
  if (s >= 0) {
    const int32_t deg = e - b;
    const int32_t big = deg / (int32_t)blockDim.x * (int32_t)blockDim.x;
    const int32_t mid = (deg - big) / 32 * 32;
    if (sub == 0) {
      const bool is_hub = hub.list && big >= hub.min * (int64_t)nslices;
      if (big && !(is_hub && slice != 0)) {
        bool listed = false, alone = false;  // alone: one slice takes it all
        if (is_hub) {
          listed = hub_append(hub, s, b, b + big);
          alone = !listed;
        }
        if (!listed) {
          const int32_t p = atomicAdd(&sm.nc, 1);
          cv[p] = s;
          cb[p] = b;
          ce[p] = alone ? ~(b + big) : b + big;
        }
      }
      if (mid) {
        // pieces of 32 edges, a run of them for each of the first slices counted
        // from slice i (bins differ in order between slices, vertices do not)
        const int32_t pieces = (mid + 31) >> 5, ways = min(nslices, pieces);
        int32_t t = slice - i % nslices;
        if (t < 0) t += nslices;
        if (t < ways) {
          const int32_t p = atomicAdd(&sm.nw, 1);
          wv[p] = s;
          wb[p] = b + big + pieces * t / ways * 32;
          we[p] = min(b + big + pieces * (t + 1) / ways * 32, b + big + mid);
        }
      }
    }
    b += big + mid;
  }
  __syncthreads();
  {  // stage 1: the remainders, 8 edges to each of the first slices
    const int32_t ways = min(nslices, 32 / kStage1);
    if (s >= 0 && slice < ways) do_range(g, f, out, s, b, e, slice * kStage1 + sub, kStage1 * ways);
  }
  const int32_t nw = sm.nw, warps = (int32_t)(blockDim.x >> 5);
  for (int32_t j = (int32_t)(threadIdx.x >> 5); j < nw; j += warps)  // stage 2
    do_range(g, f, out, wv[j], wb[j], we[j], threadIdx.x & 31, 32);
  const int32_t nc = sm.nc;
  for (int32_t j = 0; j < nc; ++j) {  // stage 3
    const int32_t end = ce[j];
    if (end < 0)
      do_range(g, f, out, cv[j], cb[j], ~end, threadIdx.x, blockDim.x);
    else
      do_range(g, f, out, cv[j], cb[j], end, slice * (int32_t)blockDim.x + threadIdx.x,
               nslices * (int32_t)blockDim.x);
  }
  __syncthreads();
}

// Between virtual CTAs: room in the stages of the output queue and, for a
// functor that parks, of its piles.
template <class F>
__device__ __forceinline__ void lb_make_room(const F &f, const DOut &out) {
  if (out.stage) stage_make_room(out, out.stage->cap / 2);
  if constexpr (lb_batch<F>::value) f.make_room();
}

// TWCE over n vertices by CTA `rank` of `nparts`: whole
// virtual CTAs in turn, or slices of them when there are fewer than CTAs.
template <class F>
__device__ __forceinline__ void lb_twce_all(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                          const DOut &out, int32_t rank, int32_t nparts, TwceSmem &sm,
                                          const HubList &hub) {
  const int32_t nv = ceil_div(n, blockDim.x / kStage1);
  if (nv >= nparts) {
    for (int32_t v = rank; v < nv; v += nparts) {
      lb_twce(g, en, n, f, out, v, 0, 1, sm, hub);
      lb_make_room(f, out);
    }
  } else if (nv > 0) {
    const int32_t slices = min(nparts / nv, hub.slices);
    if (rank < nv * slices) lb_twce(g, en, n, f, out, rank % nv, rank / nv, slices, sm, hub);
  }
}

// A virtual CTA processes one chunk of a hub list.
template <class F>
__device__ __forceinline__ void lb_chunk(const DGraph &g, const int32_t *chunk_list, const F &f,
                                         const DOut &out, int32_t vcta) {
  const int32_t *d = chunk_list + 3 * (int64_t)vcta;
  const int32_t s = __ldcg(d), b = __ldcg(d + 1), e = __ldcg(d + 2);
  do_range(g, f, out, s, b, e, threadIdx.x, blockDim.x);
}

// CTA `rank` of `nparts` drains its share of a hub list of `chunks` entries.
template <class F>
__device__ __forceinline__ void lb_hubs(const DGraph &g, const HubList &hub, int32_t chunks, const F &f,
                                        const DOut &out, int32_t rank, int32_t nparts) {
  for (int32_t c = rank; c < min(chunks, hub.cap); c += nparts) {
    lb_chunk(g, hub.list, f, out, c);
    if (out.stage) {
      __syncthreads();
      lb_make_room(f, out);
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------- CM
// CTA-wide exclusive scan of the degrees of blockDim.x frontier vertices, then
// every thread takes edges i, i+blockDim.x, ... and finds its source by an
// upper-bound search in the scan (operators.cpp:359-457).  The reference passes
// weight 0 to the UDF here (operators.cpp:451-452); this one passes the edge's
// weight.
struct CmSmem {
  int32_t total;
  int32_t warp_sums[32];
  int32_t data[1];  // 3*blockDim ints: vertex, begin, exclusive scan
};
__host__ __device__ inline size_t cm_smem_bytes(int cta) {
  return sizeof(int32_t) * (1 + 32 + 3 * cta) + 16;
}

// Block-wide exclusive scan of x; returns the exclusive prefix, total in *tot.
__device__ __forceinline__ int32_t block_exclusive_scan(int32_t x, int32_t *warp_sums,
                                                        int32_t *tot) {
  const int32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t v = x;
#pragma unroll
  for (int32_t d = 1; d < 32; d <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  if (lane == 31) warp_sums[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int32_t nwarps = blockDim.x >> 5;
    int32_t ws = lane < nwarps ? warp_sums[lane] : 0;
#pragma unroll
    for (int32_t d = 1; d < 32; d <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, ws, d);
      if (lane >= d) ws += t;
    }
    if (lane < nwarps) warp_sums[lane] = ws;  // inclusive over warps
  }
  __syncthreads();
  const int32_t base = wid ? warp_sums[wid - 1] : 0;
  *tot = warp_sums[(blockDim.x >> 5) - 1];
  return base + v - x;
}

template <class F>
__device__ __forceinline__ void lb_cm(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                      const DOut &out, int32_t vcta, CmSmem &sm) {
  const int32_t C = blockDim.x;
  int32_t *sv = sm.data, *sb = sv + C, *sx = sb + C;
  const int32_t i = vcta * C + threadIdx.x;
  int32_t deg = 0;
  if (i < n) {
    const int32_t s = en.at(i);
    const int32_t b = __ldg(g.off + s);
    deg = __ldg(g.off + s + 1) - b;
    sv[threadIdx.x] = s;
    sb[threadIdx.x] = b;
  }
  int32_t total;
  const int32_t ex = block_exclusive_scan(deg, sm.warp_sums, &total);
  sx[threadIdx.x] = ex;
  __syncthreads();
  const int32_t width = min(C, n - vcta * C);
  for (int32_t e = threadIdx.x; e < total; e += C) {
    // upper_bound(sx[0..width), e) - 1
    int32_t lo = 0, len = width;
    while (len > 0) {
      const int32_t half = len >> 1;
      if (sx[lo + half] > e) {
        len = half;
      } else {
        lo += half + 1;
        len -= half + 1;
      }
    }
    const int32_t j = lo - 1;
    const int32_t s = sv[j];
    if (!f.src_ok(s)) continue;
    do_edge(g, f, out, s, sb[j] + e - sx[j]);
  }
  __syncthreads();
}

// ------------------------------------------------------------------ STRICT
// Edge-balanced over the whole frontier: `sum` holds the exclusive scan of the
// enumerated vertices' degrees (n+1 entries); virtual CTA c owns edge ranks
// [c*per, (c+1)*per).  (The reference allocates strict_* scratch,
// graph.h:56-59, but implements no kernel.)
template <class F>
__device__ __forceinline__ void lb_strict(const DGraph &g, const Enum &en, int32_t n,
                                          const int32_t *__restrict__ sum, const F &f,
                                          const DOut &out, int32_t vcta, int32_t per) {
  const int64_t total = sum[n];
  const int64_t r0 = (int64_t)vcta * per;
  const int64_t r1 = r0 + per < total ? r0 + per : total;
  for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    int32_t lo = 0, len = n;
    while (len > 0) {
      const int32_t half = len >> 1;
      if (__ldg(sum + lo + half) > r) {
        len = half;
      } else {
        lo += half + 1;
        len -= half + 1;
      }
    }
    const int32_t j = lo - 1;
    const int32_t s = en.at(j);
    if (!f.src_ok(s)) continue;
    do_edge(g, f, out, s, __ldg(g.off + s) + (int32_t)(r - __ldg(sum + j)));
  }
}

// ---------------------------------------------------- EDGE_ONLY, run sums
// Edges [e0, e1) for a functor that adds a term per edge to the enumerated end
// (PageRank, pull): the edge list holds a vertex's edges in a row -- whole lists,
// or their parts within a destination bucket -- so a warp sums the runs among 32
// consecutive edges and adds one value a run.  An atomic per edge is what bound
// this walk (1 M vertices, 15 M edges, four buckets: 142 us an iteration at 61 %
// of the L2's rate; now 56).  Four groups of 32 edges are in flight.
template <class F, class = void>
struct lb_run_sums {
  static constexpr bool value = false;
};
template <class F>
struct lb_run_sums<F, decltype(void(F::kRunSums))> {
  static constexpr bool value = F::kRunSums;
};
template <class F>
__device__ __forceinline__ void lb_edge_runs(const DGraph &g, const F &f, int64_t e0, int64_t e1, int64_t r,
                                             int64_t width) {
  constexpr int kIn = 4;
  const int32_t lane = threadIdx.x & 31;
  for (int64_t base = e0 + (r >> 5) * (32 * kIn); base < e1; base += (width >> 5) * (32 * kIn)) {
    int32_t s[kIn], d[kIn];
    float x[kIn];
    bool ok[kIn];
#pragma unroll
    for (int j = 0; j < kIn; ++j) {
      const int64_t k = base + j * 32 + lane;
      s[j] = k < e1 ? __ldg(g.src + k) : -1;
      d[j] = k < e1 ? __ldg(g.dst + k) : -1;
    }
#pragma unroll
    for (int j = 0; j < kIn; ++j) {
      ok[j] = d[j] >= 0 && f.src_ok(s[j]) && f.dst_ok(d[j]);
      x[j] = ok[j] ? f.term(d[j]) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kIn; ++j) {
      const int32_t before = __shfl_up_sync(0xffffffffu, s[j], 1);  // by all lanes, lane 0 too
      const bool head = lane == 0 || before != s[j];
      const uint32_t heads = __ballot_sync(0xffffffffu, head), oks = __ballot_sync(0xffffffffu, ok[j]);
      const uint32_t after = lane == 31 ? 0u : heads >> (lane + 1);
      const int32_t end = after ? lane + __ffs(after) : 32;  // first lane past this one's run
#pragma unroll
      for (int i = 1; i < 32; i <<= 1) {
        const float o = __shfl_down_sync(0xffffffffu, x[j], i);
        if (lane + i < end) x[j] += o;
      }
      const uint32_t run = (end == 32 ? ~0u : (1u << end) - 1u) & ~((1u << lane) - 1u);
      if (head && (oks & run)) f.add(s[j], x[j]);
    }
  }
}

// --------------------------------------------------------------- EDGE_ONLY
// Thread per COO edge over every edge of the graph (operators.cpp:175-200);
// both endpoints go through the filters.  `r`/`width` index the calling
// thread within the grid.
template <class F>
__device__ __forceinline__ void lb_edge_only(const DGraph &g, const F &f, const DOut &out,
                                             int64_t r, int64_t width) {
  if constexpr (lb_run_sums<F>::value) {
    lb_edge_runs(g, f, 0, g.E, r, width);
    return;
  }
  for (int64_t k = r; k < g.E; k += width) {
    const int32_t s = __ldg(g.src + k);
    if (!f.src_ok(s)) continue;
    do_edge(g, f, out, s, (int32_t)k);
  }
}

// Blocked variant (operators.cpp:131-172): edges bucketed by destination
// block, buckets walked in order with a CTA barrier between them so the CTAs
// of a wave work on the same block of destinations.
template <class F>
__device__ __forceinline__ void lb_edge_only_blocked(const DGraph &g, const F &f, const DOut &out,
                                                     int64_t r, int64_t width) {
  for (int32_t b = 0; b < g.nbuckets; ++b) {
    const int32_t e0 = __ldg(g.bucket + b), e1 = __ldg(g.bucket + b + 1);
    if constexpr (lb_run_sums<F>::value) {
      lb_edge_runs(g, f, e0, e1, r, width);
      __syncthreads();
      continue;
    }
    for (int64_t k = e0 + r; k < e1; k += width) {
      const int32_t s = __ldg(g.src + k);
      if (!f.src_ok(s)) continue;
      do_edge(g, f, out, s, (int32_t)k);
    }
    __syncthreads();
  }
}

}  // namespace gg
