// Batched BC: up to 64 sources per pass in one persistent kernel.
//
// The per-source algorithm is apps/bc.cpp:28-123 (Brandes with the stored
// quantity dep' = (1 + delta) / sigma):
//   forward   sigma[v] = sum of sigma[u] over in-neighbours u one level up;
//   backward  dep'[v] = 1/sigma[v] + sum of dep'[u] over in-neighbours u at a
//             deeper level (bc.cpp pushes dep'[src] to unvisited out-neighbours,
//             i.e. every vertex receives from its in-neighbours that sit deeper);
//   final     delta[v] = (dep'[v] - 1/sigma[v]) * sigma[v], 0 when unreached.
//
// 64 sources share one traversal.  The levels come from the bit-parallel
// multi-source BFS of batch_bfs.cu (one edge visit serves all sources), whose
// queues are kept back to back as the level list Q_0, Q_1, ... (a vertex is in
// Q_d when some source first reaches it at level d).  Per-source values live
// vertex-major -- sigma[v][64], dep'[v][64] in fp64, depth[v][64] in uint16 --
// so the two gathers use one warp per (vertex, chunk of in-edges) work item with
// lane l owning sources l and l + 32: each in-neighbour costs one broadcast
// 8-byte mask load, and only the sources whose bit survives read the neighbour's
// 8-byte value.  A vertex of one chunk writes its own values (no atomics);
// hubs' chunks add fp64 partial sums atomically (sigma sums are integers, exact
// in any order).  dep' is accumulated in fp64 and written out as fp32.
//
// Grid barriers per level: two forward ([sigma of level d] + [relax of level
// d+1] | [publish of level d+1]) and two backward ([mask update of level d+1] +
// [scan of level d] | [gather of level d]).
#include <vector>

#include "batch.h"
#include "lb.cuh"

namespace gg {

constexpr int32_t kBcWidth = 64;         // sources per pass (mask bits)
constexpr int32_t kBcInFlight = 2;       // rows of a gather in flight, per lane and half
// Longest list that is one light work item (0.5 M vertices of degree 30, 64 sources,
// at 32 / 64 / 128 / 256: 7.35 / 7.34 / 7.40 / 7.41 ms; uniform degree 32, 1 M: 18.5 / 17.9 /
// 17.9 / 17.9).
constexpr int32_t kBcLight = 128;
constexpr int32_t kBcMaxLevels = 65534;  // depth is stored as uint16; 0xFFFF = unreached

struct BcState {
  uint64_t *seen, *acc, *rmask;  // rmask[v]: sources whose level at v is deeper than the current one
  uint64_t *fr[3];               // level masks, by level mod 3
  uint64_t *lm[2];               // backward: sources at v's current level, by level parity
  int32_t *qstamp;
  int32_t *lev;                  // level list
  int32_t levcap;
  int32_t *loff;                 // [kBcMaxLevels + 2] start of each level in lev
  int64_t *work;                 // (v << 32 | chunk)
  int32_t wcap;
  int32_t chunk;                 // in-edges per work item (the graph's batch tuning)
  int32_t light;                 // longest list that is one light work item: kBcLight or the chunk
  int32_t *ctr;                  // [0] level-list end, [1..2] forward items, [3..4] backward items,
                                 // [16..19] hand-out counters, [20] end of Q_0, [21..23] hub chunks;
                                 // [24..27] long items and [28..31] their hand-out, as [1..4], [16..19]
  uint16_t *depth;               // [V][64]
  double *sigma, *dep;           // [V][64]
  const int32_t *toff, *tsrc;    // in-neighbours (the CSR itself for a symmetric graph)
  const int32_t *perm;           // original id -> walked id (degree-ordered copy), or null
  int32_t V, nsrc;
  uint32_t *bar;
  int32_t *err;
  uint64_t timeout_ns;
  int32_t *hub_list;             // hub chunks of a relax (counts: ctr[21..23], by level)
  int32_t hub_cap, hub_slices;
  int32_t *stats;                // [0] levels
  int32_t *stop;
  uint64_t loop_limit_ns;
};

// Appends the work items of this lane's vertex (degree deg, -1 for a lane
// without one); the whole warp calls it together.  Lists up to st.light edges
// are one item at the front of the work array (count wcnt), longer ones items of
// st.chunk edges from its back (count hcnt): the two are handed out differently.
__device__ __forceinline__ void bc_push_items(const BcState &st, int32_t *wcnt, int32_t *hcnt, int32_t v,
                                              int32_t deg) {
  const int32_t lane = threadIdx.x & 31;
  const bool light = deg >= 0 && deg <= st.light;
  const uint32_t lights = __ballot_sync(0xffffffffu, light);
  if (lights) {
    int32_t base = 0;
    if (lane == __ffs(lights) - 1) base = atomicAdd(wcnt, __popc(lights));
    base = __shfl_sync(0xffffffffu, base, __ffs(lights) - 1);
    const int32_t at = base + __popc(lights & ((1u << lane) - 1));
    if (light) {
      if (at < st.wcap)
        st.work[at] = (int64_t)v << 32;
      else
        atomicOr(st.err, DEV_ERR_OVERFLOW);
    }
  }
  const int32_t nch = deg > st.light ? (deg + st.chunk - 1) / st.chunk : 0;
  if (!__any_sync(0xffffffffu, nch > 0)) return;
  int32_t incl = nch;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
  int32_t base = 0;
  if (lane == 31) base = atomicAdd(hcnt, total);
  base = __shfl_sync(0xffffffffu, base, 31);
  const int32_t first = base + incl - nch;
  for (int32_t c = 0; c < nch; ++c) {
    if (first + c >= st.wcap) {
      atomicOr(st.err, DEV_ERR_OVERFLOW);
      break;
    }
    st.work[st.wcap - 1 - (first + c)] = ((int64_t)v << 32) | (uint32_t)c;
  }
}

// Selects a level array without indexing the kernel-parameter arrays
// dynamically (which would copy them to local memory).
__device__ __forceinline__ uint64_t *bc_fr(const BcState &st, int32_t level) {
  const int32_t i = level % 3;
  return i == 0 ? st.fr[0] : (i == 1 ? st.fr[1] : st.fr[2]);
}
__device__ __forceinline__ uint64_t *bc_lm(const BcState &st, int32_t level) {
  return (level & 1) ? st.lm[1] : st.lm[0];
}

__device__ __forceinline__ int32_t bc_degree(const BcState &st, int32_t v) {
  return __ldg(st.toff + v + 1) - __ldg(st.toff + v);
}

// Transposes a 32 x 32 bit matrix held a row per lane: bit i of lane l's result
// is bit l of lane i's x.  Five butterfly steps, halving the block size.
__device__ __forceinline__ uint32_t bc_transpose(uint32_t x) {
  const int32_t lane = threadIdx.x & 31;
  uint32_t low = 0x0000ffffu;  // the columns of a block's left half
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const uint32_t o = __shfl_xor_sync(0xffffffffu, x, d);
    x = (lane & d) ? (x & ~low) | ((o & ~low) >> d) : (x & low) | ((o & low) << d);
    low ^= low << (d >> 1);
  }
  return x;
}

// Gather over one work item: lane sums, for its sources s in `own`, val[u][s]
// over in-neighbours u whose mask has s, in list order.  Returns the two
// partial sums.  A warp reads 32 neighbours and their masks at once, a lane
// each (an item is bound by the round trips in a row), and transposes the masks:
// every lane then has the neighbours of its own two sources and walks those.
// The additions are what the gather costs beyond the loads -- the FP64 pipe
// takes a warp-wide one every 16 cycles, whatever lanes are in it -- so their
// number is the longest lane's list instead of twice the neighbours that any
// source needs (0.5 M vertices, degree 30, 64 sources: 10.0 -> 8.6 ms).
__device__ __forceinline__ void bc_gather(const BcState &st, int32_t k0, int32_t k1, uint64_t own,
                                          const uint64_t *mask, const double *val, double &a0,
                                          double &a1) {
  const int32_t lane = threadIdx.x & 31;
  const double *v0 = val + lane, *v1 = v0 + 32;
  a0 = 0.0;
  a1 = 0.0;
  int32_t u = k0 + lane < k1 ? __ldg(st.tsrc + k0 + lane) : 0;
  for (int32_t k = k0; k < k1; k += 32) {
    const int32_t next = k + 32 + lane < k1 ? __ldg(st.tsrc + k + 32 + lane) : 0;
    const uint64_t m = k + lane < k1 ? __ldcg(mask + u) & own : 0ull;
    uint32_t t0 = bc_transpose((uint32_t)m), t1 = bc_transpose((uint32_t)(m >> 32));
    while (__any_sync(0xffffffffu, (t0 | t1) != 0u)) {
      double x[kBcInFlight], y[kBcInFlight];
#pragma unroll
      for (int j = 0; j < kBcInFlight; ++j) {
        const int32_t l0 = __ffs(t0) - 1, l1 = __ffs(t1) - 1;  // -1: none left (the shuffle wraps)
        const int32_t u0 = __shfl_sync(0xffffffffu, u, l0), u1 = __shfl_sync(0xffffffffu, u, l1);
        x[j] = t0 ? __ldcg(v0 + (int64_t)u0 * kBcWidth) : 0.0;
        y[j] = t1 ? __ldcg(v1 + (int64_t)u1 * kBcWidth) : 0.0;
        t0 &= t0 - 1;
        t1 &= t1 - 1;
      }
#pragma unroll
      for (int j = 0; j < kBcInFlight; ++j) {
        a0 += x[j];
        a1 += y[j];
      }
    }
    u = next;
  }
}

// Hand-out of a phase's work items to warps: the long ones first, one at a
// time, then the light ones in batches of up to 8 (half of what is left, spread
// over the warps), so that warps end the phase together.  With hub chunks and
// short lists in one list and batches of 32, a warp that drew a hub's
// neighbouring chunks worked for 3 ms while the rest of the GPU waited 2.2 ms
// of it at the barrier (0.5 M vertices, degree 30).
struct BcItems {
  const int32_t *cnt, *hcnt;  // items: light, long
  int32_t *wc, *hwc;          // hand-out counters
};
// Control words of the loop, read behind a barrier by one thread of the block
// (grid_barrier_then): the end of the level list, hub chunks, item counts, stop.
struct BcWords {
  int32_t end, chunks, light, longs, stop;
  __device__ __forceinline__ void items(const BcItems &w) {
    light = *(const volatile int32_t *)w.cnt;
    longs = *(const volatile int32_t *)w.hcnt;
  }
};
// False when none are left; items are work[i] for i in [i0, i1).
__device__ __forceinline__ bool bc_take(const BcState &st, const BcItems &w, int32_t n_light, int32_t n_long,
                                        int32_t nwarps, bool &longs, int32_t &i0, int32_t &i1) {
  const int32_t lane = threadIdx.x & 31;
  int32_t b = 0, B = 1;
  if (longs) {
    if (lane == 0) b = atomicAdd(w.hwc, 1);
    b = __shfl_sync(0xffffffffu, b, 0);
    if (b < n_long) {
      i0 = st.wcap - 1 - b;
      i1 = i0 + 1;
      return true;
    }
    longs = false;
  }
  if (lane == 0) {
    // a warp that finds the counter past the end takes nothing: in a level of a few
    // items the GPU's other 4,000 warps would queue on the counter
    const int32_t left = n_light - *(volatile int32_t *)w.wc;
    const int32_t per = (left / 2 + nwarps - 1) / nwarps;
    B = per < 1 ? 1 : (per > 8 ? 8 : per);
    b = left > 0 ? atomicAdd(w.wc, B) : n_light;
  }
  b = __shfl_sync(0xffffffffu, b, 0);
  B = __shfl_sync(0xffffffffu, B, 0);
  i0 = b;
  i1 = min(b + B, n_light);
  return b < n_light;
}

// f(v, chunk, first in-edge, end in-edge, whole list in one item) over a
// phase's items, a warp each.
template <class Fn>
__device__ __forceinline__ void bc_each_item(const BcState &st, const BcItems &w, const BcWords &words, int32_t nwarps,
                                             const Fn &f) {
  const int32_t n_light = min(words.light, st.wcap), n_long = min(words.longs, st.wcap);
  bool longs = n_long > 0;
  for (int32_t i0, i1; bc_take(st, w, n_light, n_long, nwarps, longs, i0, i1);)
    for (int32_t i = i0; i < i1; ++i) {
      const int64_t it = __ldcg(st.work + i);
      const int32_t v = (int32_t)(it >> 32), c = (int32_t)(uint32_t)it;
      const int32_t kb = __ldg(st.toff + v), ke = __ldg(st.toff + v + 1);
      if (ke - kb <= st.light)
        f(v, 0, kb, ke, true);
      else
        f(v, c, kb + c * st.chunk, min(ke, kb + (c + 1) * st.chunk), ke - kb <= st.chunk);
    }
}

// Items and hand-out counters of the gathers: forward, those of Q_{d+1} made by
// iteration d; backward, those of level dd.  Two of each by parity: a level's
// counts are cleared while the other's are in use.
__device__ __forceinline__ BcItems bc_forward_items(const BcState &st, int32_t d) {
  const int32_t i = d & 1;
  return BcItems{st.ctr + 1 + i, st.ctr + 24 + i, st.ctr + 16 + (1 - i), st.ctr + 28 + (1 - i)};
}
__device__ __forceinline__ BcItems bc_backward_items(const BcState &st, int32_t dd) {
  const int32_t i = dd & 1;
  return BcItems{st.ctr + 3 + i, st.ctr + 26 + i, st.ctr + 18 + i, st.ctr + 30 + i};
}

__global__ void __launch_bounds__(512, 2) k_bc_batch(DGraph g, BcState st) {
  extern __shared__ int4 smem[];
  __shared__ StageMem stage_mem;
  Stage &stage = stage_mem.s;
  __shared__ BcWords words;
  if (threadIdx.x == 0) {
    stage.init(kStageCap);
    words.stop = 0;
  }
  __syncthreads();
  const int32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t nthreads = gridDim.x * blockDim.x;
  const int32_t lane = threadIdx.x & 31;
  const int32_t nwarps = nthreads >> 5;
  LoopClock clk;
  clk.start(st.loop_limit_ns);
  bool alive = true;
  int32_t d = 0;
  int32_t b_prev = 0, b_d = 0;  // starts of Q_{d-1} and Q_d in the level list
  // End of Q_d in the level list.  Not read from the list's append counter at
  // the top of an iteration: a CTA that is ahead may already be appending
  // Q_{d+1} there while another still reads it, and CTAs that disagree on a
  // level's end disagree on when the loop ends (one leaves, the others wait at
  // the next grid barrier).  Q_0's end comes from a word the seed kernel wrote
  // and nothing appends to; each later one from the publish phase, which reads
  // the counter between the barrier that ends the appends and the one after
  // which the next level's appends begin.
  int32_t e_next = *(volatile int32_t *)(st.ctr + 20);
  // ------------------------------------------------------------- forward
  for (;; ++d) {
    const int32_t e_d = e_next;
    if (e_d == b_d) break;  // Q_d is empty
    if (stop_reached(words.stop, d)) {
      alive = false;
      break;
    }
    if (d + 1 > kBcMaxLevels) {
      if (tid == 0) atomicOr(st.err, DEV_ERR_OVERFLOW);
      alive = false;
      break;
    }
    if (tid == 0) {
      st.loff[d] = b_d;
      st.loff[d + 1] = e_d;
      st.ctr[1 + (d & 1)] = st.ctr[24 + (d & 1)] = 0;  // items of Q_{d+1}, filled by the publish below
      st.ctr[16 + ((d + 1) & 1)] = st.ctr[28 + ((d + 1) & 1)] = 0;  // hand-out of the next level's gather
      st.ctr[21 + (d + 1) % 3] = 0;    // hub chunks of the next level's relax
    }
    // sigma of Q_d from Q_{d-1} (items made by the previous publish)
    if (d > 0) {
      const uint64_t *pm = bc_fr(st, d - 1), *nm = bc_fr(st, d);
      bc_each_item(st, bc_forward_items(st, d - 1), words, nwarps,
                   [&](int32_t v, int32_t, int32_t k0, int32_t k1, bool single) {
        const uint64_t own = __ldcg(nm + v);
        double a0, a1;
        bc_gather(st, k0, k1, own, pm, st.sigma, a0, a1);
        double *row = st.sigma + (int64_t)v * kBcWidth;
        if ((own >> lane) & 1) {
          if (single) row[lane] = a0;
          else if (a0 != 0.0) atomicAdd(row + lane, a0);
        }
        if ((own >> (lane + 32)) & 1) {
          if (single) row[lane + 32] = a1;
          else if (a1 != 0.0) atomicAdd(row + lane + 32, a1);
        }
      });
    }
    // the mask array P(d) writes next held Q_{d-2}: clear those entries
    if (d >= 2) {
      uint64_t *old = bc_fr(st, d + 1);
      for (int32_t i = __ldcg(st.loff + d - 2) + tid; i < b_prev; i += nthreads) old[__ldcg(st.lev + i)] = 0;
    }
    // relax from Q_d: acc[v] |= fr[u] & ~seen[v], Q_{d+1} appended to the list
    {
      const int32_t n = e_d - b_d;
      const Enum en{st.lev + b_d, nullptr, n};
      const UMsBfs f{st.seen, bc_fr(st, d), st.acc, st.qstamp, d + 1};
      const HubList hub{st.hub_list, st.ctr + 21 + d % 3, st.hub_cap, kHubWidths * (int32_t)blockDim.x,
                        st.hub_slices};
      DOut out{};
      out.mode = OUT_SPARSE;
      out.q = st.lev;
      out.cnt = st.ctr + 0;
      out.cap = st.levcap;
      out.err = st.err;
      out.stage = &stage;
      lb_twce_all(g, en, n, f, out, blockIdx.x, gridDim.x, *reinterpret_cast<TwceSmem *>(smem), hub);
      stage_flush(out);
      const auto fetch = [&] {
        words.end = *(volatile int32_t *)out.cnt;
        words.chunks = *(volatile int32_t *)hub.cnt;
      };
      alive = grid_barrier_then(st.bar, gridDim.x, st.err, st.timeout_ns, fetch);
      if (alive && words.chunks > 0) {  // the hubs the level set aside, by all CTAs
        lb_hubs(g, hub, words.chunks, f, out, blockIdx.x, gridDim.x);
        stage_flush(out);
        alive = grid_barrier_then(st.bar, gridDim.x, st.err, st.timeout_ns, fetch);
      }
    }
    if (!alive) break;
    // publish Q_{d+1}: masks, depths, and its sigma work items
    {
      e_next = min(words.end, st.levcap);
      const int32_t m = e_next - e_d;
      const int32_t m_up = (m + 31) & ~31;
      uint64_t *nm = bc_fr(st, d + 1);
      for (int32_t i = tid; i < m_up; i += nthreads) {
        int32_t v = -1, deg = -1;
        if (i < m) {
          v = __ldcg(st.lev + e_d + i);
          const uint64_t a = __ldcg(st.acc + v);
          const uint64_t sv = __ldcg(st.seen + v);
          const uint64_t nb = a & ~sv;
          st.seen[v] = sv | nb;
          nm[v] = nb;
          st.acc[v] = 0;
          uint16_t *drow = st.depth + (int64_t)v * kBcWidth;
          for (uint64_t b = nb; b; b &= b - 1) drow[__ffsll((long long)b) - 1] = (uint16_t)(d + 1);
          deg = bc_degree(st, v);
        }
        bc_push_items(st, st.ctr + 1 + (d & 1), st.ctr + 24 + (d & 1), v, deg);
      }
    }
    clk.tick(st.stop, d, st.err);
    if (!grid_barrier_then(st.bar, gridDim.x, st.err, st.timeout_ns, [&] {
          words.items(bc_forward_items(st, d));
          words.stop = *(volatile int32_t *)st.stop;
        })) {
      alive = false;
      break;
    }
    b_prev = b_d;
    b_d = e_d;
  }
  const int32_t L = d;  // levels 0 .. L-1 are non-empty
  if (tid == 0) st.stats[0] = L;
  // ------------------------------------------------------------ backward
  // (iterations numbered on from the forward loop's, for the loop clock)
  for (int32_t dd = L - 1, it = L + 1; alive && dd >= 0; --dd, ++it) {
    if (stop_reached(words.stop, it)) break;
    if (tid == 0) {
      st.ctr[3 + ((dd + 1) & 1)] = st.ctr[26 + ((dd + 1) & 1)] = 0;   // consumed by the gather of level dd + 1
      st.ctr[18 + ((dd + 1) & 1)] = st.ctr[30 + ((dd + 1) & 1)] = 0;  // that gather's hand-out
    }
    // sources at level dd + 1 become "deeper" for the gathers from here on
    if (dd + 1 < L) {
      uint64_t *lmo = bc_lm(st, dd + 1);
      const int32_t e = __ldcg(st.loff + dd + 2);
      for (int32_t i = __ldcg(st.loff + dd + 1) + tid; i < e; i += nthreads) {
        const int32_t v = __ldcg(st.lev + i);
        st.rmask[v] = __ldcg(st.rmask + v) | __ldcg(lmo + v);
        lmo[v] = 0;
      }
    }
    // scan Q_dd: which sources sit at level dd at v, and the work items
    {
      const int32_t b = __ldcg(st.loff + dd), m = __ldcg(st.loff + dd + 1) - b;
      const int32_t m_up = (m + 31) & ~31;
      uint64_t *lmn = bc_lm(st, dd);
      for (int32_t i = tid; i < m_up; i += nthreads) {
        int32_t v = -1, deg = -1;
        if (i < m) {
          v = __ldcg(st.lev + b + i);
          const uint4 *row = reinterpret_cast<const uint4 *>(st.depth + (int64_t)v * kBcWidth);
          uint64_t mk = 0;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint4 q = __ldcg(row + j);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              if ((w[h] & 0xffffu) == (uint32_t)dd) mk |= 1ull << (8 * j + 2 * h);
              if ((w[h] >> 16) == (uint32_t)dd) mk |= 1ull << (8 * j + 2 * h + 1);
            }
          }
          lmn[v] = mk;
          deg = bc_degree(st, v);
        }
        bc_push_items(st, st.ctr + 3 + (dd & 1), st.ctr + 26 + (dd & 1), v, deg);
      }
    }
    if (!grid_barrier_then(st.bar, gridDim.x, st.err, st.timeout_ns, [&] { words.items(bc_backward_items(st, dd)); }))
      break;
    // gather: dep'[v][s] = 1/sigma[v][s] + sum over deeper in-neighbours
    {
      const uint64_t *lmn = bc_lm(st, dd);
      bc_each_item(st, bc_backward_items(st, dd), words, nwarps,
                   [&](int32_t v, int32_t c, int32_t k0, int32_t k1, bool single) {
        const uint64_t own = __ldcg(lmn + v);
        double a0, a1;
        bc_gather(st, k0, k1, own, st.rmask, st.dep, a0, a1);
        const double *srow = st.sigma + (int64_t)v * kBcWidth;
        double *row = st.dep + (int64_t)v * kBcWidth;
        if ((own >> lane) & 1) {
          const double t = a0 + (c == 0 ? 1.0 / __ldcg(srow + lane) : 0.0);
          if (single) row[lane] = t;
          else atomicAdd(row + lane, t);
        }
        if ((own >> (lane + 32)) & 1) {
          const double t = a1 + (c == 0 ? 1.0 / __ldcg(srow + lane + 32) : 0.0);
          if (single) row[lane + 32] = t;
          else atomicAdd(row + lane + 32, t);
        }
      });
    }
    clk.tick(st.stop, it, st.err);
    if (!grid_barrier_then(st.bar, gridDim.x, st.err, st.timeout_ns,
                           [&] { words.stop = *(volatile int32_t *)st.stop; }))
      break;
  }
}

// Seeds the sources, a thread of one 64-thread block per source (one thread
// walking them took 88 us); sources on the same vertex share its list entry.
__global__ void __launch_bounds__(kBcWidth) k_bcb_seed(BcState st, const int32_t *__restrict__ srcs) {
  __shared__ int32_t sv[kBcWidth];
  __shared__ uint32_t firsts[2];
  const int32_t s = threadIdx.x;
  if (blockIdx.x != 0) return;
  const int32_t v = s >= st.nsrc ? -1 : (st.perm ? st.perm[srcs[s]] : srcs[s]);
  sv[s] = v;
  __syncthreads();
  uint64_t same = 0;  // sources on this vertex
  for (int32_t i = 0; i < st.nsrc; ++i)
    if (sv[i] == v) same |= 1ull << i;
  const bool first = v >= 0 && __ffsll((long long)same) - 1 == s;
  const uint32_t ballot = __ballot_sync(0xffffffffu, first);
  if ((s & 31) == 0) firsts[s >> 5] = ballot;
  __syncthreads();
  if (first) {
    st.lev[__popc(ballot & ((1u << (s & 31)) - 1)) + (s >= 32 ? __popc(firsts[0]) : 0)] = v;
    st.seen[v] = same;
    st.fr[0][v] = same;
  }
  if (v >= 0) {
    st.depth[(int64_t)v * kBcWidth + s] = 0;
    st.sigma[(int64_t)v * kBcWidth + s] = 1.0;
  }
  if (s == 0) {
    st.ctr[0] = __popc(firsts[0]) + __popc(firsts[1]);
    st.ctr[20] = st.ctr[0];  // Q_0's end, read by every CTA before any appends to ctr[0]
    *st.stop = 0;
  }
}

// delta[s][v] = (dep'[p][s] - 1/sigma[p][s]) * sigma[p][s] as fp32 rows (v an
// original id, p its walked id), via a shared-memory transpose of 32-vertex
// tiles; also sums E_r over the sources (out-degree times the number of sources
// that reached v).
__global__ void __launch_bounds__(256) k_bcb_out(BcState st, const int32_t *__restrict__ off, float *out,
                                                 int64_t out_stride, unsigned long long *reached) {
  __shared__ float tile[kBcWidth][33];
  const int32_t V = st.V;
  unsigned long long er = 0;
  for (int32_t v0 = blockIdx.x * 32; v0 < V; v0 += gridDim.x * 32) {
    for (int32_t i = threadIdx.x; i < 32 * kBcWidth; i += blockDim.x) {
      const int32_t j = i / kBcWidth, s = i % kBcWidth;
      const int32_t v = v0 + j;
      float r = 0.f;
      if (v < V) {
        const int64_t pv = st.perm ? st.perm[v] : v;
        const double sg = st.sigma[pv * kBcWidth + s];
        if (sg != 0.0) r = (float)((st.dep[pv * kBcWidth + s] - 1.0 / sg) * sg);
      }
      tile[s][j] = r;
    }
    if (threadIdx.x < 32 && v0 + (int32_t)threadIdx.x < V) {
      const int32_t v = v0 + threadIdx.x;
      const int32_t pv = st.perm ? st.perm[v] : v;
      er += (unsigned long long)__popcll(st.seen[pv]) * (unsigned long long)(off[v + 1] - off[v]);
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < 32 * st.nsrc; i += blockDim.x) {
      const int32_t s = i / 32, j = i % 32;
      if (v0 + j < V) out[(int64_t)s * out_stride + v0 + j] = tile[s][j];
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) er += __shfl_xor_sync(0xffffffffu, er, d);
    if (threadIdx.x == 0 && er) atomicAdd(reached, er);
  }
}

// ------------------------------------------------------------------ host
BcBuffers::~BcBuffers() {
  if (owned)
    for (void *p : {(void *)masks, (void *)ints, (void *)work, (void *)depth, (void *)vals, (void *)dsrc})
      if (p) cudaFree(p);
}

static int64_t bc_levcap(int32_t V) { return (int64_t)V * kBcWidth; }
static int64_t bc_wcap(const gg_graph *g) { return (int64_t)g->csr.V + g->csr.E / kMinChunk + 64; }
static size_t bc_int_words(int32_t V) {  // qstamp, level list, level starts, counters
  return (size_t)V + (size_t)bc_levcap(V) + (kBcMaxLevels + 2) + 32;
}

gg_status bcb_buffers(gg_graph *g, bool owned, BcBuffers *b) {
  const int32_t V = g->csr.V;
  if (bc_levcap(V) >= INT32_MAX || bc_wcap(g) >= INT32_MAX)
    return set_error(GG_ERR_UNSUPPORTED, "batched BC holds 64 level-list entries per vertex in int32: "
                                         "V = %d is too large (use gg_bc)", V);
  GG_TRY(ensure_transpose(g));
  GG_TRY(ensure_hubs(g));
  // walk the degree-ordered copy: the rows of the most-gathered vertices share L2
  GG_TRY(ensure_relabel(g));
  if (!g->symmetric) GG_TRY(ensure_relabel_csc(g));  // its in-lists (a symmetric copy serves both)
  b->owned = owned;
  const size_t sz[6] = {sizeof(uint64_t) * 8 * (size_t)V, sizeof(int32_t) * bc_int_words(V),
                        sizeof(int64_t) * (size_t)bc_wcap(g), sizeof(uint16_t) * kBcWidth * (size_t)V,
                        sizeof(double) * 2 * kBcWidth * (size_t)V, sizeof(int32_t) * kBcWidth + 16};
  void **ptr[6] = {(void **)&b->masks, (void **)&b->ints, (void **)&b->work,
                   (void **)&b->depth, (void **)&b->vals, (void **)&b->dsrc};
  for (int i = 0; i < 6; ++i) {
    if (owned)
      GG_CUDA(cudaMalloc(ptr[i], sz[i]));
    else
      GG_TRY(scratch_get_app(g, i, sz[i], ptr[i]));
  }
  b->bytes_masks = sz[0];
  b->bytes_ints = sz[1];
  b->bytes_depth = sz[3];
  b->bytes_vals = sz[4];
  return GG_OK;
}

static BcState bcb_state(gg_graph *g, const BcBuffers &b, int32_t k) {
  const int32_t V = g->csr.V;
  const bool rel = g->rel && (g->symmetric || g->rel->csc.off);
  const GraphStore &t = rel ? (g->symmetric ? g->rel->g : g->rel->csc) : (g->csc ? *g->csc : g->csr);
  BcState S{};
  S.perm = rel ? g->rel->perm : nullptr;
  S.seen = b.masks;
  S.acc = b.masks + V;
  S.rmask = b.masks + 2 * (size_t)V;
  for (int i = 0; i < 3; ++i) S.fr[i] = b.masks + (3 + i) * (size_t)V;
  for (int i = 0; i < 2; ++i) S.lm[i] = b.masks + (6 + i) * (size_t)V;
  S.qstamp = b.ints;
  S.lev = b.ints + V;
  S.levcap = (int32_t)bc_levcap(V);
  S.loff = S.lev + S.levcap;
  S.ctr = S.loff + kBcMaxLevels + 2;
  S.hub_list = static_cast<int32_t *>(g->hubs.p);
  S.hub_cap = hub_capacity(g);
  S.hub_slices = slice_limit(g->max_degree);
  S.stats = S.ctr + 8;
  S.stop = S.ctr + 12;
  S.work = b.work;
  S.wcap = (int32_t)bc_wcap(g);
  S.chunk = effective_tuning(g, GG_BATCH_BC, 1).chunk;
  S.light = std::min(kBcLight, S.chunk);
  S.depth = b.depth;
  S.sigma = b.vals;
  S.dep = b.vals + (size_t)kBcWidth * V;
  S.toff = t.off;
  S.tsrc = t.dst;
  S.V = V;
  S.nsrc = k;
  S.bar = g->d_bar;
  S.err = g->d_err;
  S.timeout_ns = barrier_timeout_ns();
  S.loop_limit_ns = loop_timeout_ns();
  return S;
}

const void *bcb_kernel() { return (const void *)k_bc_batch; }

// One pass of k <= 64 sources, stream-ordered (capturable into a CUDA graph):
// reset, seed, the persistent forward + backward kernel, then the fp32 rows
// out[s * out_stride + v] and the reached-edge count (added to *reached).
gg_status bcb_enqueue(gg_graph *g, cudaStream_t st, const BcBuffers &b, int32_t k, const int32_t *dsrc,
                      float *out, int64_t out_stride, unsigned long long *reached, int32_t *stats,
                      bool timed) {
  const BcState S0 = bcb_state(g, b, k);
  BcState S = S0;
  if (stats) S.stats = stats;
  int per_sm = 0;
  const int cta = 512;
  const size_t smem = twce_smem_bytes(cta);
  GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bc_batch, cta, smem));
  if (per_sm < 1) return set_error(GG_ERR_UNSUPPORTED, "batched BC kernel does not fit an SM");
  GG_CUDA(cudaMemsetAsync(b.masks, 0, b.bytes_masks, st));
  GG_CUDA(cudaMemsetAsync(b.ints, 0, sizeof(int32_t) * (size_t)g->csr.V, st));            // qstamp
  GG_CUDA(cudaMemsetAsync(S.ctr, 0, sizeof(int32_t) * 32, st));                            // counters
  GG_CUDA(cudaMemsetAsync(b.depth, 0xff, b.bytes_depth, st));
  GG_CUDA(cudaMemsetAsync(b.vals, 0, b.bytes_vals, st));
  note_launch();
  k_bcb_seed<<<1, kBcWidth, 0, st>>>(S, dsrc);
  GG_CUDA(cudaMemsetAsync(S.bar, 0, sizeof(uint32_t) * 2, st));
  DGraph dg = (S0.perm != nullptr) ? g->rel->g.view() : g->csr.view();
  dg.nbuckets = 0;
  void *args[] = {&dg, &S};
  if (timed) GG_CUDA(cudaEventRecord(g->ev2, st));
  note_launch();
  const int bps = effective_tuning(g, GG_BATCH_BC, per_sm).blocks_per_sm;
  GG_CUDA(cudaLaunchCooperativeKernel((const void *)k_bc_batch, bps * g->sm_count, cta, args, smem, st));
  if (timed) GG_CUDA(cudaEventRecord(g->ev3, st));
  note_launch();
  k_bcb_out<<<g->sm_count * 8, 256, 0, st>>>(S, g->csr.off, out, out_stride, reached);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg

using namespace gg;

// Batched BC: dep_out[s*V + v] (fp32) for nsrc sources (host or device memory).
extern "C" gg_status gg_bc_batch(gg_graph *g, const int32_t *sources, int32_t nsrc, float *dep_out,
                                 gg_stats *stats) {
  GG_CHECK_ARG(g && sources && nsrc > 0 && dep_out, "bad arguments");
  const int32_t V = g->csr.V;
  for (int32_t i = 0; i < nsrc; ++i)
    GG_CHECK_ARG(sources[i] >= 0 && sources[i] < V, "source out of range");
  if (stats) *stats = gg_stats{};
  cudaStream_t st = g->stream;
  BcBuffers b;
  GG_TRY(bcb_buffers(g, false, &b));
  float *rows = nullptr;
  const bool direct = rows_on_device(g, dep_out);
  if (!direct) GG_TRY(scratch_get_app(g, 6, sizeof(float) * (size_t)std::min(nsrc, kBcWidth) * V, (void **)&rows));
  unsigned long long *reached = reinterpret_cast<unsigned long long *>(b.dsrc + kBcWidth);
  const uint64_t l0 = launches();
  GG_CUDA(cudaMemsetAsync(reached, 0, sizeof(unsigned long long), st));
  cudaEventRecord(g->ev0, st);
  float loop_ms = 0;
  int32_t levels = 0;
  for (int32_t base = 0; base < nsrc; base += kBcWidth) {
    const int32_t k = std::min(kBcWidth, nsrc - base);
    GG_CUDA(cudaMemcpyAsync(b.dsrc, sources + base, sizeof(int32_t) * k, cudaMemcpyDefault, st));
    float *out = direct ? dep_out + (size_t)base * V : rows;
    GG_TRY(bcb_enqueue(g, st, b, k, b.dsrc, out, V, reached, nullptr, true));
    if (!direct)
      GG_CUDA(cudaMemcpyAsync(dep_out + (size_t)base * V, out, sizeof(float) * (size_t)k * V, cudaMemcpyDefault, st));
    const BcState S = bcb_state(g, b, k);
    GG_CUDA(cudaMemcpyAsync(g->h_pinned + 30, S.stats, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    GG_CUDA(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, g->ev2, g->ev3);
    loop_ms += ms;
    levels = std::max(levels, g->h_pinned[30]);
  }
  cudaEventRecord(g->ev1, st);
  GG_CUDA(cudaEventSynchronize(g->ev1));
  GG_TRY(check_device_error(g, "bc_batch"));
  if (stats) {
    unsigned long long er = 0;
    GG_CUDA(cudaMemcpy(&er, reached, sizeof(er), cudaMemcpyDeviceToHost));
    cudaEventElapsedTime(&stats->device_ms, g->ev0, g->ev1);
    stats->loop_ms = loop_ms;
    stats->iterations = levels;
    stats->edges_traversed = 2 * (int64_t)er;  // forward + backward sweeps, as gg_bc
    stats->fused = 1;
    stats->launches = (int32_t)(launches() - l0);
  }
  return GG_OK;
}
