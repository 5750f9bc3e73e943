// Batched BFS: up to 64 sources per pass in one persistent kernel.
//
// Bit-parallel multi-source BFS: every vertex carries 64-bit masks -- `seen`
// (sources that reached it), `acc` (sources reaching it this level) and the
// level masks fr (sources for which it is on the level's frontier).  Levels run
// top-down or bottom-up (direction optimisation, as bfs.cpp's hybrid schedule
// does for one source, here for all sources at once):
//  * top-down: one traversal of an edge (u, v) serves every source,
//    acc[v] |= fr[u] & ~seen[v]; frontier vertices are load-balanced by the TWCE
//    device function of lb.cuh; a publish phase then turns new bits into the
//    next level's masks and depths;
//  * bottom-up (frontier larger than V / bu_div): groups of 8 lanes take the
//    vertices some still-expanding source has not reached and OR the level
//    masks of their in-neighbours, 32 at a time, stopping as soon as every such
//    source is found, a CTA the long lists; no atomics in global memory.
// Level masks rotate through three arrays and queues through three buffers:
// the masks of level L-1 are cleared (from its queue) while level L publishes,
// so a bottom-up scan never reads a stale mask.
//
// The result for each source equals an independent BFS (apps/bfs.cpp), because
// a source's bit enters seen[v] exactly at the first level that reaches v.
#include <vector>

#include "batch.h"
#include "lb.cuh"
#include "selector.h"

namespace gg {

__device__ __forceinline__ uint64_t *ms_fr(const MsBfsState &st, int32_t level) {
  const int32_t i = level % 3;
  return i == 0 ? st.fr[0] : (i == 1 ? st.fr[1] : st.fr[2]);
}
__device__ __forceinline__ int32_t *ms_q(const MsBfsState &st, int32_t level) {
  const int32_t i = level % 3;
  return i == 0 ? st.q[0] : (i == 1 ? st.q[1] : st.q[2]);
}

// depth[s][v] = level for every bit s of nb, the bits split over `ways` lanes.
__device__ __forceinline__ void ms_depths(const MsBfsState &st, int32_t v, uint64_t nb, int32_t level,
                                          int32_t sub, int32_t ways) {
  if (!st.depth) return;
  for (uint64_t b = nb; b; b &= b - 1) {
    const int32_t s = __ffsll((long long)b) - 1;
    if (s % ways == sub) st.depth[(int64_t)s * st.depth_stride + v] = level;
  }
}

// A thread's share of what a level adds to the next one's frontier: the sources
// found and the out-degree statistics.  Kept in registers and folded into the
// CTA's at the end of the level -- 64-bit shared-memory atomics per vertex (CAS
// loops, all on the same words) serialised a CTA that found thousands.
struct MsAcc {
  unsigned long long act, sum, sq, mx;
  __device__ __forceinline__ void note(const MsBfsState &st, int32_t v, uint64_t nb) {
    const unsigned long long d = (unsigned long long)(__ldg(st.off + v + 1) - __ldg(st.off + v));
    act |= nb;
    sum += d;
    sq += d * d;
    mx = mx > d ? mx : d;
  }
};
__device__ __forceinline__ void ms_fold(const MsAcc &t, unsigned long long *s_act, unsigned long long *s_stat) {
  if (!__any_sync(0xffffffffu, t.act != 0ull)) return;
  unsigned long long act = t.act, sum = t.sum, sq = t.sq, mx = t.mx;
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) {
    act |= __shfl_xor_sync(0xffffffffu, act, i);
    sum += __shfl_xor_sync(0xffffffffu, sum, i);
    sq += __shfl_xor_sync(0xffffffffu, sq, i);
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, mx, i);
    mx = mx > o ? mx : o;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicOr(s_act, act);
    atomicAdd(s_stat, sum);
    atomicAdd(s_stat + 1, sq);
    atomicMax(s_stat + 2, mx);
  }
}

// A bottom-up level: every vertex that some still-expanding source wants ORs the
// level masks of its in-neighbours and stops when each such source is found.  A
// lane per vertex reads the masks (coalesced) and drops vertices nobody wants or
// without in-edges; 8-lane groups walk the lists, 32 in-neighbours in flight each,
// four vertices of a warp at a time; lists longer than kMsLong are set aside for
// the whole CTA.  With a group per vertex and 8 in flight, a hub that one source
// does not reach was walked alone for 2.4 ms, whatever the level held (1 M
// vertices; a level that chose bottom-up with such a hub in it: 3.2 ms of 4.9).
// Lengths of 256 / 512 / 2,048: symmetrized R-MAT 20 1.03 / 0.92 / 0.99 ms, 22 3.76 / 3.13 /
// 3.06, directed 20 0.81 / 0.81 / 0.84; 64 lists a CTA instead of 256: 22 4.85.
constexpr int32_t kMsLong = 512;
constexpr int32_t kMsLongMax = 256;  // set aside per CTA; more are walked by groups
struct MsLong {
  int32_t n;
  uint32_t found[2];
  int32_t v[kMsLongMax];
};
__device__ __forceinline__ uint64_t ms_shfl(uint64_t x, int32_t l) {
  return __shfl_sync(0xffffffffu, (unsigned long long)x, l & 31);
}
__device__ __forceinline__ void ms_bottom_up(const MsBfsState &st, int32_t L, const uint64_t *frc, uint64_t *frn,
                                             const DOut &out, MsAcc &acc, MsLong &lg) {
  const int32_t lane = threadIdx.x & 31, sub = lane & 7, gi = lane >> 3;
  const uint32_t gmask = 0xFFu << (gi * 8);
  const uint64_t act = *(volatile unsigned long long *)(st.actm + L % 3);
  if (threadIdx.x == 0) {
    lg.n = 0;
    lg.found[0] = lg.found[1] = 0u;
  }
  __syncthreads();
  int32_t since = 0;  // vertices the CTA can have staged since there was room
  for (int64_t first = (int64_t)blockIdx.x * blockDim.x; first < st.V; first += (int64_t)gridDim.x * blockDim.x) {
    if (since + (int32_t)blockDim.x > kStageCap / 2) {
      __syncthreads();
      stage_make_room(out, kStageCap / 2 + (int32_t)blockDim.x);
      __syncthreads();
      since = 0;
    }
    since += (int32_t)blockDim.x;
    const int64_t v64 = first + threadIdx.x;
    const int32_t v = (int32_t)v64;
    uint64_t sv = 0, want = 0, found = 0;
    int32_t kb = 0, ke = 0;
    if (v64 < st.V) {
      sv = __ldcg(st.seen + v);
      want = act & ~sv;
      if (want) {
        kb = __ldg(st.toff + v);
        ke = __ldg(st.toff + v + 1);
      }
    }
    bool mine_here = want != 0 && ke > kb;
    if (mine_here && ke - kb > kMsLong) {
      const int32_t at = agg_inc(&lg.n);
      if (at < kMsLongMax) {
        lg.v[at] = v;
        mine_here = false;
      }
    }
    __syncwarp();
    uint32_t open = __ballot_sync(0xffffffffu, mine_here);
    while (open) {
      int32_t l[4];  // the next four vertices, a group each (-1: none)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        l[j] = __ffs(open) - 1;
        open &= open - 1;
      }
      const int32_t mine = gi == 0 ? l[0] : (gi == 1 ? l[1] : (gi == 2 ? l[2] : l[3]));
      const uint64_t w = ms_shfl(want, mine);
      const int32_t b = __shfl_sync(0xffffffffu, kb, mine & 31), e = __shfl_sync(0xffffffffu, ke, mine & 31);
      uint64_t f = 0;
      if (mine >= 0)
        for (int32_t k0 = b; k0 < e; k0 += 32) {
          int32_t u[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) u[j] = k0 + 8 * j + sub < e ? __ldg(st.tsrc + k0 + 8 * j + sub) : -1;
          uint64_t m = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (u[j] >= 0) m |= __ldcg(frc + u[j]);
          m &= w;
          m |= __shfl_xor_sync(gmask, (unsigned long long)m, 1);
          m |= __shfl_xor_sync(gmask, (unsigned long long)m, 2);
          m |= __shfl_xor_sync(gmask, (unsigned long long)m, 4);
          f |= m;
          if (f == w) break;
        }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t h = ms_shfl(f, j * 8);
        if (lane == l[j]) found = h;
      }
    }
    if (found) {
      st.seen[v] = sv | found;
      frn[v] = found;
      out.sparse(v);
      acc.note(st, v, found);
    }
    if (!st.depth) continue;
    // the warp's rows of one source are consecutive words: a store per source
    uint32_t any[2] = {__reduce_or_sync(0xffffffffu, (uint32_t)found),
                       __reduce_or_sync(0xffffffffu, (uint32_t)(found >> 32))};
#pragma unroll
    for (int h = 0; h < 2; ++h)
      for (uint32_t bits = any[h]; bits; bits &= bits - 1) {
        const int32_t s = 32 * h + __ffs(bits) - 1;
        if ((found >> s) & 1) st.depth[(int64_t)s * st.depth_stride + v] = L + 1;
      }
  }
  __syncthreads();
  const int32_t nl = min(lg.n, kMsLongMax);
  for (int32_t i = 0; i < nl; ++i) {
    const int32_t v = lg.v[i];
    const uint64_t sv = __ldcg(st.seen + v), want = act & ~sv;
    const int32_t kb = __ldg(st.toff + v), ke = __ldg(st.toff + v + 1), T = blockDim.x;
    uint64_t found = 0;
    for (int32_t k0 = kb; k0 < ke; k0 += 4 * T) {
      int32_t u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t k = (int64_t)k0 + j * T + threadIdx.x;
        u[j] = k < ke ? __ldg(st.tsrc + k) : -1;
      }
      uint64_t m = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (u[j] >= 0) m |= __ldcg(frc + u[j]);
      m &= want;
      const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)m), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(m >> 32));
      if (lane == 0 && lo) atomicOr(&lg.found[0], lo);
      if (lane == 0 && hi) atomicOr(&lg.found[1], hi);
      __syncthreads();
      found = (uint64_t)lg.found[1] << 32 | lg.found[0];
      __syncthreads();
      if (found == want || (int64_t)k0 + 4 * T >= ke) break;
    }
    if (threadIdx.x == 0) {
      lg.found[0] = lg.found[1] = 0u;
      if (found) {
        st.seen[v] = sv | found;
        frn[v] = found;
        out.sparse(v);
        acc.note(st, v, found);
      }
    }
    if (st.depth && threadIdx.x < kMsBfsWidth && ((found >> threadIdx.x) & 1))
      st.depth[(int64_t)threadIdx.x * st.depth_stride + v] = L + 1;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512, 3) k_msbfs(DGraph g, MsBfsState st) {
  extern __shared__ int4 smem[];
  __shared__ unsigned long long s_act;
  __shared__ unsigned long long s_stat[3];
  __shared__ MsLong long_;
  __shared__ StageMem stage_mem;
  Stage &stage = stage_mem.s;
  if (threadIdx.x == 0) stage.init(kStageCap);  // the first level's barrier comes before any append
  const int32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t nthreads = gridDim.x * blockDim.x;
  const int32_t lane = threadIdx.x & 31;
  LoopClock clk;
  clk.start(st.loop_limit_ns);
  int32_t L = 0, bu_levels = 0;
  double vis_v = 0, vis_e = 0;  // running totals of the frontiers so far (the same in every CTA)
  for (;; ++L) {
    const int32_t n = *(volatile int32_t *)(st.cnt4 + (L & 3));
    if (n == 0 || stopped(st.stop, L)) break;
    const volatile unsigned long long *ls = st.lstat + 4 * (L % 3);
    const double sd = (double)ls[0], sd2 = (double)ls[1], mx = (double)ls[2];
    if (tid == 0) {
      st.cnt4[(L + 2) & 3] = 0;
      st.actm[(L + 2) % 3] = 0ull;
      st.hub3[(L + 1) % 3] = 0;
      for (int i = 0; i < 4; ++i) st.lstat[4 * ((L + 2) % 3) + i] = 0ull;
    }
    if (threadIdx.x == 0) {
      s_act = 0ull;
      s_stat[0] = s_stat[1] = s_stat[2] = 0ull;
    }
    // direction of this level: forced, the network's, or the bu_div rule
    bool bu;
    if (st.force_dir >= 0) {
      bu = st.force_dir == 1;
    } else if (st.sel || st.feat_log) {
      float *x = reinterpret_cast<float *>(smem);  // scratch until the level's TWCE bins
      if (threadIdx.x == 0)
        selector_features(x, (double)n, sd, sd2, mx, vis_v, vis_e, L, (double)st.V, (double)st.E);
      __syncthreads();
      bu = st.sel ? selector_pull(st.sel, x, x + 16) : (st.bu_div > 0 && (int64_t)n * st.bu_div > st.V);
    } else {
      bu = st.bu_div > 0 && (int64_t)n * st.bu_div > st.V;
    }
    if (st.feat_log && L <= st.max_log && blockIdx.x == 0 && threadIdx.x == 0) {
      const float *x = reinterpret_cast<const float *>(smem);
      if (!(st.force_dir >= 0) && L < st.max_log)
        for (int i = 0; i < kSelectorFeatures; ++i) st.feat_log[L * kSelectorFeatures + i] = x[i];
      st.time_log[L] = globaltimer_ns();  // the end of level L-1 (max_log + 1 entries)
    }
    if (st.force_dir >= 0 && st.feat_log && L < st.max_log && blockIdx.x == 0 && threadIdx.x == 0) {
      float x[kSelectorFeatures];
      selector_features(x, (double)n, sd, sd2, mx, vis_v, vis_e, L, (double)st.V, (double)st.E);
      for (int i = 0; i < kSelectorFeatures; ++i) st.feat_log[L * kSelectorFeatures + i] = x[i];
    }
    vis_v = fmin((double)st.V, vis_v + n);
    vis_e = fmin((double)st.E, vis_e + sd);
    __syncthreads();
    const uint64_t *frc = ms_fr(st, L);
    uint64_t *frn = ms_fr(st, L + 1);
    int32_t *qn = ms_q(st, L + 1);
    // top-down: acc[v] |= fr[u] & ~seen[v]; the first toucher queues v
    const UMsBfs f{st.seen, frc, st.acc, st.qstamp, L + 1};
    const HubList hub{st.hub_list, st.hub3 + L % 3, st.hub_cap, kHubWidths * (int32_t)blockDim.x,
                      st.hub_slices};
    DOut out{};
    out.mode = OUT_SPARSE;
    out.q = qn;
    out.cnt = st.cnt4 + ((L + 1) & 3);
    out.cap = st.V;  // qstamp admits each vertex once per level
    out.err = st.err;
    out.stage = &stage;
    MsAcc acc{0ull, 0ull, 0ull, 0ull};
    if (!bu) {
      const Enum en{ms_q(st, L), nullptr, n};
      lb_twce_all(g, en, n, f, out, blockIdx.x, gridDim.x, *reinterpret_cast<TwceSmem *>(smem), hub);
    } else {
      ++bu_levels;
      ms_bottom_up(st, L, frc, frn, out, acc, long_);
    }
    stage_flush(out);
    if (!grid_barrier(st.bar, gridDim.x, st.err, st.timeout_ns)) break;
    if (!bu) {  // the hubs the level set aside, by all CTAs
      const int32_t chunks = *(volatile int32_t *)hub.cnt;
      if (chunks > 0) {
        lb_hubs(g, hub, chunks, f, out, blockIdx.x, gridDim.x);
        stage_flush(out);
        if (!grid_barrier(st.bar, gridDim.x, st.err, st.timeout_ns)) break;
      }
    }
    // publish (top-down levels): new bits become the next level's masks
    if (!bu) {
      const int32_t m = min(*(volatile int32_t *)(st.cnt4 + ((L + 1) & 3)), st.V);
      for (int32_t i = tid; i < m; i += nthreads) {
        const int32_t v = __ldcg(qn + i);
        const uint64_t a = __ldcg(st.acc + v);
        const uint64_t sv = __ldcg(st.seen + v);
        const uint64_t nb = a & ~sv;
        st.seen[v] = sv | nb;
        frn[v] = nb;
        st.acc[v] = 0;
        acc.note(st, v, nb);
        ms_depths(st, v, nb, L + 1, 0, 1);
      }
    }
    // the masks of level L-1 are dead: clear them for the bottom-up scans
    if (L >= 1) {
      uint64_t *old = ms_fr(st, L - 1);
      const int32_t *qo = ms_q(st, L - 1);
      const int32_t m = min(*(volatile int32_t *)(st.cnt4 + ((L - 1) & 3)), st.V);
      for (int32_t i = tid; i < m; i += nthreads) old[__ldcg(qo + i)] = 0ull;
    }
    ms_fold(acc, &s_act, s_stat);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (s_act) atomicOr(st.actm + (L + 1) % 3, s_act);
      unsigned long long *nx = st.lstat + 4 * ((L + 1) % 3);  // statistics of the next frontier
      if (s_stat[0]) {
        atomicAdd(nx, s_stat[0]);
        atomicAdd(nx + 1, s_stat[1]);
        atomicMax(nx + 2, s_stat[2]);
      }
    }
    clk.tick(st.stop, L, st.err);
    if (!grid_barrier(st.bar, gridDim.x, st.err, st.timeout_ns)) break;
  }
  if (tid == 0) {
    st.stats[0] = L;
    st.stats[1] = bu_levels;
    if (st.time_log && L <= st.max_log) st.time_log[L] = globaltimer_ns();
  }
}

// Initial state: masks cleared, depth rows -1.
__global__ void k_msbfs_init(MsBfsState st) {
  const int64_t total = (int64_t)st.nsrc * st.depth_stride;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
    st.depth[i] = -1;
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < st.V; v += gridDim.x * blockDim.x) {
    st.seen[v] = 0;
    st.acc[v] = 0;
    st.fr[0][v] = 0;
    st.fr[1][v] = 0;
    st.fr[2][v] = 0;
    st.qstamp[v] = 0;
  }
}

// Control words and sources, a thread of one 64-thread block per source (one
// thread walking the sources took 91 us of dependent round trips); sources on
// the same vertex share its queue entry.
__global__ void __launch_bounds__(kMsBfsWidth) k_msbfs_seed(MsBfsState st, const int32_t *__restrict__ srcs) {
  __shared__ int32_t sv[kMsBfsWidth];
  __shared__ unsigned long long stat[3];
  const int32_t s = threadIdx.x;
  if (blockIdx.x != 0) return;
  const int32_t v = s < st.nsrc ? srcs[s] : -1;
  sv[s] = v;
  if (s < 3) stat[s] = 0ull;
  __syncthreads();
  uint64_t same = 0;  // sources on this vertex
  for (int32_t i = 0; i < st.nsrc; ++i)
    if (sv[i] == v) same |= 1ull << i;
  const bool first = v >= 0 && __ffsll((long long)same) - 1 == s;
  const uint32_t ballot = __ballot_sync(0xffffffffu, first);
  __shared__ uint32_t firsts[2];
  if ((s & 31) == 0) firsts[s >> 5] = ballot;
  __syncthreads();
  if (first) {
    const int32_t pos = __popc(ballot & ((1u << (s & 31)) - 1)) + (s >= 32 ? __popc(firsts[0]) : 0);
    st.q[0][pos] = v;
    st.seen[v] = same;
    st.fr[0][v] = same;
    const unsigned long long d = (unsigned long long)(st.off[v + 1] - st.off[v]);  // the sources' frontier
    atomicAdd(stat, d);
    atomicAdd(stat + 1, d * d);
    atomicMax(stat + 2, d);
  }
  if (v >= 0) st.depth[(int64_t)s * st.depth_stride + v] = 0;
  __syncthreads();
  if (s < 12) st.lstat[s] = s < 3 ? stat[s] : 0ull;
  if (s < 4) st.cnt4[s] = s == 0 ? __popc(firsts[0]) + __popc(firsts[1]) : 0;
  if (s < 3) {
    st.hub3[s] = 0;
    st.actm[s] = s == 0 ? (st.nsrc >= 64 ? ~0ull : (1ull << st.nsrc) - 1) : 0ull;
  }
  if (s == 0) *st.stop = 0;
}

// ------------------------------------------------------------------ host
MsBfsBuffers::~MsBfsBuffers() {
  if (owned)
    for (void *p : {(void *)masks, (void *)ints, (void *)dsrc})
      if (p) cudaFree(p);
}

gg_status msbfs_buffers(gg_graph *g, int32_t nsrc, bool owned, MsBfsBuffers *b) {
  GG_TRY(ensure_transpose(g));  // in-lists for the bottom-up levels
  GG_TRY(ensure_hubs(g));
  const int32_t V = g->csr.V;
  b->owned = owned;
  const size_t sz[3] = {sizeof(uint64_t) * (5 * (size_t)V + 24), sizeof(int32_t) * (4 * (size_t)V + 64),
                        sizeof(int32_t) * (size_t)std::max(nsrc, kMsBfsWidth)};
  void **ptr[3] = {(void **)&b->masks, (void **)&b->ints, (void **)&b->dsrc};
  for (int i = 0; i < 3; ++i) {
    if (owned)
      GG_CUDA(cudaMalloc(ptr[i], sz[i]));
    else
      GG_TRY(scratch_get_app(g, i, sz[i], ptr[i]));
  }
  return GG_OK;
}

MsBfsState msbfs_state(gg_graph *g, const MsBfsBuffers &b, int32_t k, int32_t *depth_rows) {
  const int32_t V = g->csr.V;
  const GraphStore &t = g->csc ? *g->csc : g->csr;
  MsBfsState S{};
  S.seen = b.masks;
  S.acc = b.masks + V;
  for (int i = 0; i < 3; ++i) S.fr[i] = b.masks + (2 + i) * (size_t)V;
  S.actm = reinterpret_cast<unsigned long long *>(b.masks + 5 * (size_t)V);
  S.lstat = reinterpret_cast<unsigned long long *>(b.masks + 5 * (size_t)V + 8);
  S.qstamp = b.ints;
  for (int i = 0; i < 3; ++i) S.q[i] = b.ints + (1 + i) * (size_t)V;
  int32_t *hdr = b.ints + 4 * (size_t)V;
  S.cnt4 = hdr;          // 4
  S.stats = hdr + 8;     // 2
  S.stop = hdr + 12;
  S.hub3 = hdr + 16;     // 3
  S.hub_list = static_cast<int32_t *>(g->hubs.p);
  S.hub_cap = hub_capacity(g);
  S.hub_slices = slice_limit(g->max_degree);
  S.toff = t.off;
  S.tsrc = t.dst;
  S.V = V;
  const gg_batch_tuning tn = effective_tuning(g, GG_BATCH_BFS, 1);
  S.bu_div = tn.bottom_up_div;
  S.loop_limit_ns = loop_timeout_ns();
  S.depth = depth_rows;
  S.depth_stride = V;
  S.nsrc = k;
  S.bar = g->d_bar;
  S.err = g->d_err;
  S.timeout_ns = barrier_timeout_ns();
  S.sel = g->batch_selector[GG_BATCH_BFS] ? selector_params(g->batch_selector[GG_BATCH_BFS]) : nullptr;
  S.force_dir = -1;
  S.off = g->csr.off;
  S.E = g->csr.E;
  return S;
}

bool rows_on_device(const gg_graph *g, const void *out) {
  cudaPointerAttributes pa{};
  if (cudaPointerGetAttributes(&pa, out) != cudaSuccess) {
    cudaGetLastError();  // not an address CUDA knows: the copy decides
    return false;
  }
  return pa.type == cudaMemoryTypeDevice && pa.device == g->device && reinterpret_cast<uintptr_t>(out) % 4 == 0;
}

const void *msbfs_kernel() { return (const void *)k_msbfs; }

// One pass of k <= 64 sources: reset, seed, the persistent loop writing the
// depth rows.  Stream-ordered only, so it can be captured into a CUDA graph.
gg_status msbfs_enqueue(gg_graph *g, cudaStream_t st, const MsBfsState &S, const int32_t *dsrc,
                        bool timed) {
  int per_sm = 0;
  const int cta = 512;
  const size_t smem = twce_smem_bytes(cta);
  GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_msbfs, cta, smem));
  if (per_sm < 1) return set_error(GG_ERR_UNSUPPORTED, "batched BFS kernel does not fit an SM");
  note_launch();
  k_msbfs_init<<<g->sm_count * 8, 256, 0, st>>>(S);
  note_launch();
  k_msbfs_seed<<<1, kMsBfsWidth, 0, st>>>(S, dsrc);
  GG_CUDA(cudaMemsetAsync(S.bar, 0, sizeof(uint32_t) * 2, st));
  DGraph dg = g->csr.view();
  dg.nbuckets = 0;
  MsBfsState arg = S;
  void *args[] = {&dg, &arg};
  if (timed) GG_CUDA(cudaEventRecord(g->ev2, st));
  note_launch();
  const int bps = effective_tuning(g, GG_BATCH_BFS, per_sm).blocks_per_sm;
  GG_CUDA(cudaLaunchCooperativeKernel((const void *)k_msbfs, bps * g->sm_count, cta, args, smem, st));
  if (timed) GG_CUDA(cudaEventRecord(g->ev3, st));
  return GG_OK;
}

}  // namespace gg

using namespace gg;

// Batched BFS: depth_out[s*V + v] for nsrc sources (host or device memory).
extern "C" gg_status gg_bfs_batch(gg_graph *g, const int32_t *sources, int32_t nsrc,
                                  int32_t *depth_out, gg_stats *stats) {
  GG_CHECK_ARG(g && sources && nsrc > 0 && depth_out, "bad arguments");
  const int32_t V = g->csr.V;
  for (int32_t i = 0; i < nsrc; ++i)
    GG_CHECK_ARG(sources[i] >= 0 && sources[i] < V, "source out of range");
  if (stats) *stats = gg_stats{};
  cudaStream_t st = g->stream;
  MsBfsBuffers b;
  GG_TRY(msbfs_buffers(g, nsrc, false, &b));
  int32_t *depth = nullptr;
  const bool direct = rows_on_device(g, depth_out);
  if (!direct)
    GG_TRY(scratch_get_app(g, 3, sizeof(int32_t) * (size_t)std::min(nsrc, kMsBfsWidth) * V, (void **)&depth));
  const uint64_t l0 = launches();
  cudaEventRecord(g->ev0, st);
  float loop_ms = 0;
  int32_t levels = 0;
  for (int32_t base = 0; base < nsrc; base += kMsBfsWidth) {
    const int32_t k = std::min(kMsBfsWidth, nsrc - base);
    const MsBfsState S = msbfs_state(g, b, k, direct ? depth_out + (size_t)base * V : depth);
    GG_CUDA(cudaMemcpyAsync(b.dsrc, sources + base, sizeof(int32_t) * k, cudaMemcpyDefault, st));
    GG_TRY(msbfs_enqueue(g, st, S, b.dsrc, true));
    if (!direct)
      GG_CUDA(cudaMemcpyAsync(depth_out + (size_t)base * V, depth, sizeof(int32_t) * (size_t)k * V,
                              cudaMemcpyDefault, st));
    GG_CUDA(cudaMemcpyAsync(g->h_pinned + 30, S.stats, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    GG_CUDA(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, g->ev2, g->ev3);
    loop_ms += ms;
    levels = std::max(levels, g->h_pinned[30]);
  }
  cudaEventRecord(g->ev1, st);
  GG_CUDA(cudaEventSynchronize(g->ev1));
  GG_TRY(check_device_error(g, "bfs_batch"));
  if (stats) {
    cudaEventElapsedTime(&stats->device_ms, g->ev0, g->ev1);
    stats->loop_ms = loop_ms;
    stats->iterations = levels;
    stats->fused = 1;
    stats->launches = (int32_t)(launches() - l0);
  }
  return GG_OK;
}

// Attaches a selector network to a graph's batched kernels (NULL detaches it).
extern "C" gg_status gg_batch_set_selector(gg_graph *g, int32_t app, const gg_selector *sel) {
  GG_CHECK_ARG(g, "graph is NULL");
  if (app != GG_BATCH_BFS)
    return set_error(GG_ERR_UNSUPPORTED, "only batched BFS takes a learned per-level choice");
  g->batch_selector[app] = sel;
  return GG_OK;
}

// Training data for the batched BFS direction: the first min(nsrc, 64) sources
// traversed with every level top-down, then with every level bottom-up (twice
// each; a level's masks after it are the same either way, so level l starts
// from the same state in every run).  feats[l][12]: the features of level l;
// times[l][2]: its best time in ms top-down and bottom-up.
extern "C" gg_status gg_batch_collect(gg_graph *g, int32_t app, const int32_t *sources, int32_t nsrc,
                                      int32_t max_rows, float *feats, float *times, int32_t *nrows) {
  GG_CHECK_ARG(g && sources && nsrc > 0 && feats && times && nrows && max_rows > 0, "bad arguments");
  if (app != GG_BATCH_BFS) return set_error(GG_ERR_UNSUPPORTED, "timings are collected for batched BFS");
  const int32_t V = g->csr.V;
  for (int32_t i = 0; i < nsrc; ++i) GG_CHECK_ARG(sources[i] >= 0 && sources[i] < V, "source out of range");
  *nrows = 0;
  cudaStream_t st = g->stream;
  const int32_t k = std::min(nsrc, kMsBfsWidth);
  MsBfsBuffers b;
  GG_TRY(msbfs_buffers(g, k, false, &b));
  int32_t *depth = nullptr;
  GG_TRY(scratch_get_app(g, 3, sizeof(int32_t) * (size_t)k * V, (void **)&depth));
  float *dfeat = nullptr;
  unsigned long long *dtime = nullptr;
  GG_CUDA(dev_alloc(&dfeat, sizeof(float) * kSelectorFeatures * (size_t)max_rows, st));
  GG_CUDA(dev_alloc(&dtime, sizeof(unsigned long long) * ((size_t)max_rows + 1), st));
  std::vector<float> best(2 * (size_t)max_rows, INFINITY);
  std::vector<unsigned long long> ht((size_t)max_rows + 1);
  int32_t levels = -1;
  gg_status status = GG_OK;
  for (int rep = 0; rep < 4 && status == GG_OK; ++rep) {
    const int dir = rep & 1;
    MsBfsState S = msbfs_state(g, b, k, depth);
    S.force_dir = dir;
    S.feat_log = dfeat;
    S.time_log = dtime;
    S.max_log = max_rows;
    if (cudaMemcpyAsync(b.dsrc, sources, sizeof(int32_t) * k, cudaMemcpyDefault, st) != cudaSuccess ||
        (status = msbfs_enqueue(g, st, S, b.dsrc, false)) != GG_OK)
      break;
    int32_t lv = 0;
    if (cudaMemcpyAsync(&lv, S.stats, sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      status = set_error(GG_ERR_CUDA, "batched BFS timing run failed");
      break;
    }
    if ((status = check_device_error(g, "batch_collect")) != GG_OK) break;
    if (levels >= 0 && lv != levels) {
      status = set_error(GG_ERR_STATE, "level counts differ between direction runs (%d, %d)", levels, lv);
      break;
    }
    levels = lv;
    const int32_t rows = std::min(levels, max_rows);
    cudaMemcpy(ht.data(), dtime, sizeof(unsigned long long) * ((size_t)rows + 1), cudaMemcpyDeviceToHost);
    for (int32_t l = 0; l < rows; ++l)
      best[2 * l + dir] = std::min(best[2 * l + dir], (float)((double)(ht[l + 1] - ht[l]) * 1e-6));
    if (rep == 0)
      cudaMemcpy(feats, dfeat, sizeof(float) * kSelectorFeatures * (size_t)rows, cudaMemcpyDeviceToHost);
  }
  cudaFreeAsync(dfeat, st);
  cudaFreeAsync(dtime, st);
  GG_TRY(status);
  *nrows = std::min(levels, max_rows);
  for (int32_t i = 0; i < 2 * *nrows; ++i) times[i] = best[i];
  return GG_OK;
}
