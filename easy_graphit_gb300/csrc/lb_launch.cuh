// Kernels wrapping the load-balancing device functions, and the host-side
// dispatch of one edgeset.apply launch (the switch of operators.cpp:631-647).
// Included by one translation unit per UDF so each UDF's kernels compile in
// parallel.
#pragma once

#include <type_traits>

#include "engine.h"
#include "lb.cuh"
#include "udf.cuh"

namespace gg {

// A kernel's stages: appends to the output queue and, for the relax UDF, to the
// far piles (Stage, common.cuh).  begin() before the work, end() after it, by the
// whole CTA.  UDFs that track nothing have none, and a launch of at most
// kStagedGrid CTAs on a graph of short lists (DOut::few) appends to the queue
// directly: its count is not what binds there, and the stage's barriers and the
// reservation at the end of the kernel are a tenth of it (BFS on a 200^2 grid, 399
// launches of at most 13 CTAs: WM 10.4 -> 10.0 ms, TWCE 11.95 -> 11.4).  With longer
// lists a CTA finds enough to be worth it (complete graph of 400 vertices, a thread
// per vertex: 703 us staged, 822 not).
constexpr uint32_t kStagedGrid = 64;
template <class F>
struct KernelStages {
  static constexpr int kStages = !F::kPushes ? 0 : (lb_batch<F>::value ? 3 : 1);
  StageMem st[kStages > 0 ? kStages : 1];
  __device__ __forceinline__ void begin(F &f, DOut &out) {
    if constexpr (kStages > 0) {
      if (threadIdx.x < kStages) st[threadIdx.x].s.init(kStageCap);
      __syncthreads();
      if ((out.mode == OUT_SPARSE || out.mode == OUT_SPARSE_DEDUP) && !(out.few && gridDim.x <= kStagedGrid))
        out.stage = &st[0].s;
      if constexpr (kStages == 3) f.stage_parks(&st[1].s, &st[2].s);
    }
  }
  __device__ __forceinline__ void end(const F &f, const DOut &out) {
    if constexpr (kStages > 0) {
      if (out.stage) stage_flush(out);
      f.flush();
    }
  }
};
template <class F>
struct NoStages {
  __device__ __forceinline__ void begin(F &, DOut &) {}
  __device__ __forceinline__ void end(const F &, const DOut &) {}
};
// Shared memory only where there is something to stage.
#define GG_STAGES(F, f, out)                                                       \
  using Stages_ = std::conditional_t<F::kPushes, KernelStages<F>, NoStages<F>>;    \
  __shared__ Stages_ stages_;                                                      \
  stages_.begin(f, out)
#define GG_STAGES_END(f, out) stages_.end(f, out)

template <class F>
__global__ void __launch_bounds__(1024) k_vertex(DGraph g, Enum en, F f, DOut out) {
  GG_STAGES(F, f, out);
  const int32_t n = en.count();
  const int32_t nv = ceil_div(n, blockDim.x);
  for (int32_t v = blockIdx.x; v < nv; v += gridDim.x) lb_vertex(g, en, n, f, out, v);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024) k_wm(DGraph g, Enum en, F f, DOut out) {
  GG_STAGES(F, f, out);
  const int32_t n = en.count();
  const int32_t nv = ceil_div(n, blockDim.x >> 5);
  for (int32_t v = blockIdx.x; v < nv; v += gridDim.x) lb_wm(g, en, n, f, out, v);
  GG_STAGES_END(f, out);
}

// One whole CTA per enumerated vertex (TWC large bin).
template <class F>
__global__ void __launch_bounds__(1024) k_cta(DGraph g, Enum en, F f, DOut out) {
  GG_STAGES(F, f, out);
  const int32_t n = en.count();
  for (int32_t v = blockIdx.x; v < n; v += gridDim.x) {
    const int32_t s = en.at(v);
    do_range(g, f, out, s, __ldg(g.off + s), __ldg(g.off + s + 1), threadIdx.x, blockDim.x);
  }
  GG_STAGES_END(f, out);
}

// TWCE, and with a hub list that takes every CTA part ETWC.
template <class F>
__global__ void __launch_bounds__(1024) k_twce(DGraph g, Enum en, F f, DOut out, HubList hub) {
  GG_STAGES(F, f, out);
  extern __shared__ int4 smem_raw[];
  lb_twce_all(g, en, en.count(), f, out, blockIdx.x, gridDim.x, *reinterpret_cast<TwceSmem *>(smem_raw), hub);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024)
    k_chunks(DGraph g, const int32_t *chunks, const int32_t *chunk_cnt, int32_t cap, F f, DOut out) {
  GG_STAGES(F, f, out);
  const int32_t n = min(*(volatile const int32_t *)chunk_cnt, cap);
  for (int32_t v = blockIdx.x; v < n; v += gridDim.x) lb_chunk(g, chunks, f, out, v);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024) k_cm(DGraph g, Enum en, F f, DOut out) {
  GG_STAGES(F, f, out);
  extern __shared__ int4 smem_raw[];
  CmSmem &sm = *reinterpret_cast<CmSmem *>(smem_raw);
  const int32_t n = en.count();
  const int32_t nv = ceil_div(n, blockDim.x);
  for (int32_t v = blockIdx.x; v < nv; v += gridDim.x) lb_cm(g, en, n, f, out, v, sm);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024)
    k_strict(DGraph g, Enum en, const int32_t *sum, F f, DOut out, int32_t per) {
  GG_STAGES(F, f, out);
  const int32_t n = en.count();
  const int32_t nv = ceil_div(sum[n], per);
  for (int32_t v = blockIdx.x; v < nv; v += gridDim.x) lb_strict(g, en, n, sum, f, out, v, per);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024) k_edge_only(DGraph g, F f, DOut out) {
  GG_STAGES(F, f, out);
  lb_edge_only(g, f, out, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
               (int64_t)gridDim.x * blockDim.x);
  GG_STAGES_END(f, out);
}

template <class F>
__global__ void __launch_bounds__(1024) k_edge_only_blocked(DGraph g, F f, DOut out) {
  GG_STAGES(F, f, out);
  lb_edge_only_blocked(g, f, out, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
                       (int64_t)gridDim.x * blockDim.x);
  GG_STAGES_END(f, out);
}

// Helpers implemented in frontier.cu (not UDF-specific).
gg_status twc_bin(gg_graph *G, const DGraph &g, const Enum &en, int32_t n_host, int32_t cta,
                  int32_t **bins, int32_t **bin_cnt);
gg_status strict_scan(gg_graph *G, const DGraph &g, const Enum &en, int32_t n_host,
                      int32_t **sum);
gg_status etwc_scratch(gg_graph *G, int64_t max_chunks, int32_t **chunks, int32_t **cnt);

template <class K>
inline int grid_for(K kernel, int cta, size_t smem, int sm_count, int64_t nvcta) {
  const int res = resident_grid((const void *)kernel, cta, smem, sm_count);
  if (nvcta < 0) return res;
  return (int)std::max<int64_t>(1, std::min<int64_t>(nvcta, res));
}

// Grid of a TWCE launch: the resident CTAs, or up to kTwceWaves times as many
// slices when the frontier is small (a slice without work ends after one read
// of its vertices, so hubs are split finely even where every CTA has some: unfused
// BFS on a symmetrized R-MAT 17 / 20 / 22, 1 wave 316 / 636 / 1,580 us, 4 waves 311 / 598 /
// 1,574, 16 waves 400 / 649 / 1,545).
constexpr int kTwceWaves = 4;
template <class F>
void launch_twce(const EdgeLaunch &L, const F &f, const HubList &hub) {
  auto k = k_twce<F>;
  const size_t sm = twce_smem_bytes(L.cta);
  const int res = resident_grid((const void *)k, L.cta, sm, L.graph->sm_count);
  int grid = res;
  if (L.n_host >= 0) {
    const int64_t nv = ceil_div(L.n_host, L.cta / kStage1);
    if (nv < (int64_t)kTwceWaves * res)
      grid = (int)(nv * std::max<int64_t>(1, std::min<int64_t>(kTwceWaves * (int64_t)res / nv, hub.slices)));
  }
  note_launch();
  k<<<grid, L.cta, sm, L.graph->stream>>>(L.g, L.en, f, L.out, hub);
}

template <class F>
gg_status launch_lb(const EdgeLaunch &L, const F &f) {
  gg_graph *G = L.graph;
  cudaStream_t st = G->stream;
  const int cta = L.cta;
  const int sms = G->sm_count;
  const int64_t n = L.n_host;
  if (n == 0 && L.lb != GG_LB_EDGE_ONLY) return GG_OK;
  HubList hub;
  if (!L.pull || G->symmetric) hub.slices = slice_limit(G->max_degree);  // in-lists of a directed graph are not bounded
  switch (L.lb) {
    case GG_LB_EDGE_ONLY: {
      if (L.g.nbuckets > 0) {
        auto k = k_edge_only_blocked<F>;
        { gg::note_launch(); k<<<grid_for(k, cta, 0, sms, -1), cta, 0, st>>>(L.g, f, L.out); }
      } else {
        auto k = k_edge_only<F>;
        { gg::note_launch(); k<<<grid_for(k, cta, 0, sms, -1), cta, 0, st>>>(L.g, f, L.out); }
      }
      break;
    }
    case GG_LB_VERTEX_BASED: {
      auto k = k_vertex<F>;
      { gg::note_launch(); k<<<grid_for(k, cta, 0, sms, n < 0 ? -1 : ceil_div(n, cta)), cta, 0, st>>>(L.g, L.en, f, L.out); }
      break;
    }
    case GG_LB_WM: {
      auto k = k_wm<F>;
      { gg::note_launch(); k<<<grid_for(k, cta, 0, sms, n < 0 ? -1 : ceil_div(n, cta / 32)), cta, 0, st>>>(L.g, L.en, f,
                                                                                     L.out); }
      break;
    }
    case GG_LB_TWCE: {
      launch_twce(L, f, hub);
      break;
    }
    case GG_LB_ETWC: {
      // Stage 1+2 in-CTA, hub edges as chunks of 4*cta edges on a global list.
      const int32_t chunk = kHubChunk * cta;
      int32_t *chunks = nullptr, *cnt = nullptr;
      const int64_t maxc = (int64_t)L.g.E / chunk + (n < 0 ? L.g.V : n) + 1;
      GG_TRY(etwc_scratch(G, maxc, &chunks, &cnt));
      GG_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int32_t), st));
      hub.list = chunks;
      hub.cnt = cnt;
      hub.cap = (int32_t)maxc;
      hub.min = 0;
      launch_twce(L, f, hub);
      auto k2 = k_chunks<F>;
      { gg::note_launch(); k2<<<grid_for(k2, cta, 0, sms, -1), cta, 0, st>>>(L.g, chunks, cnt, (int32_t)maxc, f, L.out); }
      break;
    }
    case GG_LB_CM: {
      auto k = k_cm<F>;
      const size_t sm = cm_smem_bytes(cta);
      { gg::note_launch(); k<<<grid_for(k, cta, sm, sms, n < 0 ? -1 : ceil_div(n, cta)), cta, sm, st>>>(L.g, L.en, f,
                                                                                  L.out); }
      break;
    }
    case GG_LB_TWC: {
      int32_t *bins = nullptr, *bin_cnt = nullptr;
      GG_TRY(twc_bin(G, L.g, L.en, (int32_t)n, cta, &bins, &bin_cnt));
      const int64_t cap = n < 0 ? L.g.V : n;
      Enum small{bins, bin_cnt + 0, -1}, mid{bins + cap, bin_cnt + 1, -1},
          large{bins + 2 * cap, bin_cnt + 2, -1};
      auto k1 = k_vertex<F>;
      auto k2 = k_wm<F>;
      auto k3 = k_cta<F>;
      { gg::note_launch(); k1<<<grid_for(k1, cta, 0, sms, -1), cta, 0, st>>>(L.g, small, f, L.out); }
      { gg::note_launch(); k2<<<grid_for(k2, cta, 0, sms, -1), cta, 0, st>>>(L.g, mid, f, L.out); }
      { gg::note_launch(); k3<<<grid_for(k3, cta, 0, sms, -1), cta, 0, st>>>(L.g, large, f, L.out); }
      break;
    }
    case GG_LB_STRICT: {
      int32_t *sum = nullptr;
      GG_TRY(strict_scan(G, L.g, L.en, (int32_t)n, &sum));
      auto k = k_strict<F>;
      { gg::note_launch(); k<<<grid_for(k, cta, 0, sms, -1), cta, 0, st>>>(L.g, L.en, sum, f, L.out, 8 * cta); }
      break;
    }
    default:
      return set_error(GG_ERR_UNSUPPORTED, "load balancing %d not supported", L.lb);
  }
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

template <class U>
gg_status launch_dir(EdgeLaunch L, const U &u) {
  L.out.few = (!L.pull || L.graph->symmetric) && L.graph->max_degree <= kStage1;
  if (L.pull) return launch_lb(L, EdgeF<U, true>{u, L.in_src, L.in_dst, L.filter});
  return launch_lb(L, EdgeF<U, false>{u, L.in_src, L.in_dst, L.filter});
}

}  // namespace gg
