// PageRank pull iteration for PULL + TWC schedules: the vertices fall into three
// classes by in-degree (thread / warp / tiles of a CTA per vertex, the TWC binning
// of graph.h:48-54 applied to the pull gather), and every iteration is one launch
// that fuses pr.cpp's three steps
//   contrib[u] = old[u] / outdeg[u];   new[v] = sum contrib[u];
//   old[v] = (1-d)/V + d * new[v]
// (apps/pr.cpp:28-41).  Each vertex's sum is formed in a fixed order -- by its
// owner, or for hubs from per-tile partial sums added in tile order -- so there
// are no float atomics and results are bit-identical across runs.  The next
// iteration's contributions go to the other half of a double buffer.
//
// The iteration runs on the degree-ordered copy of the graph (relabel.cu): the
// contributions of the high-degree vertices, read by most in-edges, share cache
// lines, and the classes are ranges of ids -- that order goes by floor(log2(degree +
// 1)), so a boundary at 2^k - 1 is found by bisection and no bins are built.  Ranks
// come back to the caller's ids at the end.
//
// What bounds the gathers is the L1's rate of scattered sectors (74 % of it in the
// warp class), so every lane keeps four contrib loads in flight and the classes
// run side by side: in launches of their own they left its tails empty three times
// an iteration (directed R-MAT 22, an iteration: 49 + 142 + 31 + 5 us in four
// launches, now 183 in one).
#include <algorithm>
#include <vector>

#include "engine.h"

namespace gg {

constexpr int32_t kPrSmallMax = 31;   // in-degree < 31: one thread
constexpr int32_t kPrMidMax = 4095;   // < 4095: one warp; else tiles of kPrTile edges
constexpr int32_t kPrTile = 4096;     // in-edges per CTA tile of a hub: 16 a thread
constexpr int32_t kPrThreads = 256;
constexpr int32_t kPrMidPer = 4;      // most vertices a warp of the middle class takes

struct PrArgs {
  const int32_t *toff, *tsrc;   // CSC
  const int32_t *off;           // forward CSR (out-degrees)
  const float *contrib;         // this iteration
  float *contrib_next;          // next iteration
  float *rank;                  // old_rank
  float beta, damp;
};

__device__ __forceinline__ void pr_finish(const PrArgs &a, int32_t v, float s) {
  const float r = a.beta + a.damp * s;
  a.rank[v] = r;
  a.contrib_next[v] = r / (float)(a.off[v + 1] - a.off[v]);  // a sink divides by 0, as pr.cpp
}

// Sum of contrib over in-edges k = k0, k0 + step, ... < k1, four loads in flight.
__device__ __forceinline__ float pr_gather(const PrArgs &a, int32_t k0, int32_t k1, int32_t step) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int32_t k = k0;
  for (; k + 3 * step < k1; k += 4 * step) {
    const int32_t u0 = __ldg(a.tsrc + k), u1 = __ldg(a.tsrc + k + step);
    const int32_t u2 = __ldg(a.tsrc + k + 2 * step), u3 = __ldg(a.tsrc + k + 3 * step);
    s0 += __ldg(a.contrib + u0);
    s1 += __ldg(a.contrib + u1);
    s2 += __ldg(a.contrib + u2);
    s3 += __ldg(a.contrib + u3);
  }
  for (; k < k1; k += step) s0 += __ldg(a.contrib + __ldg(a.tsrc + k));
  return (s0 + s1) + (s2 + s3);
}

// One iteration.  Hubs are vertices [0, nh), their tiles in vertex order: tile t
// covers in-edges [tile_k[t], + kPrTile) of tile_v[t], hub v owns tiles [first[v],
// first[v + 1]).  The middle class is [nh, mid), the rest single threads'.  Blocks
// come in that order, the longest work first.
struct PrIter {
  PrArgs a;
  const int32_t *first, *tile_v, *tile_k;
  double *partial;  // [ntiles]
  int32_t *done;    // [nh] tiles of a hub summed so far; zero between iterations
  int32_t ntiles, nh, mid, V, mid_blocks, mid_per;
};

__global__ void __launch_bounds__(kPrThreads) k_pr_iter(PrIter p) {
  const PrArgs &a = p.a;
  const int32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t b = (int32_t)blockIdx.x;
  if (b < p.ntiles) {
    __shared__ float part[kPrThreads / 32];
    const int32_t v = p.tile_v[b];
    const int32_t kb = p.tile_k[b], ke = min(kb + kPrTile, __ldg(a.toff + v + 1));
    float s = pr_gather(a, kb + (int32_t)threadIdx.x, ke, kPrThreads);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) part[wid] = s;
    __syncthreads();
    if (threadIdx.x != 0) return;
    // the warps' and the tiles' sums are few: added in fp64, they round once
    double sum = 0.0;
    for (int w = 0; w < kPrThreads / 32; ++w) sum += (double)part[w];
    const int32_t t0 = p.first[v], t1 = p.first[v + 1];
    p.partial[b] = sum;
    __threadfence();
    if (atomicAdd(p.done + v, 1) != t1 - t0 - 1) return;
    __threadfence();  // the hub's last tile adds them all, in tile order
    sum = 0.0;
    for (int32_t t = t0; t < t1; ++t) sum += __ldcg(p.partial + t);
    p.done[v] = 0;
    pr_finish(a, v, (float)sum);
    return;
  }
  b -= p.ntiles;
  if (b < p.mid_blocks) {
    const int32_t v0 = p.nh + (b * (kPrThreads / 32) + wid) * p.mid_per, v1 = min(v0 + p.mid_per, p.mid);
    for (int32_t v = v0; v < v1; ++v) {
      float s = pr_gather(a, __ldg(a.toff + v) + lane, __ldg(a.toff + v + 1), 32);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (lane == 0) pr_finish(a, v, s);
    }
    return;
  }
  b -= p.mid_blocks;
  const int64_t v = (int64_t)p.mid + (int64_t)b * kPrThreads + threadIdx.x;
  if (v < p.V) pr_finish(a, (int32_t)v, pr_gather(a, __ldg(a.toff + v), __ldg(a.toff + v + 1), 1));
}

// bounds[i] = first vertex whose in-degree class lies below the i-th boundary
// (in-degrees fall from class to class; a thread bisects for each).
__global__ void k_pr_bounds(const int32_t *__restrict__ toff, int32_t V, int32_t *__restrict__ bounds) {
  if (threadIdx.x >= 2) return;
  const int32_t least = threadIdx.x == 0 ? kPrMidMax : kPrSmallMax;
  int32_t lo = 0, len = V;
  while (len > 0) {
    const int32_t half = len >> 1, v = lo + half;
    if (__ldg(toff + v + 1) - __ldg(toff + v) >= least) {
      lo = v + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  bounds[threadIdx.x] = lo;
}

__global__ void k_pr_unperm(const float *__restrict__ rank_new, const int32_t *__restrict__ perm, int32_t V,
                            float *__restrict__ rank) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    rank[v] = rank_new[perm[v]];
}

__global__ void k_pr_init(const int32_t *__restrict__ off, int32_t V, float inv_v, float *rank, float *contrib) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    rank[v] = inv_v;  // pr.cpp:43-46
    contrib[v] = inv_v / (float)(off[v + 1] - off[v]);
  }
}

// The classes' ranges and the hubs' tiles.  Hubs are few: their tile list is laid
// out on the host.
static gg_status pr_plan(gg_graph *g, const GraphStore &t, PrIter *P) {
  const int32_t V = g->csr.V;
  cudaStream_t st = g->stream;
  void *p = nullptr;
  GG_TRY(scratch_get(g, 3, sizeof(int32_t) * 2, &p));
  note_launch();
  k_pr_bounds<<<1, 32, 0, st>>>(t.off, V, (int32_t *)p);
  GG_CUDA(cudaGetLastError());
  int32_t bounds[2];
  GG_CUDA(cudaMemcpyAsync(bounds, p, sizeof(bounds), cudaMemcpyDeviceToHost, st));
  GG_CUDA(cudaStreamSynchronize(st));
  const int32_t nh = bounds[0];
  P->nh = nh;
  P->mid = bounds[1];
  P->V = V;
  // Vertices of a middle warp: as many as the class has for each warp of the GPU, so
  // that a small one is spread over it (ten iterations, four a warp / as here: complete
  // graph of 400 vertices 114 / 86 us, directed R-MAT 17 317 / 191).
  const int32_t warps = g->sm_count * (2048 / 32);
  P->mid_per = std::min(kPrMidPer, std::max(1, (bounds[1] - nh) / warps));
  P->mid_blocks = ceil_div(bounds[1] - nh, kPrThreads / 32 * P->mid_per);
  P->ntiles = 0;
  if (nh == 0) return GG_OK;
  std::vector<int32_t> off(nh + 1), plan(nh + 1, 0), tv, tk;
  GG_CUDA(cudaMemcpyAsync(off.data(), t.off, sizeof(int32_t) * off.size(), cudaMemcpyDeviceToHost, st));
  GG_CUDA(cudaStreamSynchronize(st));
  for (int32_t v = 0; v < nh; ++v) {
    plan[v] = (int32_t)tv.size();
    for (int64_t k = off[v]; k < off[v + 1]; k += kPrTile) {
      tv.push_back(v);
      tk.push_back((int32_t)k);
    }
  }
  const int32_t ntiles = (int32_t)tv.size();
  plan[nh] = ntiles;
  plan.insert(plan.end(), tv.begin(), tv.end());
  plan.insert(plan.end(), tk.begin(), tk.end());
  // layout: first[nh + 1] tile_v[ntiles] tile_k[ntiles], partial[ntiles] on an
  // 8-byte boundary, done[nh]
  const size_t words = (plan.size() + 1) / 2 * 2;
  GG_TRY(scratch_get(g, 2, sizeof(int32_t) * (words + 2 * (size_t)ntiles + (size_t)nh), &p));
  int32_t *d = (int32_t *)p;
  GG_CUDA(cudaMemcpyAsync(d, plan.data(), sizeof(int32_t) * plan.size(), cudaMemcpyHostToDevice, st));
  P->first = d;
  P->tile_v = d + nh + 1;
  P->tile_k = P->tile_v + ntiles;
  P->partial = reinterpret_cast<double *>(d + words);
  P->done = d + words + 2 * (size_t)ntiles;
  P->ntiles = ntiles;
  GG_CUDA(cudaMemsetAsync(P->done, 0, sizeof(int32_t) * (size_t)nh, st));
  GG_CUDA(cudaStreamSynchronize(st));  // the host vector goes out of scope
  return GG_OK;
}

gg_status pagerank_pull_twc(gg_graph *g, int32_t iters, float damping, float *rank_out, float *contrib2) {
  GG_TRY(ensure_relabel(g));
  GG_TRY(ensure_relabel_csc(g));
  const int32_t V = g->csr.V;
  const GraphStore &t = g->symmetric ? g->rel->g : g->rel->csc;  // in-lists in new ids
  float *rank = nullptr;  // ranks in new ids
  GG_TRY(scratch_get_app(g, 4, sizeof(float) * std::max(V, 1), (void **)&rank));
  PrIter P{};
  GG_TRY(pr_plan(g, t, &P));
  cudaStream_t st = g->stream;
  const float inv_v = (float)(1.0 / V);
  note_launch();
  k_pr_init<<<g->sm_count * 8, 256, 0, st>>>(g->rel->g.off, V, inv_v, rank, contrib2);
  PrArgs &a = P.a;
  a.toff = t.off;
  a.tsrc = t.dst;
  a.off = g->rel->g.off;  // out-degrees in new ids
  a.rank = rank;
  a.beta = (float)((1.0 - (double)damping) / V);  // pr.cpp:37
  a.damp = damping;
  const int blocks = std::max(1, P.ntiles + P.mid_blocks + ceil_div(V - P.mid, kPrThreads));
  for (int32_t it = 0; it < iters; ++it) {
    a.contrib = contrib2 + (size_t)(it & 1) * V;
    a.contrib_next = contrib2 + (size_t)((it + 1) & 1) * V;
    note_launch();
    k_pr_iter<<<blocks, kPrThreads, 0, st>>>(P);
  }
  note_launch();
  k_pr_unperm<<<g->sm_count * 8, 256, 0, st>>>(rank, g->rel->perm, V, rank_out);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg
