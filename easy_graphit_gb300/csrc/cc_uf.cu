// Connected components with fuse_kernel on: a lock-free union-find whose roots
// are always the smallest id of their tree, driven in the sampling order of
// Afforest (Sutton, Ben-Nun, Barak: "Optimizing Parallel Graph Connectivity
// Computation via Subgraph Sampling", IPDPS 2018).
//
//   init     parent[v] = min(v, first neighbour of v)  (adjacency lists are
//            sorted, so that is v's smallest neighbour)
//   sample   compress init's chains; union(v, first neighbour of v) where that
//            neighbour is larger (init joined a smaller one) and union(v, second
//            neighbour of v), a few scouts before the rest; compress every
//            vertex to its root
//   giant    c = the most frequent root among 1,024 spread-out vertices
//   finish   every vertex whose root is not c unions with the rest of its
//            neighbours -- out-neighbours after the two sampled ones and, on a
//            directed graph, all in-neighbours -- so every edge with an end
//            outside c's tree is seen from that end; edges inside c's tree
//            change nothing and are skipped
//   final    label[v] = find(v)
//
// union(u, v) finds both roots with path halving and hooks the larger root
// under the smaller with a CAS, retrying from the new roots if another thread
// hooked first.  Every step keeps parent[x] <= x, so a tree's root is its
// smallest vertex and the final labels are the minimum id of each (weakly)
// connected component -- the canonical labels cc.cpp's hook / pointer-jump
// rounds converge to (apps/cc.cpp:23-77).  Concurrent path-halving stores only
// ever move a vertex up its own tree, so the races are benign.
#include <algorithm>
#include <vector>

#include "engine.h"

namespace gg {

// Reads go through L1.  Once trees have merged, most walks end at the same few
// roots, and with every read sent to L2 those lines served one warp at a time
// (second sampling pass on a symmetrized R-MAT 22: 646 us; 268 us through L1).
// A stale line is harmless: it holds an older ancestor of x, so the walk stays
// in x's tree, stores only ancestors, and a stale root is found out by the CAS
// in uf_union, whose answer is the true parent.
__device__ __forceinline__ int32_t uf_find(int32_t *parent, int32_t x) {
  for (;;) {
    const int32_t p = __ldca(parent + x);
    if (p == x) return x;
    const int32_t gp = __ldca(parent + p);
    if (gp == p) return p;
    parent[x] = gp;  // path halving
    x = gp;
  }
}

__device__ __forceinline__ void uf_union(int32_t *parent, int32_t u, int32_t v) {
  int32_t ru = uf_find(parent, u), rv = uf_find(parent, v);
  while (ru != rv) {
    if (ru < rv) {
      const int32_t t = ru;
      ru = rv;
      rv = t;
    }
    const int32_t old = atomicCAS(parent + ru, ru, rv);  // hook the larger root
    if (old == ru) return;
    ru = uf_find(parent, old);
    rv = uf_find(parent, rv);
  }
}

__global__ void k_uf_init(const int32_t *__restrict__ off, const int32_t *__restrict__ dst, int32_t V,
                          int32_t *__restrict__ parent) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int32_t b = off[v];
    parent[v] = (off[v + 1] > b) ? min(v, dst[b]) : v;
  }
}

// Link v with its out-neighbour number r (the sampling rounds), over the
// groups of 32 vertices that `part` names: all of them, the scouts (every
// `every`-th group) or the others.
enum : int32_t { UF_ALL = 0, UF_SCOUTS = 1, UF_OTHERS = 2 };
__global__ void k_uf_sample(const int32_t *__restrict__ off, const int32_t *__restrict__ dst, int32_t V, int32_t r,
                            int32_t part, int32_t every, int32_t *__restrict__ parent) {
  const int32_t groups = ceil_div(V, 32), lane = threadIdx.x & 31;
  const int32_t scouts = ceil_div(groups, every);
  const int32_t n = part == UF_ALL ? groups : (part == UF_SCOUTS ? scouts : groups - scouts);
  for (int32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    const int32_t gi = part == UF_ALL ? i : (part == UF_SCOUTS ? i * every : i + i / (every - 1) + 1);
    const int64_t v64 = (int64_t)gi * 32 + lane;
    if (v64 >= V) continue;
    const int32_t v = (int32_t)v64, b = off[v];
    if (off[v + 1] - b > r) {
      const int32_t u = dst[b + r];
      if (u != v && (r > 0 || u > v)) uf_union(parent, v, u);  // init joined a smaller first one
    }
  }
}

__global__ void k_uf_compress(int32_t *__restrict__ parent, int32_t V) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    parent[v] = uf_find(parent, v);
}

// roots[i] = parent of vertex floor(i * V / n) (spread over the id range).
__global__ void k_uf_probe(const int32_t *__restrict__ parent, int32_t V, int32_t n, int32_t *__restrict__ roots) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    roots[i] = parent[(int32_t)((int64_t)i * V / n)];
}

// Unions of the vertices outside c's tree with list entries [off[v] + skip,
// off[v+1]).  A thread walks a short list; lists longer than 64 entries are
// walked by the whole warp, one after another.
__global__ void k_uf_finish(const int32_t *__restrict__ off, const int32_t *__restrict__ adj, int32_t V,
                            int32_t skip, int32_t c, int32_t *__restrict__ parent) {
  const int32_t lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t end = (V + stride - 1) / stride * stride;  // whole warps iterate together
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < end; i += stride) {
    const int32_t v = (int32_t)i;
    int32_t b = 0, e = 0;
    if (v < V && __ldcg(parent + v) != c) {
      b = off[v] + skip;
      e = off[v + 1];
    }
    uint32_t big = __ballot_sync(0xffffffffu, e - b > 64);
    while (big) {
      const int32_t l = __ffs(big) - 1;
      big &= big - 1;
      const int32_t vv = __shfl_sync(0xffffffffu, v, l);
      const int32_t bb = __shfl_sync(0xffffffffu, b, l), ee = __shfl_sync(0xffffffffu, e, l);
      for (int32_t k = bb + lane; k < ee; k += 32) {
        const int32_t u = adj[k];
        if (u != vv) uf_union(parent, vv, u);
      }
    }
    if (e - b <= 64)
      for (int32_t k = b; k < e; ++k) {
        const int32_t u = adj[k];
        if (u != v) uf_union(parent, v, u);
      }
  }
}

__global__ void k_uf_final(int32_t *__restrict__ parent, int32_t V, int32_t *__restrict__ labels) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    labels[v] = uf_find(parent, v);
}

constexpr int32_t kUfProbes = 1024;
// Vertices of the second sampling round that go first.  Whole calls with 1,024 / 16,384 /
// 65,536: symmetrized R-MAT 20 313 / 279 / 274 us, 22 438 / 453 / 438, uniform degree 16, 4 M
// vertices, 667 / 658 / 607, degree 32, 1 M, 729 / 304 / 334, 2048^2 grid 872 / 751 / 832.
constexpr int32_t kUfScouts = 16384;

gg_status cc_union_find(gg_graph *g, int32_t *labels, int32_t *parent) {
  const GraphStore &f = g->csr;
  const int32_t V = f.V;
  if (V == 0) return GG_OK;
  if (!g->symmetric) GG_TRY(ensure_transpose(g));  // in-lists: weak components
  cudaStream_t st = g->stream;
  const int grid = g->sm_count * 8;
  note_launch();
  k_uf_init<<<grid, 256, 0, st>>>(f.off, f.dst, V, parent);
  // flatten init's first-neighbour chains before the unions walk them
  note_launch();
  k_uf_compress<<<grid, 256, 0, st>>>(parent, V);
  note_launch();
  k_uf_sample<<<grid, 256, 0, st>>>(f.off, f.dst, V, 0, UF_ALL, 2, parent);
  // The second round is where the big trees meet: with every thread of the GPU
  // hooking the same few roots at once it is bound by failed CASes.  A few
  // thousand scouts join those trees first; the rest then find one root
  // (symmetrized R-MAT 22, both launches: 268 us unsplit, 270 with 262,144
  // scouts, 145 with 65,536, 114 with 16,384, 104 with 4,096 but a slower whole).
  // A graph whose scouts would be more than a sixteenth goes in one launch.
  const int32_t every = V / kUfScouts;
  if (every >= 16) {
    note_launch();
    k_uf_sample<<<grid, 256, 0, st>>>(f.off, f.dst, V, 1, UF_SCOUTS, every, parent);
  }
  note_launch();
  k_uf_sample<<<grid, 256, 0, st>>>(f.off, f.dst, V, 1, every >= 16 ? UF_OTHERS : UF_ALL, std::max(every, 2), parent);
  note_launch();
  k_uf_compress<<<grid, 256, 0, st>>>(parent, V);
  // the giant tree's root, by majority over spread-out vertices
  const int32_t n = std::min(kUfProbes, std::max(V, 1));
  void *p = nullptr;
  GG_TRY(scratch_get(g, 1, sizeof(int32_t) * kUfProbes, &p));
  int32_t *d_roots = (int32_t *)p;
  note_launch();
  k_uf_probe<<<ceil_div(n, 256), 256, 0, st>>>(parent, V, n, d_roots);
  GG_CUDA(cudaGetLastError());
  std::vector<int32_t> roots(n);
  GG_CUDA(cudaMemcpyAsync(roots.data(), d_roots, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st));
  GG_CUDA(cudaStreamSynchronize(st));
  std::sort(roots.begin(), roots.end());
  int32_t c = V > 0 ? roots[0] : 0, best = 0;
  for (int32_t i = 0, j; i < n; i = j) {
    for (j = i; j < n && roots[j] == roots[i]; ++j) {
    }
    if (j - i > best) {
      best = j - i;
      c = roots[i];
    }
  }
  note_launch();
  k_uf_finish<<<grid, 256, 0, st>>>(f.off, f.dst, V, 2, c, parent);
  if (!g->symmetric) {
    note_launch();
    k_uf_finish<<<grid, 256, 0, st>>>(g->csc->off, g->csc->dst, V, 0, c, parent);
  }
  note_launch();
  k_uf_final<<<grid, 256, 0, st>>>(parent, V, labels);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

}  // namespace gg
