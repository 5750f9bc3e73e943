// Betweenness centrality from one source in one persistent kernel: the
// fuse_kernel form of bc.cpp's two sweeps (apps/bc.cpp:64-123).  Unfused, every
// level is an edge launch, a vertex launch, a list insertion and a frontier size
// read back, twice: 22 launches and as many round trips to the host for the five
// levels of a 0.1 M-vertex R-MAT, 690 us, of which the edges are a third.
//
//   forward   level by level over the queue: an edge into an unreached vertex or
//             one reached at this very level adds sigma[u] to sigma[v], and the
//             first such edge queues v.  Queues follow each other in `lev`, which
//             is bc.cpp's stack of levels.
//   backward  deepest level first: dep[v] += 1 / sigma[v] for its vertices, then
//             their edges into shallower vertices add dep[u] to dep[v].
//   final     dep[v] = (dep[v] - 1 / sigma[v]) * sigma[v], 0 where unreached.
//
// The depth of a vertex stands for bc.cpp's visited flags: in the forward sweep
// unvisited means no depth yet or this level's, in the backward sweep, where
// levels are marked from the deepest up, it means a smaller depth than the edge's
// source.  Sums are fp64, as in the unfused form.
#include "bq_loop.cuh"
#include "engine.h"

namespace gg {

struct BcArgs {
  DGraph g;
  int32_t *depth, *lev, *loff;  // loff[d]: start of level d in lev
  double *sigma, *dep;
  float *out;
  int32_t *cnt3, *hub3;         // queue and hub-chunk counts, rotating by level / edge pass
  int32_t *hub_list;
  int32_t hub_cap, hub_min, hub_slices;
  uint32_t *bar;
  int32_t *err, *stats, *stop;
  uint64_t timeout_ns, loop_limit_ns;
  int32_t src;
};

struct UBcFwd {
  static constexpr bool kWeight = false;
  int32_t *depth;
  double *sigma;
  int32_t level;
  __device__ __forceinline__ bool src_ok(int32_t) const { return true; }
  __device__ __forceinline__ bool dst_ok(int32_t v) const {
    const int32_t d = __ldcg(depth + v);
    return d == -1 || d == level;
  }
  __device__ __forceinline__ int32_t apply(int32_t u, int32_t v, int32_t) const {
    const int32_t was = __ldcg(depth + v) == -1 ? atomicCAS(depth + v, -1, level) : level;
    atomicAdd(sigma + v, __ldcg(sigma + u));  // reached at this level, here or by another thread
    return was == -1 ? v : -1;
  }
};

struct UBcBwd {
  static constexpr bool kWeight = false;
  const int32_t *depth;
  double *dep;
  int32_t level;  // of the sources
  __device__ __forceinline__ bool src_ok(int32_t) const { return true; }
  __device__ __forceinline__ bool dst_ok(int32_t v) const {
    const int32_t d = __ldcg(depth + v);  // written earlier in this kernel: not through the read-only path
    return d >= 0 && d < level;
  }
  __device__ __forceinline__ int32_t apply(int32_t u, int32_t v, int32_t) const {
    atomicAdd(dep + v, __ldcg(dep + u));
    return -1;
  }
};

__global__ void k_bc_setup(BcArgs a) {
  for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.g.V; v += gridDim.x * blockDim.x) {
    a.depth[v] = v == a.src ? 0 : -1;
    a.sigma[v] = v == a.src ? 1.0 : 0.0;
    a.dep[v] = 0.0;
  }
  if (blockIdx.x != 0) return;
  const int32_t t = threadIdx.x;
  if (t < 3) {
    a.cnt3[t] = t == 0;
    a.hub3[t] = 0;
  }
  if (t < 2) {
    a.bar[t] = 0;
    a.stats[t] = 0;
  }
  if (t == 0) {
    a.lev[0] = a.src;
    a.loff[0] = 0;
    a.loff[1] = 1;
    *a.stop = 0;
  }
}

// One edge pass over n queued vertices: the strategy, then the hubs it set aside.
// False when a barrier gave up.
template <int LB, class F>
__device__ __forceinline__ bool bc_pass(const BcArgs &a, const int32_t *q, int32_t n, const F &f, const DOut &out,
                                        int4 *smem, int32_t pass) {
  const HubList hub{a.hub_list, a.hub3 + pass % 3, a.hub_cap, a.hub_min, a.hub_slices};
  if (blockIdx.x == 0 && threadIdx.x == 0) a.hub3[(pass + 1) % 3] = 0;
  run_lb<LB>(a.g, Enum{q, nullptr, n}, n, f, out, smem, blockIdx.x, gridDim.x, hub);
  if (out.stage) stage_flush(out);
  if (!grid_barrier(a.bar, gridDim.x, a.err, a.timeout_ns)) return false;
  const int32_t chunks = *(volatile int32_t *)hub.cnt;
  if (chunks == 0) return true;
  lb_hubs(a.g, hub, chunks, f, out, blockIdx.x, gridDim.x);
  if (out.stage) stage_flush(out);
  return grid_barrier(a.bar, gridDim.x, a.err, a.timeout_ns);
}

template <int LB>
__global__ void __launch_bounds__(1024) k_bc_fused(BcArgs a) {
  extern __shared__ int4 smem[];
  __shared__ StageMem stage_mem;
  Stage &stage = stage_mem.s;
  if (threadIdx.x == 0) stage.init(kStageCap);
  __syncthreads();
  const int32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  LoopClock clk;
  clk.start(a.loop_limit_ns);
  int32_t level = 1, base = 0, n = 1, pass = 0;  // base, n: the queue of level - 1
  bool alive = true;
  for (;; ++level, ++pass) {
    if (stopped(a.stop, pass + 1)) {
      alive = false;
      break;
    }
    if (tid == 0) a.cnt3[(level + 1) % 3] = 0;
    DOut out{};
    out.mode = OUT_SPARSE;
    out.q = a.lev + base + n;
    out.cnt = a.cnt3 + level % 3;
    out.cap = a.g.V - base - n;  // a vertex is queued once
    out.err = a.err;
    out.stage = &stage;
    clk.tick(a.stop, pass + 1, a.err);
    const UBcFwd f{a.depth, a.sigma, level};
    if (!bc_pass<LB>(a, a.lev + base, n, f, out, smem, pass)) {
      alive = false;
      break;
    }
    base += n;
    n = min(*(volatile int32_t *)(a.cnt3 + level % 3), a.g.V - base);
    if (tid == 0) a.loff[level + 1] = base + n;  // read after the next barrier, or by this thread's block
    if (n == 0) break;
  }
  // levels 0 .. level - 1 hold vertices; level L = level - 1 is the deepest
  for (int32_t d = level - 1; alive && d >= 1; --d) {
    ++pass;
    if (stopped(a.stop, pass + 1)) {
      alive = false;
      break;
    }
    const int32_t b = __ldcg(a.loff + d), e = __ldcg(a.loff + d + 1);
    for (int32_t i = b + tid; i < e; i += nthreads) {
      const int32_t v = __ldcg(a.lev + i);
      a.dep[v] = __ldcg(a.dep + v) + 1.0 / __ldcg(a.sigma + v);
    }
    clk.tick(a.stop, pass + 1, a.err);
    if (!grid_barrier(a.bar, gridDim.x, a.err, a.timeout_ns)) {
      alive = false;
      break;
    }
    const UBcBwd f{a.depth, a.dep, d};
    alive = bc_pass<LB>(a, a.lev + b, e - b, f, DOut{}, smem, pass);
  }
  if (alive)
    for (int32_t v = tid; v < a.g.V; v += nthreads) {
      const double s = __ldcg(a.sigma + v);
      // the source's own 1 / sigma is added here: no pass reads it
      const double t = v == a.src ? __ldcg(a.dep + v) + 1.0 / s : __ldcg(a.dep + v);
      a.out[v] = s != 0.0 ? (float)((t - 1.0 / s) * s) : 0.0f;
    }
  if (tid == 0) a.stats[0] = level;
}

gg_status fused_bc(gg_graph *g, const gg_schedule *s, int32_t src, int32_t *depth, int32_t *lev, int32_t *loff,
                   double *sigma, double *dep64, float *out) {
  GG_TRY(ensure_hubs(g));
  const int cta = s->cta_size;
  const int lb = s->load_balancing;
  BcArgs a{};
  a.g = g->csr.view();
  a.g.nbuckets = 0;
  a.depth = depth;
  a.lev = lev;
  a.loff = loff;
  a.sigma = sigma;
  a.dep = dep64;
  a.out = out;
  a.cnt3 = g->d_misc + 40;
  a.hub3 = g->d_misc + 49;
  a.hub_list = static_cast<int32_t *>(g->hubs.p);
  a.hub_cap = hub_capacity(g);
  a.hub_min = kHubWidths * cta;
  a.hub_slices = slice_limit(g->max_degree);
  a.bar = g->d_bar;
  a.err = g->d_err;
  a.stats = g->d_misc + 44;
  a.stop = g->d_misc + 48;
  a.timeout_ns = barrier_timeout_ns();
  a.loop_limit_ns = loop_timeout_ns();
  a.src = src;
  const void *kernel = lb == GG_LB_TWCE ? (const void *)k_bc_fused<GG_LB_TWCE>
                       : lb == GG_LB_WM ? (const void *)k_bc_fused<GG_LB_WM>
                       : lb == GG_LB_CM ? (const void *)k_bc_fused<GG_LB_CM>
                                        : (const void *)k_bc_fused<GG_LB_VERTEX_BASED>;
  const size_t smem = lb == GG_LB_TWCE ? twce_smem_bytes(cta) : (lb == GG_LB_CM ? cm_smem_bytes(cta) : 0);
  int per_sm = 0;
  GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, cta, smem));
  if (per_sm < 1) return set_error(GG_ERR_UNSUPPORTED, "fused kernel does not fit on an SM");
  note_launch();
  k_bc_setup<<<std::max(1, std::min(ceil_div(a.g.V, 256), g->sm_count * 8)), 256, 0, g->stream>>>(a);
  GG_CUDA(cudaGetLastError());
  const int grid = loop_grid(g, per_sm, cta);
  void *args[] = {&a};
  GG_CUDA(cudaEventRecord(g->ev2, g->stream));
  note_launch();
  GG_CUDA(cudaLaunchCooperativeKernel(kernel, grid, cta, args, smem, g->stream));
  GG_CUDA(cudaEventRecord(g->ev3, g->stream));
  g->loop_timed = true;
  return GG_OK;
}

}  // namespace gg
