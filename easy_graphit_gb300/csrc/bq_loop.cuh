// The delta-stepping step machine over the bucket queue of bucket_queue.cuh,
// run by the persistent single-source loop (fused.cu, k_sssp_bq).
#pragma once

#include "bucket_queue.cuh"
#include "engine.h"
#include "lb.cuh"
#include "udf.cuh"

namespace gg {

// Runs one LB strategy over the n enumerated vertices; CTA `rank` of `nparts`
// takes every nparts-th virtual CTA (nparts = 1: one CTA does all of it).
template <int LB, class F>
__device__ __forceinline__ void run_lb(const DGraph &g, const Enum &en, int32_t n, const F &f,
                                       const DOut &out, int4 *smem, int32_t rank, int32_t nparts,
                                       const HubList &hub) {
  if (LB == GG_LB_VERTEX_BASED) {
    const int32_t nv = ceil_div(n, blockDim.x);
    for (int32_t v = rank; v < nv; v += nparts) lb_vertex(g, en, n, f, out, v);
  } else if (LB == GG_LB_WM) {
    const int32_t nv = ceil_div(n, blockDim.x >> 5);
    for (int32_t v = rank; v < nv; v += nparts) lb_wm(g, en, n, f, out, v);
  } else if (LB == GG_LB_TWCE) {
    lb_twce_all(g, en, n, f, out, rank, nparts, *reinterpret_cast<TwceSmem *>(smem), hub);
  } else {
    const int32_t nv = ceil_div(n, blockDim.x);
    for (int32_t v = rank; v < nv; v += nparts)
      lb_cm(g, en, n, f, out, v, *reinterpret_cast<CmSmem *>(smem));
  }
}

// ------------------------------------------------------ delta-stepping SSSP
// The sssp.cpp loop (apps/sssp.cpp:47-52) over the bucket queue of
// bucket_queue.cuh, as a sequence of steps, each one of
//   relax     the frontier with cutoff cur+delta (improvements below it queue
//             the vertex, the others park it on a far pile),
//   hubs      the chunks of long lists that the relax set aside (lb.cuh), by
//             all CTAs; part of that relax: same window, same output queue,
//   lo-min    exact minimum of the low pile's live entries,
//   lo-split  window entries to the frontier, the rest to the next low pile
//             (a window reaching past the horizon splits the high pile too),
//   hi-min / hi-split  the same over the high pile when the low pile holds
//             nothing live (a refill, which also sets the next horizon).
// Between steps the CTAs that run them synchronise (a grid barrier, or
// __syncthreads when one CTA runs them).  Frontier counts and minima rotate
// through three slots: a step clears the slot two steps ahead, whose readers
// finished before the previous synchronisation.
enum : int32_t { BQ_RELAX = 0, BQ_LOMIN = 1, BQ_LOSPLIT = 2, BQ_HIMIN = 3, BQ_HISPLIT = 4, BQ_DONE = 5, BQ_HUBS = 6 };
constexpr uint64_t kSoloSliceNs = 1000000;

struct BqArgs {
  DGraph g;
  int32_t *q0, *q1;  // frontier queues
  int64_t qcap;
  int32_t *dist;
  BqBuffers b;       // stamps, piles, control words
  uint32_t *bar;
  int32_t *err;
  uint64_t timeout_ns, loop_limit_ns;
  int32_t delta;
  int32_t solo_max;     // largest relax step (frontier entries) CTA 0 runs alone
  int32_t solo_pile_max;  // largest pile step (pile entries) CTA 0 runs alone
  int32_t fill_target;  // low-pile entries a refill aims for
  int32_t width0;       // first horizon width, in buckets
  int32_t *hub_list;    // hub chunks (HubList); their counts are control words
  int32_t hub_cap, hub_min, hub_slices;
  int32_t stage_cap, stage_at;  // the three stages: entries each, where they start in shared memory
  int32_t alone_max;    // frontier entries up to which hubs' threads queue near vertices unclaimed
  int32_t near_cap;     // frontier entries a mesh session takes: at most kMeshNear
  int32_t mesh;         // largest out-degree <= 32: one-CTA sessions run in shared memory (bq_mesh_session)
};

// Loop state, the same in every CTA: every decision is taken from control
// words read after a barrier.
struct BqLoop {
  int32_t it;     // step number (slot rotation)
  int32_t in;     // frontier queue read by this step
  int32_t cur;    // window start
  int32_t g, gh;  // low / high pile generations
  int32_t hz;     // horizon
  int32_t k;      // horizon width in buckets
  int32_t phase;  // 0: normal, 1: after a lo-min, 2: after a hi-min
  int32_t relax, adv;
  int32_t hub;    // 1: the last step was a relax, whose hub chunks may be pending
};
constexpr int kBqLoopInts = 11;
static_assert(sizeof(BqLoop) == kBqLoopInts * sizeof(int32_t), "BqLoop is published as ints");

struct BqStep {
  int32_t kind, work, m;
};

// Small enough for CTA 0 alone: frontier entries of a relax, pile entries of
// the other steps (one load and a compare each).
__device__ __forceinline__ bool bq_small(const BqStep &st, const BqArgs &a) {
  return st.kind != BQ_HUBS && st.work <= (st.kind == BQ_RELAX ? a.solo_max : a.solo_pile_max);
}

// The next step (pure: every CTA computes the same one).
__device__ __forceinline__ BqStep bq_decide(const BqLoop &s, const int32_t *ctl, int32_t delta) {
  const volatile int32_t *c = ctl;
  const int32_t prev = (s.it + 2) % 3;
  if (s.hub) {
    const int32_t n = c[BQ_NEAR + prev];  // loaded with the hub count: one round trip
    const int32_t nh = c[BQ_HUB + (s.relax + 2) % 3];
    if (nh > 0) return BqStep{BQ_HUBS, nh, 0};
    if (n > 0) return BqStep{BQ_RELAX, n, 0};
  }
  if (s.phase == 1) {
    const int32_t m = c[BQ_MIN + prev];
    if (m != INT_MAX) {
      const bool cross = bq_clamp((int64_t)m + delta) > s.hz;  // the window reaches the high pile
      return BqStep{BQ_LOSPLIT, c[BQ_LO + (s.g & 1)] + (cross ? c[BQ_HI + (s.gh & 1)] : 0), m};
    }
    const int32_t nh = c[BQ_HI + (s.gh & 1)];
    return nh > 0 ? BqStep{BQ_HIMIN, nh, 0} : BqStep{BQ_DONE, 0, 0};
  }
  if (s.phase == 2) {
    const int32_t m = c[BQ_MIN + prev];
    return m != INT_MAX ? BqStep{BQ_HISPLIT, c[BQ_HI + (s.gh & 1)], m} : BqStep{BQ_DONE, 0, 0};
  }
  const int32_t n = c[BQ_NEAR + prev];
  if (n > 0) return BqStep{BQ_RELAX, n, 0};
  const int32_t nl = c[BQ_LO + (s.g & 1)];
  if (nl > 0) return BqStep{BQ_LOMIN, nl, 0};
  const int32_t nh = c[BQ_HI + (s.gh & 1)];
  return nh > 0 ? BqStep{BQ_HIMIN, nh, 0} : BqStep{BQ_DONE, 0, 0};
}

// One step, CTA `rank` of `nparts` taking its share.
// `ctl` holds the control words: global memory in grid mode, CTA 0's shared
// copy in a one-CTA session.  `stages`: three in shared memory, empty.
template <int LB>
__device__ __forceinline__ void bq_step(BqLoop &s, const BqArgs &a, const BqStep &st, int32_t *ctl,
                                        int32_t rank, int32_t nparts, int4 *smem, int32_t *red, Stage *const *stages) {
  const bool lead = rank == 0 && threadIdx.x == 0;
  if (lead) {
    ctl[BQ_NEAR + (s.it + 1) % 3] = 0;
    ctl[BQ_MIN + (s.it + 1) % 3] = INT_MAX;
  }
  const int32_t U = bq_clamp((int64_t)s.cur + a.delta);  // cutoff of the current window
  int32_t *qin = s.in ? a.q1 : a.q0, *qout = s.in ? a.q0 : a.q1;
  DOut front{};
  front.mode = OUT_SPARSE;
  front.q = qout;
  front.cnt = ctl + BQ_NEAR + s.it % 3;
  front.cap = a.qcap;
  front.err = a.err;
  // appends are staged where many CTAs share the counts; one CTA has them in
  // shared memory anyway
  const bool staged = nparts > 1;
  if (staged) front.stage = stages[0];
  Stage *st_lo = staged ? stages[1] : nullptr, *st_hi = staged ? stages[2] : nullptr;
  const int32_t lo_next = (s.g + 1) & 1;
  if (st.kind == BQ_RELAX || st.kind == BQ_HUBS) {
    const bool hubs = st.kind == BQ_HUBS;
    // a hub step finishes the relax before it: into that step's queue and count
    if (hubs) {
      front.q = qin;
      front.cnt = ctl + BQ_NEAR + (s.it + 2) % 3;
    }
    const uint32_t near_tag = bq_near_tag(s.relax - (hubs ? 1 : 0));
    const DFar far{a.b.stamp, a.b.lo[s.g & 1], ctl + BQ_LO + (s.g & 1), a.b.hi[s.gh & 1],
                   ctl + BQ_HI + (s.gh & 1), bq_lo_tag(s.g), bq_hi_tag(s.gh), s.hz, a.b.V, a.err, st_lo, st_hi,
                   near_tag, !hubs && st.work <= a.alone_max ? 0u : near_tag};
    const EdgeF<USssp, false> f{USssp{a.dist, U, far}, DIn{IN_ALL, nullptr, nullptr},
                                DIn{IN_ALL, nullptr, nullptr}, false};
    if (hubs) {
      const HubList hub{a.hub_list, nullptr, a.hub_cap, 0};
      lb_hubs(a.g, hub, st.work, f, front, rank, nparts);
      if (staged) {
        stage_flush(front);
        far.flush();
      }
      s.hub = 0;
      return;
    }
    if (lead) ctl[BQ_HUB + (s.relax + 1) % 3] = 0;
    const HubList hub{a.hub_list, ctl + BQ_HUB + s.relax % 3, a.hub_cap, a.hub_min, a.hub_slices};
    const int32_t n = (int64_t)st.work > a.qcap ? (int32_t)a.qcap : st.work;  // past qcap only after a flagged overflow
    run_lb<LB>(a.g, Enum{qin, nullptr, n}, n, f, front, smem, rank, nparts, hub);
    if (staged) {
      stage_flush(front);
      far.flush();
    }
    s.in ^= 1;
    s.relax++;
    s.phase = 0;
    s.hub = 1;
    s.it++;
    return;
  }
  s.hub = 0;
  switch (st.kind) {
    case BQ_LOMIN:
      if (s.phase == 0) s.adv++;
      if (lead) {
        ctl[BQ_LO + lo_next] = 0;
        ctl[BQ_HI + ((s.gh + 1) & 1)] = 0;
        ctl[BQ_FILL + ((s.gh + 1) & 1)] = 0;
      }
      bq_pile_min(a.b.lo[s.g & 1], min(st.work, a.b.V), a.dist, U, ctl + BQ_MIN + s.it % 3, rank, nparts, red);
      s.phase = 1;
      break;
    case BQ_LOSPLIT: {
      const int32_t win = bq_clamp((int64_t)st.m + a.delta);
      const int32_t n_lo = min(*(volatile int32_t *)(ctl + BQ_LO + (s.g & 1)), a.b.V);
      if (win <= s.hz) {
        const BqSplitOut o{a.b.stamp, a.b.lo[lo_next], ctl + BQ_LO + lo_next, bq_lo_tag(s.g + 1),
                           nullptr, nullptr, 0, INT_MAX, nullptr, a.b.V, false, st_lo, st_hi};
        bq_pile_split(a.b.lo[s.g & 1], n_lo, a.dist, U, win, front, o, a.err, rank, nparts);
        o.flush(a.err);
      } else {
        // the window reaches past the horizon: split both piles under a new one
        const int32_t hi_next = (s.gh + 1) & 1;
        s.k = bq_adapt_width(s.k, *(volatile int32_t *)(ctl + BQ_FILL + (s.gh & 1)), a.fill_target);
        const int32_t hz = bq_clamp((int64_t)st.m + (int64_t)s.k * a.delta);
        BqSplitOut o{a.b.stamp, a.b.lo[lo_next], ctl + BQ_LO + lo_next, bq_lo_tag(s.g + 1),
                     a.b.hi[hi_next], ctl + BQ_HI + hi_next, bq_hi_tag(s.gh + 1), hz, nullptr, a.b.V, true,
                     st_lo, st_hi};
        bq_pile_split(a.b.lo[s.g & 1], n_lo, a.dist, U, win, front, o, a.err, rank, nparts);
        o.fill = ctl + BQ_FILL + hi_next;
        bq_pile_split(a.b.hi[s.gh & 1], min(*(volatile int32_t *)(ctl + BQ_HI + (s.gh & 1)), a.b.V), a.dist, U,
                      win, front, o, a.err, rank, nparts);
        o.flush(a.err);
        s.hz = hz;
        s.gh++;
      }
      s.cur = st.m;
      s.g++;
      s.in ^= 1;
      s.phase = 0;
      break;
    }
    case BQ_HIMIN: {
      if (s.phase == 0) s.adv++;
      const int32_t hi_next = (s.gh + 1) & 1;
      if (lead) {
        ctl[BQ_LO + lo_next] = 0;
        ctl[BQ_HI + hi_next] = 0;
        ctl[BQ_FILL + hi_next] = 0;
      }
      bq_pile_min(a.b.hi[s.gh & 1], min(st.work, a.b.V), a.dist, U, ctl + BQ_MIN + s.it % 3, rank, nparts, red);
      s.phase = 2;
      break;
    }
    case BQ_HISPLIT: {
      const int32_t hi_next = (s.gh + 1) & 1;
      s.k = bq_adapt_width(s.k, *(volatile int32_t *)(ctl + BQ_FILL + (s.gh & 1)), a.fill_target);
      const int32_t hz = bq_clamp((int64_t)st.m + (int64_t)s.k * a.delta);
      const BqSplitOut o{a.b.stamp, a.b.lo[lo_next], ctl + BQ_LO + lo_next, bq_lo_tag(s.g + 1),
                         a.b.hi[hi_next], ctl + BQ_HI + hi_next, bq_hi_tag(s.gh + 1), hz,
                         ctl + BQ_FILL + hi_next, a.b.V, false, st_lo, st_hi};
      bq_pile_split(a.b.hi[s.gh & 1], min(st.work, a.b.V), a.dist, U, bq_clamp((int64_t)st.m + a.delta), front,
                    o, a.err, rank, nparts);
      o.flush(a.err);
      s.cur = st.m;
      s.hz = hz;
      s.g++;
      s.gh++;
      s.in ^= 1;
      s.phase = 0;
      break;
    }
    default:
      break;
  }
  if (staged) stage_flush(front);
  s.it++;
}

// ---------------------------------------------------------- mesh sessions
// CTA 0's one-CTA mode on a graph of short lists (largest out-degree at most
// kMeshMaxDegree): the same rule and the same counts, with the frontier and the
// low pile in shared memory.  A bucket is bound by its dependent L2 round trips.
// In bq_step's form an advance is two steps (minimum, split) and a relax reads
// queue, offsets, edges, targets and answers of the stamp claims one after the
// other, 15 to 20 trips and as many barriers a bucket; here
//  * an advance reads the pile's priorities once (one trip), reduces them and
//    splits the pile from shared memory;
//  * a relax has two trips: a vertex's edges, then the targets' distances,
//    stamps and edge ranges together; what it queues carries priority and edge
//    range.  Four lanes share a vertex, an edge each;
//  * a park decides by the stamp it read and raises the stamp without waiting
//    for the answer: a vertex parked twice in one round may be listed twice,
//    which the claims at the end of the session undo: the piles and the queue
//    in global memory get a vertex once.
// An entry that an advance takes or finds settled can never be parked again
// (its distance stays below every later cutoff), so a session needs one mark.
// 700 x 501 grid, delta 128 (1,344 buckets, 3 relaxes each): 24-29 -> 12.9 ms;
// a session's relax of 250 vertices takes 5,000 cycles, of 8 2,300, an advance
// over a pile of 900 3,900 (bq_step: 7,300 a step).
constexpr int32_t kMeshMaxDegree = 32;
constexpr int32_t kMeshNear = 1024;  // frontier entries a session holds
constexpr int32_t kMeshLow = 2048;   // low-pile entries
constexpr int32_t kMeshHigh = 1024;  // high parks buffered between flushes
struct BqMeshSmem {
  int4 near_[2][kMeshNear];  // v, priority, first edge, end edge
  int4 lo[2][kMeshLow];      // v, priority at the last scan, first edge, end edge
  int32_t hi[kMeshHigh];
  int32_t n_near[2], n_lo[2], n_hi, spill, full, min3[3], quit;
};

// Places of a warp's appends to up to three lists, `to` the list of this lane's
// entry (-1: none) and `cnt` on lane i list i's count: one shared-memory atomic
// a list.  The whole warp calls it.
__device__ __forceinline__ int32_t mesh_places(int32_t to, int32_t *cnt) {
  const int32_t lane = threadIdx.x & 31;
  const uint32_t m0 = __ballot_sync(0xffffffffu, to == 0), m1 = __ballot_sync(0xffffffffu, to == 1),
                 m2 = __ballot_sync(0xffffffffu, to == 2);
  if (!(m0 | m1 | m2)) return 0;
  const int32_t own = __popc(lane == 0 ? m0 : (lane == 1 ? m1 : m2));
  int32_t base = 0;
  if (lane < 3 && own) base = atomicAdd(cnt, own);
  base = __shfl_sync(0xffffffffu, base, to & 3);
  return base + __popc((to == 0 ? m0 : (to == 1 ? m1 : m2)) & ((1u << lane) - 1));
}

// Buffered high parks to the high pile of generation gh; the whole CTA calls it
// between barriers.
__device__ __forceinline__ void mesh_flush_high(const BqLoop &s, const BqArgs &a, int32_t *sctl, BqMeshSmem &m) {
  const int32_t n = min(m.n_hi, kMeshHigh);
  const uint32_t tag = bq_hi_tag(s.gh);
  for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const int32_t v = m.hi[i];
    if (stamp_claim(a.b.stamp, v, tag) >= tag) continue;  // listed, or since parked lower
    const int32_t pos = agg_inc(sctl + BQ_HI + (s.gh & 1));
    if (pos < a.b.V)
      a.b.hi[s.gh & 1][pos] = v;
    else
      atomicOr(a.err, DEV_ERR_OVERFLOW);
  }
  __syncthreads();
  if (threadIdx.x == 0) m.n_hi = 0;
}

// A window vertex to the frontier queue in global memory, once a session: `step`
// is the relax step that will read the queue.  A session spills in its last round
// only, so that step is the same for all of its spills.
__device__ __forceinline__ void mesh_spill(const BqArgs &a, BqMeshSmem &m, int32_t step, int32_t *q, int32_t v) {
  const uint32_t tag = bq_spill_tag(step);
  if (stamp_claim(a.b.stamp, v, tag) >= tag) return;
  const int32_t qp = atomicAdd(&m.spill, 1);
  if (qp < a.qcap)
    q[qp] = v;
  else
    atomicOr(a.err, DEV_ERR_OVERFLOW);
}

// Relaxes, at the priorities they were listed with (a vertex lowered since is
// listed again; reading its distance first costs the trip more than the rare
// repeat), the n vertices of near_[in]: improvements below U to near_[in ^ 1]
// (count *n_out, the queue q when that is full), the others parked.  Four lanes
// share a vertex, an edge each, J vertices of a lane in flight.
template <int J>
__device__ __forceinline__ void mesh_relax_pass(const BqLoop &s, const BqArgs &a, int32_t *sctl, BqMeshSmem &m,
                                                int32_t n, int32_t in, int32_t L, int32_t U,
                                                int32_t *n_out, int32_t *q) {
  const int32_t per = blockDim.x >> 2, lane = threadIdx.x & 31, lo_next = (s.g + 1) & 1;
  const uint32_t lo_tag = bq_lo_tag(s.g), lo_mark = bq_lo_mark(s.g), next_tag = bq_lo_tag(s.g + 1);
  const uint32_t hi_mark = bq_hi_mark(s.gh), hi_tag = bq_hi_tag(s.gh);
  uint32_t *const stamps = reinterpret_cast<uint32_t *>(a.b.stamp);
  int32_t *cnt = lane == 0 ? n_out : (lane == 1 ? &m.n_lo[L] : &m.n_hi);
  // a warp without a vertex leaves at once: in a round of a few vertices the
  // others' empty instructions would cost more than the loads
  for (int32_t w0 = (threadIdx.x & ~31) >> 2; w0 < n; w0 += J * per) {
    bool more = true;
    for (int32_t hop = threadIdx.x & 3; more; hop += 4) {
      int32_t d[J], np[J], prev[J], db[J], de[J];
      uint32_t st[J];
      more = false;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int32_t i = w0 + (lane >> 2) + j * per;
        const int4 x = i < n ? m.near_[in][i] : make_int4(0, 0, 0, 0);
        const int32_t k = x.z + hop;
        const bool ok = k < x.w;
        d[j] = ok ? __ldg(a.g.dst + k) : -1;
        np[j] = ok ? x.y + __ldg(a.g.w + k) : INT_MAX;
        more |= k + 4 < x.w;
      }
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const bool ok = d[j] >= 0;
        prev[j] = ok ? __ldcg(a.dist + d[j]) : INT_MIN;
        st[j] = ok ? __ldcg(stamps + d[j]) : 0u;
        db[j] = ok ? __ldg(a.g.off + d[j]) : 0;
        de[j] = ok ? __ldg(a.g.off + d[j] + 1) : 0;
      }
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int32_t v = d[j], p = np[j];
        int32_t to = -1;  // 0 frontier, 1 low pile, 2 high pile
        if (p < prev[j]) {
          asm volatile("red.relaxed.gpu.global.min.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(a.dist + v)), "r"(p)
                       : "memory");
          if (p < U)
            to = 0;
          else if (p < s.hz)
            to = st[j] >= lo_tag ? -1 : 1;
          else
            to = st[j] >= hi_mark ? -1 : 2;
        }
        const int32_t pos = mesh_places(to, cnt);
        if (to == 0) {
          if (pos < a.near_cap) {
            m.near_[in ^ 1][pos] = make_int4(v, p, db[j], de[j]);
          } else {
            m.full = 1;
            mesh_spill(a, m, s.relax + 1, q, v);
          }
        } else if (to == 1) {
          if (pos < kMeshLow) {
            stamp_raise(a.b.stamp, v, lo_mark);
            m.lo[L][pos] = make_int4(v, p, db[j], de[j]);
          } else {
            m.full = 1;
            if (stamp_claim(a.b.stamp, v, next_tag) < next_tag) {
              const int32_t gp = atomicAdd(sctl + BQ_LO + lo_next, 1);
              if (gp < a.b.V)
                a.b.lo[lo_next][gp] = v;
              else
                atomicOr(a.err, DEV_ERR_OVERFLOW);
            }
          }
        } else if (to == 2) {
          if (pos < kMeshHigh) {
            stamp_raise(a.b.stamp, v, hi_mark);
            m.hi[pos] = v;
          } else if (stamp_claim(a.b.stamp, v, hi_tag) < hi_tag) {
            const int32_t gp = atomicAdd(sctl + BQ_HI + (s.gh & 1), 1);
            if (gp < a.b.V)
              a.b.hi[s.gh & 1][gp] = v;
            else
              atomicOr(a.err, DEV_ERR_OVERFLOW);
          }
        }
      }
      more = __any_sync(0xffffffffu, more);
    }
  }
}

// Runs relaxes and advances while they fit.  On return the loop state and control
// words are as after a bq_step, ready for bq_decide.
__device__ __forceinline__ void bq_mesh_session(BqLoop &s, const BqArgs &a, int32_t *sctl, BqMeshSmem &m,
                                                int32_t n, uint64_t t0) {
  const uint32_t next_tag = bq_lo_tag(s.g + 1);
  const int32_t lo_next = (s.g + 1) & 1, T = blockDim.x, lane = threadIdx.x & 31;
  int32_t *const q = s.in ? a.q1 : a.q0;
  int32_t nl = sctl[BQ_LO + (s.g & 1)];
  for (int32_t i = threadIdx.x; i < n; i += T) {
    const int32_t v = __ldcg(q + i);
    m.near_[0][i] = make_int4(v, __ldcg(a.dist + v), __ldg(a.g.off + v), __ldg(a.g.off + v + 1));
  }
  for (int32_t i = threadIdx.x; i < nl; i += T) {
    const int32_t v = __ldcg(a.b.lo[s.g & 1] + i);
    m.lo[0][i] = make_int4(v, 0, __ldg(a.g.off + v), __ldg(a.g.off + v + 1));
  }
  __syncthreads();  // nl is read by every thread before it changes
  if (threadIdx.x == 0) {
    m.n_near[0] = m.n_near[1] = 0;
    m.n_lo[0] = nl;
    m.n_hi = 0;
    m.spill = m.full = m.quit = 0;
    m.min3[0] = m.min3[1] = m.min3[2] = INT_MAX;
    sctl[BQ_LO + lo_next] = 0;  // low parks that do not fit, then the write-back
  }
  int32_t in = 0, L = 0, adv = 0, cross = INT_MAX;
  for (int32_t rounds = 1;; ++rounds) {
    __syncthreads();
    // The session's time slice, and overflows, on a count of all rounds; read at the
    // end of this one, behind its barriers.  Tested in relaxes alone, on the same
    // count, it never came up where relaxes and advances take turns (a line of unit
    // weights at delta 1: every 16th round an advance), and only the horizon, seconds
    // away, ended the session.  64 rounds are 0.1 to 0.5 ms.
    if (threadIdx.x == 0 && (rounds & 63) == 0)
      m.quit = globaltimer_ns() - t0 > kSoloSliceNs || (*(volatile int32_t *)a.err & DEV_ERR_OVERFLOW) != 0;
    const int32_t U = bq_clamp((int64_t)s.cur + a.delta);
    if (n > 0) {
      // ---- relax: near_[in] -> near_[in ^ 1], lo[L], hi
      int32_t *n_out = &m.n_near[in ^ 1];
      // a second vertex per lane only where the frontier has that many
      if (n <= T >> 2)
        mesh_relax_pass<1>(s, a, sctl, m, n, in, L, U, n_out, q);
      else
        mesh_relax_pass<2>(s, a, sctl, m, n, in, L, U, n_out, q);
      s.relax++;
      __syncthreads();
      in ^= 1;
      n = min(m.n_near[in], a.near_cap);
      const bool leave = m.full || m.quit;
      const bool flush = m.n_hi > kMeshHigh / 2;
      __syncthreads();
      if (threadIdx.x == 0) m.n_near[in ^ 1] = 0;
      if (flush) mesh_flush_high(s, a, sctl, m);
      if (leave) break;
    } else {
      // ---- advance: the exact minimum of the live entries, then the split
      nl = min(m.n_lo[L], kMeshLow);
      int32_t mn = INT_MAX;
      constexpr int kIn = 4;  // priorities a thread reads at once
      for (int32_t i0 = threadIdx.x; i0 < nl; i0 += kIn * T) {
        int32_t p[kIn];
#pragma unroll
        for (int j = 0; j < kIn; ++j) p[j] = i0 + j * T < nl ? __ldcg(a.dist + m.lo[L][i0 + j * T].x) : -1;
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
          if (i0 + j * T < nl) m.lo[L][i0 + j * T].y = p[j];
          if (p[j] >= U) mn = min(mn, p[j]);
        }
      }
      mn = __reduce_min_sync(0xffffffffu, mn);
      if ((threadIdx.x & 31) == 0 && mn != INT_MAX) atomicMin(&m.min3[adv % 3], mn);
      __syncthreads();
      mn = m.min3[adv % 3];
      if (threadIdx.x == 0) {
        m.min3[(adv + 1) % 3] = INT_MAX;
        m.n_lo[L ^ 1] = 0;
        if (mn == INT_MAX) m.n_lo[L] = 0;  // nothing live below the horizon: a refill is next
      }
      __syncthreads();
      if (mn == INT_MAX) break;
      if (bq_clamp((int64_t)mn + a.delta) > s.hz) {  // the window reaches the high pile: bq_step's split
        cross = mn;
        break;
      }
      const int32_t win = bq_clamp((int64_t)mn + a.delta);
      int32_t *cnt = lane == 0 ? &m.n_near[in] : &m.n_lo[L ^ 1];
      for (int32_t i0 = 0; i0 < nl; i0 += T) {
        const int32_t i = i0 + threadIdx.x;
        const int4 x = i < nl ? m.lo[L][i] : make_int4(0, -1, 0, 0);
        const int32_t to = x.y < U ? -1 : (x.y < win ? 0 : 1);  // below U: settled since it was parked
        const int32_t pos = mesh_places(to, cnt);
        if (to == 1) m.lo[L ^ 1][pos] = x;
        if (to == 0) {
          if (pos < a.near_cap) {
            m.near_[in][pos] = x;
          } else {
            m.full = 1;
            mesh_spill(a, m, s.relax, q, x.x);
          }
        }
      }
      L ^= 1;
      s.cur = mn;
      s.adv++;
      adv++;
      __syncthreads();
      n = min(m.n_near[in], a.near_cap);
      if (m.full || m.quit) break;
    }
  }
  // ---- back to the queues and piles in global memory, a vertex once per pile
  __syncthreads();
  mesh_flush_high(s, a, sctl, m);
  nl = min(m.n_lo[L], kMeshLow);
  for (int32_t i = threadIdx.x; i < nl; i += T) {
    const int32_t v = m.lo[L][i].x;
    if (stamp_claim(a.b.stamp, v, next_tag) >= next_tag) continue;
    const int32_t pos = agg_inc(sctl + BQ_LO + lo_next);
    if (pos < a.b.V)
      a.b.lo[lo_next][pos] = v;
    else
      atomicOr(a.err, DEV_ERR_OVERFLOW);
  }
  for (int32_t i = threadIdx.x; i < n; i += T) mesh_spill(a, m, s.relax, q, m.near_[in][i].x);
  __syncthreads();
  n = (int32_t)min((int64_t)m.spill, a.qcap);
  s.g++;
  s.phase = 0;
  s.hub = 0;
  if (cross != INT_MAX) {  // as after a lo-min that found it
    s.phase = 1;
    s.adv++;
  }
  if (threadIdx.x == 0) {
    sctl[BQ_NEAR + (s.it + 2) % 3] = n;
    sctl[BQ_NEAR + s.it % 3] = sctl[BQ_NEAR + (s.it + 1) % 3] = 0;
    sctl[BQ_MIN + (s.it + 2) % 3] = cross;
    sctl[BQ_MIN + s.it % 3] = sctl[BQ_MIN + (s.it + 1) % 3] = INT_MAX;
    sctl[BQ_HUB] = sctl[BQ_HUB + 1] = sctl[BQ_HUB + 2] = 0;
    if (cross != INT_MAX) {  // what a lo-min clears for the next generations
      sctl[BQ_LO + ((s.g + 1) & 1)] = 0;
      sctl[BQ_HI + ((s.gh + 1) & 1)] = 0;
      sctl[BQ_FILL + ((s.gh + 1) & 1)] = 0;
    }
  }
  __syncthreads();
}

}  // namespace gg
