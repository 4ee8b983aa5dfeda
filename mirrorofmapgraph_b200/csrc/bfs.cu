// bfs.cu -- breadth-first search (struct bfs, Algorithms/BFS/bfs.h:28-262).
//
// Per level one of two kernels does the work and the last CTA to finish closes
// the level (swap queues, pick the next direction, stop or continue):
//
//  push (top-down)  input: vertex queue. Each CTA takes a tile of up to 256 frontier
//                   vertices and bins them by out-degree: >= CTA_TH edges are
//                   expanded by the whole CTA, >= 32 by one warp, the rest by a
//                   block-wide scan over the remaining degrees (thread-level
//                   bin), so every edge load is coalesced. A neighbour is claimed
//                   with atomicOr on a visited bitmap (1 bit per vertex); the
//                   winner writes depth = level + 1 and appends itself to the
//                   output queue with a warp-aggregated atomic.
//                   This replaces expand_atomic + contract_atomic
//                   (GASengine/vertex_centric/expand_atomic/cta.cuh:268-759,
//                   contract_atomic/cta.cuh:203-612): no edge-sized frontier is
//                   ever materialised, the dedup is exact, and BFS's contract
//                   (label := iteration + 1, bfs.h:229-255) is fused in.
//  pull (bottom-up) every unvisited vertex scans its in-edges for a parent whose
//                   depth equals the current level and stops at the first hit.
//                   A warp owns 32 consecutive vertices, i.e. one bitmap word,
//                   so visited words are updated without atomics. An in-neighbour
//                   of an unvisited vertex that is visited at all was reached in
//                   the last level, so the test is one bit of the bitmap as the
//                   level found it (the level writes a second one).
//
// The direction switch (Beamer's heuristic: go bottom-up when the frontier's
// out-edges exceed 1/14 of the unexplored edges, back when the frontier drops
// below n/24) is evaluated on the device.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "engine.cuh"
#include "expand.cuh"
#define MG_PRB_NO_PLAN_KERNELS
#include "pr_binned.cuh"

namespace mg {

constexpr int BFS_NT = 256;
constexpr int BFS_CTA_TH = 512;   // out-degree at or above which a CTA expands the vertex
constexpr int PULL_SERIAL = 8;    // in-edges a lane scans alone before others help
constexpr int PULL_QUAD = 256;    // in-edges four lanes scan before the whole warp does
// Beamer's direction rule (mg_tuning.bfs_alpha / bfs_beta, defaults 14 and 24):
// pull when the frontier's out-edges exceed the unvisited vertices' out-edges /
// alpha, back to push when the frontier holds fewer than n / beta vertices. AUTO
// runs top-down only on graphs of mean out-degree <= bfs_sparse_degree (8).

struct BfsArgs {
  const int32_t *ro, *ci;  // out-edges (CSR)
  const int32_t *co, *ri;  // in-edges (CSC; the CSR itself for symmetric graphs)
  int32_t *label;
  uint32_t *vis, *vis2;  // visited bitmaps, current by DevCtl::vsel (vis2 nullptr: only vis, updated in place)
  int32_t *q0, *q1;
  int32_t qcap;
  int32_t mode;      // MG_DIR_*
  int32_t can_pull;  // in-edges available and traversal direction allows it
  int32_t both;      // directed == 0 on a non-symmetric graph: expand CSR and CSC
  int64_t n;
  int64_t m_total;
  int32_t *big_v;  // grid-strided bin of the push direction (BIG_CAP entries)
  DevCtl *ctl;
  cudaGraphConditionalHandle h;
  int32_t use_cond;
  uint32_t bar_extra;            // test hook (mg_debug_barrier_skew): a barrier that cannot complete
  unsigned long long bar_limit;  // barrier polls before MG_ERR_TIMEOUT
  // tuned thresholds (mg_tuning): CTA-bin and grid-bin out-degrees, the warp-bin
  // deferral rule, the persistent kernel's frontier limits, Beamer's constants
  int32_t cta_th, grid_th, defer_warp;
  int32_t persist_max;
  int64_t persist_edges;
  int64_t alpha, beta;
};

// The graph's tuned BFS thresholds into the kernel arguments.
inline void bfs_tuning(BfsArgs &a, const mg_tuning &t) {
  a.cta_th = t.bfs_cta_th;
  a.grid_th = t.bfs_grid_th;
  a.defer_warp = t.bfs_defer_warp;
  a.persist_max = t.bfs_persist_max;
  a.persist_edges = t.bfs_persist_edges;
  a.alpha = t.bfs_alpha;
  a.beta = t.bfs_beta;
}

// Whether the BFS thresholds are the defaults.
inline bool bfs_tuning_default(const mg_tuning &t) {
  const mg_tuning d = tuning_defaults();
  return t.bfs_cta_th == d.bfs_cta_th && t.bfs_grid_th == d.bfs_grid_th && t.bfs_defer_warp == d.bfs_defer_warp &&
         t.bfs_persist_max == d.bfs_persist_max && t.bfs_persist_edges == d.bfs_persist_edges &&
         t.bfs_alpha == d.bfs_alpha && t.bfs_beta == d.bfs_beta && t.bfs_sparse_degree == d.bfs_sparse_degree &&
         t.bfs_ctas_per_sm == d.bfs_ctas_per_sm && t.bfs_tail_max == d.bfs_tail_max &&
         t.bfs_tail_edges == d.bfs_tail_edges;
}

__device__ void bfs_level_end(const BfsArgs &a) {
  DevCtl *c = a.ctl;
  const int cur = vload(&c->cur);
  const int32_t nf = vload(&c->qlen[cur ^ 1]);
  const int64_t mf = vload(&c->mf_next);
  const int64_t vdeg = vload(&c->visited_deg) + mf;
  const int lvl = vload(&c->level) + 1;
  trace_level(c, lvl - 1, vload(&c->dir) == 1 ? MG_DIR_PULL : MG_DIR_PUSH, vload(&c->qlen[cur]),
              vload(&c->mf_front), 0.0);
  if (vload(&c->dir) == 1 && a.vis2) c->vsel ^= 1;  // the level wrote the other bitmap
  c->visited_deg = vdeg;
  c->mf_front = mf;
  c->level = lvl;
  c->qlen[cur] = 0;
  c->cur = cur ^ 1;
  c->mf_next = 0;
  c->blocks_done = 0;
  c->big_len = 0;
  // the persistent kernel's per-level counters start from zero when it next runs
  for (int k = 0; k < 3; k++) {
    c->pq[k] = 0;
    c->pm[k] = 0;
    c->pb[k] = 0;
  }
  const bool over = vload(&c->overflow) != 0;
  const bool done = nf == 0 || lvl >= c->iter_cap || over;
  int dir = vload(&c->dir);
  if (!done) {
    if (a.mode == MG_DIR_PULL) {
      dir = a.can_pull ? 1 : 0;
    } else if (a.mode == MG_DIR_PUSH || !a.can_pull) {
      dir = 0;
    } else if (dir == 0) {
      if (mf > (a.m_total - vdeg) / a.alpha) dir = 1;
    } else {
      if ((int64_t)nf * a.beta < a.n) dir = 0;
    }
  }
  if (dir == 1 && !done) c->levels_pull += 1;
  c->dir = dir;
  c->nf_next = nf;
  if (over) c->status = MG_ERR_QUEUE_OVERFLOW;
  __threadfence();
  c->done = done ? 1 : 0;
  loop_signal(a.ctl, a.h, a.use_cond, done);
}

// What a level kernel reads from the control block: by one thread per block, since
// every warp of the grid reading one L2 sector queues for microseconds (more than an
// empty kernel takes otherwise).
struct BfsEnter {
  int32_t skip, cur, nin, level;
  int64_t mf;
  uint32_t *vis, *vis_out;  // the visited bitmap as the level found it, and the one it writes
};

// Early exit shared by the level kernels: true if the run is over (then it makes sure
// the loop stops) or the level goes the other way. Every thread of the block calls it.
__device__ __forceinline__ bool bfs_skip(const BfsArgs &a, int want_dir, BfsEnter &en) {
  DevCtl *c = a.ctl;
  if (threadIdx.x == 0) {
    const int32_t done = vload(&c->done), dir = vload(&c->dir), cur = vload(&c->cur), vsel = vload(&c->vsel);
    en.level = vload(&c->level);
    const int32_t q0 = vload(&c->qlen[0]), q1 = vload(&c->qlen[1]);
    en.cur = cur;
    en.nin = cur ? q1 : q0;
    en.mf = vload(&c->mf_front);
    en.vis = vsel ? a.vis2 : a.vis;
    en.vis_out = a.vis2 ? (vsel ? a.vis : a.vis2) : a.vis;
    en.skip = done || dir != want_dir;
    if (done) loop_over(a.ctl, a.h, a.use_cond);
  }
  __syncthreads();
  return en.skip != 0;
}

// Per-thread state of a push level (plain copies, so nothing is read through
// the kernel-parameter block).
struct PushCtx {
  int32_t *label;
  uint32_t *vis;
  const int32_t *ro;
  int32_t *qout;
  int32_t *qlen_out;
  int32_t *overflow;
  int32_t qcap;
  int32_t level;
  int64_t mf;
  BlockQueue *bq = nullptr;  // staging of discoveries (nullptr: straight to the queue)
};

__device__ __forceinline__ void bfs_visit(PushCtx &x, int32_t u) {
  const uint32_t bit = 1u << (u & 31);
  uint32_t *wp = x.vis + (u >> 5);
  bool disc = false;
  if (!(*wp & bit)) {
    uint32_t old = atomicOr(wp, bit);
    disc = !(old & bit);
  }
  if (disc) {
    x.label[u] = x.level + 1;
    x.mf += x.ro[u + 1] - x.ro[u];
  }
  staged_append(x.bq, disc, u, x.qout, x.qlen_out, x.qcap, x.overflow);
}

__global__ void __launch_bounds__(BFS_NT) bfs_push_kernel(BfsArgs a) {
  __shared__ ExpandSmem<BFS_NT> sm;
  __shared__ BlockQueue bq;
  __shared__ int64_t s_sum[BFS_NT / 32 + 1];
  __shared__ BfsEnter en;
  if (bfs_skip(a, 0, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  const int32_t nin = en.nin;
  const int32_t *qin = cur ? a.q1 : a.q0;
  PushCtx x{a.label, en.vis, a.ro, cur ? a.q0 : a.q1, &c->qlen[cur ^ 1], &c->overflow, a.qcap, en.level, 0};
  bq_init(bq);
  x.bq = &bq;
  int64_t insp = 0, nexp = 0;
  const BigList big{a.big_v, &c->big_len, defer_threshold<BFS_NT>(nin, a.cta_th, a.grid_th, a.defer_warp)};
  const int tl = tile_lanes<BFS_NT>(nin, en.mf), tn = tl * (BFS_NT / 32);
  for (int64_t tile = (int64_t)blockIdx.x * tn; tile < nin; tile += (int64_t)gridDim.x * tn) {
    const int64_t i = tile + warp_id() * tl + lane_id();
    const int32_t v = lane_id() < tl && i < nin ? qin[i] : -1;
    nexp += v >= 0;
    const int32_t *ci = a.ci, *ri = a.ri;
    expand_tile<BFS_NT, BFS_CTA_TH>(sm, a.ro, v, insp, [&](int32_t, int32_t k) { bfs_visit(x, ci[k]); }, &big, -1,
                                    a.cta_th);
    if (a.both)
      expand_tile<BFS_NT, BFS_CTA_TH>(sm, a.co, v, insp, [&](int32_t, int32_t k) { bfs_visit(x, ri[k]); }, nullptr,
                                      -1, a.cta_th);
  }
  bq_flush(bq, x.qout, x.qlen_out, x.qcap, x.overflow);
  const int64_t bmf = block_sum<BFS_NT>(x.mf, s_sum);
  const int64_t bins = block_sum<BFS_NT>(insp, s_sum);
  const int64_t bexp = block_sum<BFS_NT>(nexp, s_sum);
  if (threadIdx.x == 0) {
    if (bmf) atomicAdd((unsigned long long *)&c->mf_next, (unsigned long long)bmf);
    if (bins) atomicAdd((unsigned long long *)&c->edges_inspected, (unsigned long long)bins);
    if (bexp) atomicAdd((unsigned long long *)&c->vertices_expanded, (unsigned long long)bexp);
  }
}

// Persistent push levels for small frontiers (high-diameter graphs such as
// lattices, where a BFS has thousands of levels of a few thousand vertices and
// per-level launches dominate). One cooperative launch runs level after level,
// with a grid barrier between the expansion and the level end, while the level is
// a push level with at most bfs_persist_max frontier vertices and bfs_persist_edges
// frontier out-edges; it then returns and the per-level kernels continue from the
// same control block. Vertices of GRID_TH or more edges are deferred as in the
// per-level push and expanded by the whole grid after a second barrier, which
// only levels that deferred one take.
constexpr unsigned long long PERSIST_WAIT = 1ull << 22;  // barrier polls (seconds at most) before giving up

__global__ void __launch_bounds__(BFS_NT) bfs_persist_kernel(BfsArgs a) {
  // The tile pass and the grid-strided pass are separated by a grid barrier.
  __shared__ union {
    ExpandSmem<BFS_NT> e;
    BigSmem<BFS_NT> b;
  } sm;
  __shared__ BlockQueue bq;
  __shared__ int64_t s_sum[BFS_NT / 32 + 1];
  // Read by one thread per block (at entry, and behind each barrier): every warp of
  // the grid reading one L2 sector queues for microseconds.
  __shared__ struct {
    int32_t lvl, sel, nin, cap, skip, pq, pb, ok;
    int64_t mf, vdeg, pm;
    uint32_t *vis;
  } s_c;
  DevCtl *c = a.ctl;
  unsigned gen = 0;  // thread 0: the barrier's generation, moved by nobody else's arrival alone
  // Entry state, as the seed kernel or the last per-level kernel left it; every
  // block reads the same values and then takes the same decisions level by level.
  if (threadIdx.x == 0) {
    gen = vload(&c->bar_gen);
    const int32_t done = vload(&c->done), dir = vload(&c->dir), q0 = vload(&c->qlen[0]), q1 = vload(&c->qlen[1]);
    s_c.lvl = vload(&c->level);
    s_c.sel = vload(&c->cur);
    s_c.mf = vload(&c->mf_front);
    s_c.vdeg = vload(&c->visited_deg);
    s_c.cap = vload(&c->iter_cap);
    s_c.vis = vload(&c->vsel) ? a.vis2 : a.vis;
    s_c.nin = s_c.sel ? q1 : q0;
    s_c.skip = done || dir != 0 || s_c.nin > a.persist_max || s_c.mf > a.persist_edges;
  }
  __syncthreads();
  if (s_c.skip) return;
  const int32_t l0 = s_c.lvl, iter_cap = s_c.cap;
  int32_t lvl = l0, sel = s_c.sel, nin = s_c.nin;
  int64_t mf = s_c.mf, vdeg = s_c.vdeg;
  uint32_t *vis = s_c.vis;
  // Grid barrier (bounded) that ends with the counters of slot `out` in s_c.
  auto barrier = [&](int out) {
    __syncthreads();
    if (threadIdx.x == 0) {
      int ok = 1;
      __threadfence();
      if (atomicAdd(&c->bar_count, 1u) + 1 == gridDim.x + a.bar_extra) {
        c->bar_count = 0;
        __threadfence();
        atomicAdd(&c->bar_gen, 1u);
      } else {
        unsigned long long it = 0;
        while (vload(&c->bar_gen) == gen) {
          if (++it > a.bar_limit) {
            ok = 0;
            break;
          }
        }
      }
      gen++;
      __threadfence();
      s_c.pq = vload(&c->pq[out]);
      s_c.pb = vload(&c->pb[out]);
      s_c.pm = vload(&c->pm[out]);
      s_c.ok = ok;
    }
    __syncthreads();
    return s_c.ok != 0;
  };
  bq_init(bq);
  for (;;) {
    // Per-level counters rotate over three slots: this level appends to `out`;
    // `zero` is the slot the next level appends to (nobody touches it now).
    const int out = (lvl - l0 + 1) % 3, zero = (lvl - l0 + 2) % 3;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->pq[zero] = 0;
      c->pm[zero] = 0;
      c->pb[zero] = 0;
    }
    const int32_t *qin = sel ? a.q1 : a.q0;
    PushCtx x{a.label, vis, a.ro, sel ? a.q0 : a.q1, &c->pq[out], &c->overflow, a.qcap, lvl, 0};
    x.bq = &bq;
    const BigList big{a.big_v, &c->pb[out], defer_threshold<BFS_NT>(nin, a.cta_th, a.grid_th, a.defer_warp)};
    const int32_t *ci = a.ci, *ri = a.ri;
    int64_t insp = 0, nexp = 0;
    const int tl = tile_lanes<BFS_NT>(nin, mf), tn = tl * (BFS_NT / 32);
    for (int64_t tile = (int64_t)blockIdx.x * tn; tile < nin; tile += (int64_t)gridDim.x * tn) {
      const int64_t i = tile + warp_id() * tl + lane_id();
      const int32_t v = lane_id() < tl && i < nin ? qin[i] : -1;
      nexp += v >= 0;
      expand_tile<BFS_NT, BFS_CTA_TH>(sm.e, a.ro, v, insp, [&](int32_t, int32_t k) { bfs_visit(x, ci[k]); }, &big,
                                      -1, a.cta_th);
      if (a.both)
        expand_tile<BFS_NT, BFS_CTA_TH>(sm.e, a.co, v, insp, [&](int32_t, int32_t k) { bfs_visit(x, ri[k]); },
                                        nullptr, -1, a.cta_th);
    }
    bq_flush(bq, x.qout, x.qlen_out, x.qcap, x.overflow);
    const int64_t bmf = block_sum<BFS_NT>(x.mf, s_sum);
    const int64_t bins = block_sum<BFS_NT>(insp, s_sum);
    const int64_t bexp = block_sum<BFS_NT>(nexp, s_sum);
    if (threadIdx.x == 0) {
      if (bmf) atomicAdd((unsigned long long *)&c->pm[out], (unsigned long long)bmf);
      if (bins) atomicAdd((unsigned long long *)&c->edges_inspected, (unsigned long long)bins);
      if (bexp) atomicAdd((unsigned long long *)&c->vertices_expanded, (unsigned long long)bexp);
    }
    if (!barrier(out)) {
      if (threadIdx.x == 0) {
        c->status = MG_ERR_TIMEOUT;
        c->done = 1;
      }
      return;
    }
    if (s_c.pb > 0) {
      // The deferred vertices' edges, spread over the whole grid.
      x.mf = 0;
      expand_big<BFS_NT>(sm.b, a.ro, big, [&](int32_t, int32_t k) { bfs_visit(x, ci[k]); });
      bq_flush(bq, x.qout, x.qlen_out, x.qcap, x.overflow);
      const int64_t bmf2 = block_sum<BFS_NT>(x.mf, s_sum);
      if (threadIdx.x == 0 && bmf2) atomicAdd((unsigned long long *)&c->pm[out], (unsigned long long)bmf2);
      if (!barrier(out)) {
        if (threadIdx.x == 0) {
          c->status = MG_ERR_TIMEOUT;
          c->done = 1;
        }
        return;
      }
    }
    // Level end (bfs_level_end's rules), computed alike in every block.
    if (blockIdx.x == 0 && threadIdx.x == 0) trace_level(c, lvl, MG_DIR_PUSH, nin, mf, 0.0);
    const int32_t nf = s_c.pq;
    mf = s_c.pm;
    vdeg += mf;
    lvl += 1;
    sel ^= 1;
    const bool over = nf > a.qcap;  // not the flag: a faster block may have set it in the next level
    const bool done = nf == 0 || lvl >= iter_cap || over;
    int dir = 0;
    if (a.mode == MG_DIR_PULL) dir = a.can_pull ? 1 : 0;
    else if (a.mode == MG_DIR_AUTO && a.can_pull && mf > (a.m_total - vdeg) / a.alpha) dir = 1;
    if (done || dir != 0 || nf > a.persist_max || mf > a.persist_edges) {
      // Hand over to the per-level kernels (or finish) with their control state.
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        c->level = lvl;
        c->cur = sel;
        c->qlen[sel] = nf;
        c->qlen[sel ^ 1] = 0;
        c->visited_deg = vdeg;
        c->mf_front = mf;
        c->mf_next = 0;
        c->blocks_done = 0;
        c->big_len = 0;
        c->nf_next = nf;
        c->dir = dir;
        if (dir == 1 && !done) c->levels_pull += 1;
        if (over) c->status = MG_ERR_QUEUE_OVERFLOW;
        __threadfence();
        c->done = done ? 1 : 0;
      }
      return;
    }
    nin = nf;
  }
}

// Grid-strided bin of a push level: the deferred hubs' edges spread over every
// CTA; the last CTA closes the level.
__global__ void __launch_bounds__(BFS_NT) bfs_push_big_kernel(BfsArgs a) {
  __shared__ BigSmem<BFS_NT> sm;
  __shared__ BlockQueue bq;
  __shared__ int64_t s_sum[BFS_NT / 32 + 1];
  __shared__ BfsEnter en;
  if (bfs_skip(a, 0, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  PushCtx x{a.label, en.vis, a.ro, cur ? a.q0 : a.q1, &c->qlen[cur ^ 1], &c->overflow, a.qcap, en.level, 0};
  bq_init(bq);
  x.bq = &bq;
  const int32_t *ci = a.ci;
  expand_big<BFS_NT>(sm, a.ro, BigList{a.big_v, &c->big_len}, [&](int32_t, int32_t k) { bfs_visit(x, ci[k]); });
  bq_flush(bq, x.qout, x.qlen_out, x.qcap, x.overflow);
  const int64_t bmf = block_sum<BFS_NT>(x.mf, s_sum);
  if (threadIdx.x == 0 && bmf) atomicAdd((unsigned long long *)&c->mf_next, (unsigned long long)bmf);
  if (last_block(&c->blocks_done) && threadIdx.x == 0) bfs_level_end(a);
}

// Latency bounds it: few edges are read (R-MAT s22, three levels: 11 M), each at the
// end of a chain of dependent loads. So the next word's bits and offsets are loaded
// while this one is scanned; a lane tests a sector of indices at a time, 8 bits in
// flight; vertices still without a parent after that are taken eight at a time by
// four lanes each, 32 edges per step (a warp per vertex took up to 32 turns for a word
// of vertices of middling degree, a lane per vertex up to the longest row); and
// discoveries are staged per warp (one queue atomic per word queued 130,000 of them on
// one address). Largest level of R-MAT s22: 191 us one edge and one depth load at a
// time, 115 us now.
// BITS: the test reads the bitmap the level found (else the depth, and the one bitmap
// is updated in place).
template <bool BITS>
__global__ void __launch_bounds__(BFS_NT, 6) bfs_pull_kernel(BfsArgs a) {
  __shared__ int64_t s_sum[BFS_NT / 32 + 1];
  __shared__ int32_t s_stage[BFS_NT / 32][WS_CAP];
  __shared__ BfsEnter en;
  if (bfs_skip(a, 1, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  const int32_t level = en.level;
  const uint32_t *vis = en.vis;
  uint32_t *vout = en.vis_out;
  int32_t *qout = cur ? a.q0 : a.q1;
  int32_t *qlen_out = &c->qlen[cur ^ 1];
  WarpStage st{s_stage[warp_id()], 0};
  const int lane = lane_id();
  const int32_t nwords = (int32_t)((a.n + 31) >> 5), wstride = (int32_t)(gridDim.x * (BFS_NT / 32));
  const bool same = a.ro == a.co;  // the in-degree is the out-degree
  int64_t mf = 0, insp = 0, nexp = 0;
  // any parent among the sector at e of edges [b, end): all eight loads are issued
  // before the first is tested
  auto sector = [&](int32_t e, int32_t b, int32_t end) {
    int32_t u[8];
    uint32_t x[8];
    prb_load8(a.ri + e, u);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const bool in = e + j >= b && e + j < end;
      if (BITS) x[j] = in ? __ldg(vis + (u[j] >> 5)) : 0u;
      else x[j] = in ? (uint32_t)a.label[u[j]] : ~0u;
    }
    bool f = false;
#pragma unroll
    for (int j = 0; j < 8; j++) f |= BITS ? ((x[j] >> (u[j] & 31)) & 1u) != 0 : x[j] == (uint32_t)level;
    insp += min(e + 8, end) - max(e, b);
    return f;
  };
  // a word's bits and its vertices' offsets, loaded one word ahead
  auto fetch = [&](int32_t w, uint32_t &vw, int32_t &beg, int32_t &end) {
    vw = FULL;
    beg = end = 0;
    if (w >= nwords) return;
    vw = vis[w];
    const int64_t v = ((int64_t)w << 5) + lane;
    if (v < a.n) {
      beg = a.co[v];
      end = a.co[v + 1];
    }
  };
  int32_t w = blockIdx.x * (BFS_NT / 32) + warp_id();
  uint32_t vw, vw1;
  int32_t beg, end, beg1, end1;
  fetch(w, vw, beg, end);
  for (; w < nwords; w += wstride, vw = vw1, beg = beg1, end = end1) {
    fetch(w + wstride, vw1, beg1, end1);
    if (vw == FULL) {
      if (BITS && lane == 0) vout[w] = FULL;
      continue;
    }
    const int64_t v = ((int64_t)w << 5) + lane;
    const bool need = v < a.n && !((vw >> lane) & 1u);
    bool found = false;
    nexp += need;
    const int32_t lim = min(end, (beg & ~7) + PULL_SERIAL);
    if (need && beg < end) found = sector(beg & ~7, beg, lim);
    unsigned pend = __ballot_sync(FULL, need && !found && lim < end);
    unsigned far = 0;  // lanes whose vertex is left for the whole warp
    while (pend) {
      // quad q takes the q-th waiting vertex
      unsigned m = pend;
      for (int q = lane >> 2; q > 0; q--) m &= m - 1;
      const int l = m ? __ffs(m) - 1 : 0;
      const int32_t b = __shfl_sync(FULL, lim, l), en0 = __shfl_sync(FULL, end, l);
      const int32_t en = m ? min(en0, b + PULL_QUAD) : b;
      const unsigned mine = 0xfu << (lane & ~3);
      bool f = false;
      for (int32_t e = (b & ~7) + 8 * (lane & 3); __any_sync(FULL, !f && e - 8 * (lane & 3) < en); e += 32) {
        if (!f && e < en && e + 8 > b) f = sector(e, b, en);
        f = (__ballot_sync(FULL, f) & mine) != 0;
      }
      // back to the vertices' lanes: the r-th waiting vertex was quad r's
      const unsigned fq = __ballot_sync(FULL, f), mq = __ballot_sync(FULL, en0 > en);
      const int r = 4 * __popc(pend & lanemask_lt());
      const bool served = ((pend >> lane) & 1u) && r < 32;
      if (served) found = (fq >> r) & 1u;
      far |= __ballot_sync(FULL, served && !found && ((mq >> r) & 1u));
      pend = __ballot_sync(FULL, ((pend >> lane) & 1u) && !served);
    }
    while (far) {
      const int l = __ffs(far) - 1;
      far &= far - 1;
      const int32_t b = __shfl_sync(FULL, lim, l) + PULL_QUAD, en = __shfl_sync(FULL, end, l);
      bool f = false;
      for (int32_t e0 = b & ~7; e0 < en && !f; e0 += 256) {
        const int32_t e = e0 + 8 * lane;
        f = __any_sync(FULL, e < en && e + 8 > b && sector(e, b, en));
      }
      if (lane == l) found = f;
    }
    const unsigned fm = __ballot_sync(FULL, found);
    if (lane == 0 && (fm || BITS)) vout[w] = vw | fm;
    if (found) {
      a.label[v] = level + 1;
      mf += same ? end - beg : a.ro[v + 1] - a.ro[v];
    }
    ws_push(st, found, (int32_t)v, qout, qlen_out, a.qcap, &c->overflow);
  }
  ws_flush(st, qout, qlen_out, a.qcap, &c->overflow);
  const int64_t bmf = block_sum<BFS_NT>(mf, s_sum);
  const int64_t bins = block_sum<BFS_NT>(insp, s_sum);
  const int64_t bexp = block_sum<BFS_NT>(nexp, s_sum);
  if (threadIdx.x == 0) {
    if (bmf) atomicAdd((unsigned long long *)&c->mf_next, (unsigned long long)bmf);
    if (bins) atomicAdd((unsigned long long *)&c->edges_inspected, (unsigned long long)bins);
    if (bexp) atomicAdd((unsigned long long *)&c->vertices_expanded, (unsigned long long)bexp);
  }
  if (last_block(&c->blocks_done) && threadIdx.x == 0) bfs_level_end(a);
}

// labels := -1, visited := 0.
__global__ void bfs_clear_kernel(int32_t *label, uint32_t *vis, int64_t n) {
  const int64_t nw = (n + 31) >> 5;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    label[i] = -1;
    if (i < nw) vis[i] = 0;
  }
}

// Seeds the sources (duplicates collapse) and initialises the control block.
__global__ void bfs_seed_kernel(BfsArgs a, const int32_t *srcs, int32_t nsrc, int32_t iter_cap, int32_t dir0) {
  __shared__ int64_t s_sum[1024 / 32 + 1];
  DevCtl *c = a.ctl;
  int64_t mf = 0;
  for (int i = threadIdx.x; i < nsrc; i += blockDim.x) {
    const int32_t s = srcs[i];
    const uint32_t bit = 1u << (s & 31);
    const uint32_t old = atomicOr(&a.vis[s >> 5], bit);
    if (!(old & bit)) {
      a.label[s] = 0;
      mf += a.ro[s + 1] - a.ro[s];
      int pos = atomicAdd(&c->qlen[0], 1);
      if (pos < a.qcap) a.q0[pos] = s;
      else c->overflow = 1;
    }
  }
  const int64_t t = block_sum<1024>(mf, s_sum);
  if (threadIdx.x == 0) {
    c->visited_deg = t;
    c->mf_front = t;
    c->level = 0;
    c->cur = 0;
    c->dir = dir0;
    c->iter_cap = iter_cap;
    c->done = (iter_cap <= 0 || c->overflow) ? 1 : 0;
    if (c->overflow) c->status = MG_ERR_QUEUE_OVERFLOW;
  }
}

// A whole BFS of a small graph in one launch of one thread-block cluster: clear,
// seeds, every level, counters. Levels are separated by the hardware cluster
// barrier (well under a microsecond), where a grid barrier of every SM takes about
// three and a launch per level more, and the level's lengths live in the first
// CTA's shared memory. Each CTA keeps a copy of the visited bitmap, refreshed per
// level, so most edges to vertices already reached end there; the others claim
// their vertex with one atomic on the bitmap in L2. Latency bounds it: about eight
// dependent memory round trips per level. Top-down only: the edges it could skip
// bottom-up cost less than the extra passes at these sizes.
//
// The limits are where the cluster's 8 SMs stop beating the whole grid's per-level
// kernels: 1 M edges, R-MAT 194 us against 226, uniform 150 against 218 (32 K edges:
// 85 and 204, 68 and 179).
constexpr int SB_NT = 1024;
constexpr int SB_CLUSTER = 8;
constexpr int64_t SB_MAX_N = 1 << 17;
constexpr int64_t SB_MAX_M = 1 << 20;
constexpr int SB_CH = 256;   // edges per chunk of a heavy vertex
constexpr int SB_U = 4;      // edges a lane has in flight
constexpr int SB_SRC = 8;    // sources passed by value

struct SmallBfs {
  int32_t src[SB_SRC];
  const int32_t *dsrc;  // more sources than SB_SRC (else nullptr)
  int32_t nsrc;
  int32_t iter_cap;
  int2 *chunks;  // {first edge | 1 << 31 for a CSC edge, end}
};

// Most chunks of a level: a vertex of at least SB_CH edges has under twice its
// edges / SB_CH, in each direction.
inline int32_t small_bfs_chunks(int64_t m) { return (int32_t)(4 * (m / SB_CH) + 64); }

__global__ void __cluster_dims__(SB_CLUSTER, 1, 1) __launch_bounds__(SB_NT, 1)
    bfs_small_kernel(BfsArgs a, SmallBfs sb) {
  namespace cg = cooperative_groups;
  __shared__ uint32_t s_vis[SB_MAX_N / 32];
  __shared__ BlockQueue bq;
  __shared__ int32_t s_len[3], s_chunk[3];
  __shared__ unsigned long long s_mf[3], s_tot[2];
  cg::cluster_group cl = cg::this_cluster();
  DevCtl *c = a.ctl;
  const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = lane_id();
  const bool lead = rank == 0 && tid == 0;
  const int32_t nthr = SB_CLUSTER * SB_NT, gt = tid * SB_CLUSTER + rank;
  const int32_t nw = nthr / 32, gw = warp_id() * SB_CLUSTER + rank;
  int32_t *len = cl.map_shared_rank(s_len, 0), *chunk = cl.map_shared_rank(s_chunk, 0);
  unsigned long long *mfs = cl.map_shared_rank(s_mf, 0), *tot = cl.map_shared_rank(s_tot, 0);
  const int32_t nwords = (int32_t)((a.n + 31) >> 5);
  for (int32_t i = rank * SB_NT + tid; i < a.n; i += nthr) a.label[i] = -1;
  for (int32_t i = rank * SB_NT + tid; i < nwords; i += nthr) a.vis[i] = 0u;
  if (rank == 0) {
    for (int i = tid; i < (int)(sizeof(DevCtl) / 4); i += SB_NT) reinterpret_cast<int32_t *>(c)[i] = 0;
    if (tid < 3) {
      s_len[tid] = 0;
      s_chunk[tid] = 0;
      s_mf[tid] = 0;
    }
    if (tid < 2) s_tot[tid] = 0;
  }
  bq_init(bq);
  cl.sync();
  if (rank == 0) {
    for (int i = tid; i < sb.nsrc; i += SB_NT) {
      const int32_t v = sb.dsrc ? sb.dsrc[i] : sb.src[i];
      const uint32_t bit = 1u << (v & 31);
      if (!(atomicOr(a.vis + (v >> 5), bit) & bit)) {
        a.label[v] = 0;
        const int pos = atomicAdd(&s_len[0], 1);
        if (pos < a.qcap) a.q0[pos] = v;
        else c->overflow = 1;
      }
    }
  }
  cl.sync();
  int32_t nin = len[0];
  int32_t lvl = 0, sel = 0;
  bool over = nin > a.qcap;  // from the level's own length, see its end
  bool done = over || sb.iter_cap <= 0;
  int64_t insp = 0, nexp = 0, vdeg = 0;
  // claims the items u (-1: none) of a lane, issued together
  auto claim = [&](const int32_t (&u)[SB_U], int32_t *qout, int32_t *qlen) {
    uint32_t old[SB_U];
#pragma unroll
    for (int r = 0; r < SB_U; r++) {
      const uint32_t bit = 1u << (u[r] & 31);
      old[r] = FULL;
      if (u[r] >= 0 && !(s_vis[u[r] >> 5] & bit)) {
        old[r] = atomicOr(a.vis + (u[r] >> 5), bit);
        atomicOr(s_vis + (u[r] >> 5), bit);
      }
    }
#pragma unroll
    for (int r = 0; r < SB_U; r++) {
      const bool fresh = u[r] >= 0 && !((old[r] >> (u[r] & 31)) & 1u);
      if (fresh) a.label[u[r]] = lvl + 1;
      staged_append(&bq, fresh, u[r], qout, qlen, a.qcap, &c->overflow);
    }
  };
  // the edges of the warp's vertices (a lane each), concatenated
  auto walk = [&](int32_t beg, int32_t deg, const int32_t *__restrict__ adj, int32_t flag, int32_t *qout, int32_t *qlen,
                  int32_t *clen) {
    const int32_t nch = deg >= SB_CH ? (deg + SB_CH - 1) / SB_CH : 0;
    if (nch) {
      const int32_t base = atomicAdd(clen, nch);
      for (int32_t j = 0; j < nch; j++)  // within the capacity: a level's vertices are distinct
        sb.chunks[base + j] = make_int2((beg + j * SB_CH) | flag, min(beg + (j + 1) * SB_CH, beg + deg));
      deg = 0;
    }
    __syncwarp();
    const int32_t inc = warp_inclusive_scan(deg);
    const int32_t total = __shfl_sync(FULL, inc, 31);
    const int32_t ex = inc - deg, kb = beg - ex;
    for (int32_t b0 = 0; b0 < total; b0 += 32 * SB_U) {
      int32_t u[SB_U];
#pragma unroll
      for (int r = 0; r < SB_U; r++) {
        const int32_t j = b0 + r * 32 + lane;
        int l = 0;
#pragma unroll
        for (int sft = 16; sft > 0; sft >>= 1)
          if (__shfl_sync(FULL, ex, l + sft) <= j) l += sft;
        const int32_t k = __shfl_sync(FULL, kb, l) + j;
        u[r] = j < total ? adj[k] : -1;
      }
      claim(u, qout, qlen);
    }
  };
  while (!done) {
    // counters in a ring of three: this level adds to `out`; nobody reads or adds to
    // the next level's now
    const int out = (lvl + 1) % 3, zero = (lvl + 2) % 3;
    if (lead) {
      s_len[zero] = 0;
      s_chunk[zero] = 0;
      s_mf[zero] = 0;
    }
    for (int32_t i = tid; i < nwords; i += SB_NT) s_vis[i] = __ldcg(a.vis + i);
    __syncthreads();
    const int32_t *qin = sel ? a.q1 : a.q0;
    int32_t *qout = sel ? a.q0 : a.q1, *qlen = len + out, *clen = chunk + out;
    // a small frontier is spread over all the warps
    const int32_t per = max(1, min(32, (nin + nw - 1) / nw));
    int64_t front = 0;
    for (int32_t base = gw * per; base < nin; base += nw * per) {
      const int32_t i = base + lane;
      const int32_t v = lane < per && i < nin ? __ldcg(qin + i) : -1;
      int32_t beg = 0, deg = 0, cb = 0, cdeg = 0;
      if (v >= 0) {
        beg = a.ro[v];
        deg = a.ro[v + 1] - beg;
        if (a.both) {
          cb = a.co[v];
          cdeg = a.co[v + 1] - cb;
        }
        front += deg;
        insp += deg + cdeg;
        nexp++;
      }
      walk(beg, deg, a.ci, 0, qout, qlen, clen);
      if (a.both) walk(cb, cdeg, a.ri, INT_MIN, qout, qlen, clen);
    }
    front = warp_sum(front);
    if (lane == 0 && front) atomicAdd(mfs + out, (unsigned long long)front);
    cl.sync();
    const int32_t nch = chunk[out];
    if (nch > 0) {
      for (int32_t ch = gw; ch < nch; ch += nw) {
        const int2 e = __ldcg(sb.chunks + ch);
        const int32_t k0 = e.x & INT_MAX;
        const int32_t *adj = e.x < 0 ? a.ri : a.ci;
        for (int32_t b = k0; b < e.y; b += 32 * SB_U) {
          int32_t u[SB_U];
#pragma unroll
          for (int r = 0; r < SB_U; r++) u[r] = b + r * 32 + lane < e.y ? adj[b + r * 32 + lane] : -1;
          claim(u, qout, qlen);
        }
      }
    }
    bq_flush(bq, qout, qlen, a.qcap, &c->overflow);
    cl.sync();
    // Level end, alike in every CTA: a CTA that leaves takes its shared memory with it. So
    // an overflow shows in the level's length, which counts what did not fit; the flag in
    // the control block may be a faster CTA's, from the next level.
    const int64_t mf = (int64_t)mfs[out];
    const int32_t nf = len[out];
    over = nf > a.qcap;
    if (lead) {
      trace_level(c, lvl, MG_DIR_PUSH, nin, mf, 0.0);
      vdeg += mf;
    }
    lvl++;
    sel ^= 1;
    nin = nf;
    done = nf == 0 || lvl >= sb.iter_cap || over;
  }
  // an iteration cap leaves a frontier that was reached but not expanded
  const int32_t *qin = sel ? a.q1 : a.q0;
  int64_t rest = 0;
  for (int32_t i = gt; i < min(nin, a.qcap); i += nthr) {
    const int32_t v = __ldcg(qin + i);
    rest += a.ro[v + 1] - a.ro[v];
  }
  insp = warp_sum(insp);
  nexp = warp_sum(nexp);
  rest = warp_sum(rest + vdeg);
  if (lane == 0) {
    if (insp) atomicAdd(tot, (unsigned long long)insp);
    if (nexp) atomicAdd(tot + 1, (unsigned long long)nexp);
    if (rest) atomicAdd((unsigned long long *)&c->visited_deg, (unsigned long long)rest);
  }
  cl.sync();  // the last access to the first CTA's shared memory
  if (lead) {
    c->edges_inspected = (int64_t)s_tot[0];
    c->vertices_expanded = (int64_t)s_tot[1];
    c->level = lvl;
    if (over) c->status = MG_ERR_QUEUE_OVERFLOW;
    c->done = 1;
  }
}

}  // namespace mg

// Blocks of the persistent kernel: every SM's resident share (0 when the
// occupancy query fails).
static int persist_grid(mg_graph *g) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mg::bfs_persist_kernel, mg::BFS_NT, 0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return occ > 0 ? g->num_sms * std::min(occ, 4) : 0;
}

extern "C" mg_status mg_bfs(mg_graph *g, const int32_t *srcs, int32_t nsrc, int32_t *depth, const mg_opts *opts,
                            mg_stats *stats) {
  using namespace mg;
  if (!g || !srcs || nsrc <= 0 || !depth) {
    mg_set_error("mg_bfs: null argument or nsrc <= 0");
    return MG_ERR_ARG;
  }
  mg_opts o;
  std::memset(&o, 0, sizeof(o));
  o.directed = 1;
  if (opts) o = *opts;
  if (o.direction < MG_DIR_AUTO || o.direction > MG_DIR_PULL) {
    mg_set_error("mg_bfs: invalid direction %d", o.direction);
    return MG_ERR_ARG;
  }
  for (int32_t i = 0; i < nsrc; i++) {
    if (srcs[i] < 0 || srcs[i] >= g->n) {
      mg_set_error("mg_bfs: source %d out of range [0, %lld)", srcs[i], (long long)g->n);
      return MG_ERR_ARG;
    }
  }
  const bool symmetric = (g->flags & MG_GRAPH_SYMMETRIC) != 0;
  const bool undirected = o.directed == 0 && !symmetric;
  if (undirected && !g->has_csc) {
    mg_set_error("mg_bfs: directed=0 needs the CSC (graph created with MG_GRAPH_NO_CSC)");
    return MG_ERR_UNSUPPORTED;
  }
  MG_TRY(graph_enter(g));
  if (o.device_output) MG_TRY(check_device_ptr(g, depth, "mg_bfs", "depth"));
  const int64_t n = g->n;
  int64_t qcap64 = o.queue_sizing > 0 ? (int64_t)std::ceil(o.queue_sizing * (double)n) : n;
  qcap64 = std::max<int64_t>(1, std::min<int64_t>(qcap64, n));
  const int32_t qcap = (int32_t)qcap64;
  const int64_t nwords = (n + 31) / 32;
  const size_t need = Carve::need({sizeof(int32_t) * (size_t)n, sizeof(uint32_t) * (size_t)nwords,
                                   sizeof(uint32_t) * (size_t)nwords, sizeof(int32_t) * (size_t)qcap, sizeof(int32_t) * (size_t)qcap,
                                   sizeof(int32_t) * (size_t)nsrc, sizeof(int32_t) * (size_t)BIG_CAP,
                                   sizeof(int2) * (size_t)(n <= SB_MAX_N && g->m <= SB_MAX_M ? small_bfs_chunks(g->m)
                                                                                             : 0)});
  MG_TRY(ws_reserve(g, g->ws_main, need));
  Carve cv(g->ws_main.ptr);
  int32_t *label_ws = cv.take<int32_t>(n);
  uint32_t *vis = cv.take<uint32_t>(nwords), *vis2 = cv.take<uint32_t>(nwords);
  int32_t *q0 = cv.take<int32_t>(qcap);
  int32_t *q1 = cv.take<int32_t>(qcap);
  int32_t *dsrc = cv.take<int32_t>(nsrc);
  int32_t *big_v = cv.take<int32_t>(BIG_CAP);
  int32_t *label = o.device_output ? depth : label_ws;
  cudaStream_t s = g->stream;

  BfsArgs a;
  std::memset(&a, 0, sizeof(a));  // the loop-graph signature compares its bytes
  bfs_tuning(a, g->tune);
  a.ro = g->ro;
  a.ci = g->ci;
  a.co = g->has_csc ? g->co : g->ro;
  a.ri = g->has_csc ? g->ri : g->ci;
  a.label = label;
  a.vis = vis;
  a.vis2 = vis2;
  a.q0 = q0;
  a.q1 = q1;
  a.qcap = qcap;
  // AUTO on sparse graphs (mean out-degree <= 8: lattices, road networks) stays
  // top-down: a bottom-up level scans every unvisited vertex and, far from a thin
  // wavefront, finds no early exit (4096^2 lattice: 7.8 ms with Beamer's rule,
  // 6.7 ms top-down only).
  a.mode = (o.direction == MG_DIR_AUTO && g->m <= (int64_t)g->tune.bfs_sparse_degree * g->n) ? MG_DIR_PUSH
                                                                                           : o.direction;
  a.can_pull = g->has_csc && !undirected;
  a.both = undirected ? 1 : 0;
  a.n = n;
  a.m_total = g->m;
  a.big_v = big_v;
  a.ctl = g->ctl;
  a.h = 0;
  a.use_cond = 0;
  a.bar_extra = (uint32_t)debug_barrier_extra();
  a.bar_limit = a.bar_extra ? debug_barrier_limit() : PERSIST_WAIT;

  const int32_t iter_cap = o.iter_num > 0 ? (int32_t)std::min<int64_t>(o.iter_num, n + 1) : (int32_t)(n + 1);
  const bool use_graph = o.use_graph >= 0;
  // Small graphs in one cluster launch, unless the caller asked for bottom-up levels
  // or the per-level kernels (host-driven loop, thresholds of its own for them), or a
  // test skews the grid barriers.
  const bool small = n <= SB_MAX_N && g->m <= SB_MAX_M && use_graph && o.direction != MG_DIR_PULL &&
                     a.bar_extra == 0 && bfs_tuning_default(g->tune);
  if (!small || nsrc > SB_SRC)
    MG_CUDA_TRY(cudaMemcpyAsync(dsrc, srcs, sizeof(int32_t) * nsrc, cudaMemcpyHostToDevice, s));
  MG_CUDA_TRY(cudaEventRecord(g->ev0, s));
  int64_t persist_launches = 0;
  bool tail = false;
  if (small) {
    SmallBfs sb;
    std::memset(&sb, 0, sizeof(sb));
    for (int i = 0; i < std::min(nsrc, SB_SRC); i++) sb.src[i] = srcs[i];
    sb.dsrc = nsrc > SB_SRC ? dsrc : nullptr;
    sb.nsrc = nsrc;
    sb.iter_cap = iter_cap;
    sb.chunks = cv.take<int2>(small_bfs_chunks(g->m));
    bfs_small_kernel<<<SB_CLUSTER, SB_NT, 0, s>>>(a, sb);
    MG_CUDA_TRY(cudaGetLastError());
  } else {
    MG_CUDA_TRY(cudaMemsetAsync(g->ctl, 0, sizeof(DevCtl), s));
    bfs_clear_kernel<<<g->num_sms * 8, 256, 0, s>>>(label, vis, n);
    bfs_seed_kernel<<<1, 1024, 0, s>>>(a, dsrc, nsrc, iter_cap, 0);
    MG_CUDA_TRY(cudaGetLastError());
    // Small push levels first, in one persistent cooperative launch (all blocks
    // resident); a device that cannot co-schedule the grid skips it.
    const int pgrid = persist_grid(g);
    if (pgrid > 0 && o.direction != MG_DIR_PULL) {
      BfsArgs pa = a;
      void *params[] = {&pa};
      if (cudaLaunchCooperativeKernel((const void *)bfs_persist_kernel, dim3(pgrid), dim3(BFS_NT), params, 0, s) ==
          cudaSuccess)
        persist_launches = 1;
      cudaGetLastError();
    }

    const int grid = g->num_sms * g->tune.bfs_ctas_per_sm;
    struct Sig {
      BfsArgs a;
      int grid;
      int32_t tail_max, tail_edges;
    } sig;
    std::memset(&sig, 0, sizeof(sig));
    sig.a = a;
    sig.grid = grid;
    sig.tail_max = g->tune.bfs_tail_max;
    sig.tail_edges = g->tune.bfs_tail_edges;
    // Tail levels: one CTA runs the persistent kernel at the top of every iteration
    // (its grid barrier is the CTA's own), so a run of tiny push levels (at most
    // bfs_tail_max vertices and bfs_tail_edges out-edges) costs one launch instead of
    // a launch sequence per level; on a larger frontier it returns at once and the
    // per-level kernels go on from the same control block.
    BfsArgs ta = a;
    ta.persist_max = g->tune.bfs_tail_max;
    ta.persist_edges = g->tune.bfs_tail_edges;
    tail = ta.persist_max > 0 && ta.persist_edges > 0 && o.direction != MG_DIR_PULL;
    LoopBody body = [a, ta, tail, grid](cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) {
      BfsArgs b = a;
      b.h = h;
      b.use_cond = use_cond;
      if (tail) bfs_persist_kernel<<<1, BFS_NT, 0, st>>>(ta);
      bfs_push_kernel<<<grid, BFS_NT, 0, st>>>(b);
      bfs_push_big_kernel<<<grid, BFS_NT, 0, st>>>(b);
      bfs_pull_kernel<true><<<grid + grid / 2, BFS_NT, 0, st>>>(b);  // less state per warp than the push kernels
    };
    MG_TRY(run_loop(g, SLOT_BFS, &sig, sizeof(sig), o.use_graph, body, n + 2));
  }
  MG_CUDA_TRY(cudaEventRecord(g->ev1, s));
  if (!o.device_output) MG_TRY(copy_out(g, depth, label, sizeof(int32_t) * n, 0));
  MG_TRY(fetch_ctl(g));
  const DevCtl &hc = *g->ctl_host;
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->iterations = hc.level;
    stats->edges_traversed = hc.visited_deg;
    stats->edges_inspected = hc.edges_inspected;
    stats->bytes_compulsory = 4 * hc.edges_inspected + 16 * hc.vertices_expanded + 4 * n +
                              (int64_t)hc.levels_pull * ((n + 7) / 8);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    stats->kernel_ms = ms;
    stats->status_detail = hc.levels_pull;
    const int64_t per = 3 + (tail ? 1 : 0);
    stats->launches = small ? 1 : 2 + persist_launches + loop_launches(g, per);
  }
  if (hc.status == MG_ERR_TIMEOUT) {
    mg_set_error("mg_bfs: a grid barrier of the persistent levels timed out");
    return MG_ERR_TIMEOUT;
  }
  if (hc.status != 0) {
    mg_set_error("mg_bfs: frontier exceeded queue capacity %d", qcap);
    return (mg_status)hc.status;
  }
  return MG_OK;
}

// ---- BFS over a fixed, statically allocated scratch area -------------------
// mg_bfs grows the graph's workspace on demand, which allocates device memory on
// the first call and whenever a call needs more. Some callers cannot allow that:
// a serving process that reserved its device memory up front and must not grow it
// while requests run, code called from inside a memory allocator (which must not
// re-enter the allocator), or a caller that keeps every device allocation under
// its own accounting. This variant takes its frontier queues, visited bitmap,
// source list and deferred-hub list from one file-scope device array of fixed
// size, writes depths straight into the caller's device buffer, and drives the
// level loop from the host (no executable graph is instantiated).
namespace mg {

constexpr int64_t NOALLOC_MAX_N = MG_BFS_NOALLOC_MAX_VERTICES;
constexpr int64_t NOALLOC_MAX_SRC = MG_BFS_NOALLOC_MAX_SOURCES;
constexpr size_t noalloc_round(size_t b) { return (b + 255) & ~(size_t)255; }
// Layout (bytes, each part 256-aligned): visited bitmap, two frontier queues,
// sources, deferred hubs.
constexpr size_t NOALLOC_VIS = 0;
constexpr size_t NOALLOC_Q0 = NOALLOC_VIS + noalloc_round(sizeof(uint32_t) * ((NOALLOC_MAX_N + 31) / 32));
constexpr size_t NOALLOC_Q1 = NOALLOC_Q0 + noalloc_round(sizeof(int32_t) * NOALLOC_MAX_N);
constexpr size_t NOALLOC_SRC = NOALLOC_Q1 + noalloc_round(sizeof(int32_t) * NOALLOC_MAX_N);
constexpr size_t NOALLOC_BIG = NOALLOC_SRC + noalloc_round(sizeof(int32_t) * NOALLOC_MAX_SRC);
constexpr size_t NOALLOC_BYTES = NOALLOC_BIG + noalloc_round(sizeof(int32_t) * BIG_CAP);  // 8,540,160 bytes

// Nothing in it has to start at zero: every call clears the bitmap itself and
// writes the queues, sources and hub list before reading them.
static __device__ __align__(256) uint32_t bfs_noalloc_scratch[NOALLOC_BYTES / sizeof(uint32_t)];

// Waits for a stream when it goes out of scope.
struct StreamDrain {
  cudaStream_t s;
  ~StreamDrain() { cudaStreamSynchronize(s); }
};

// Device address of the scratch array, resolved once per device (the first call
// on a device; later calls reuse the cached address).
static std::mutex noalloc_mu;
static std::vector<char *> noalloc_addr;

static mg_status noalloc_scratch_of(int device, char **out) {
  std::lock_guard<std::mutex> lk(noalloc_mu);
  if ((int)noalloc_addr.size() <= device) noalloc_addr.resize(device + 1, nullptr);
  if (!noalloc_addr[device]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, bfs_noalloc_scratch);
    if (e != cudaSuccess) {
      mg_set_error("mg_bfs_noalloc: cudaGetSymbolAddress of the scratch array failed on device %d: %s", device,
                   cudaGetErrorString(e));
      return MG_ERR_CUDA;
    }
    noalloc_addr[device] = static_cast<char *>(p);
  }
  *out = noalloc_addr[device];
  return MG_OK;
}

}  // namespace mg

extern "C" mg_status mg_bfs_noalloc(mg_graph *g, const int32_t *srcs, int32_t nsrc, int32_t *depth,
                                    const mg_opts *opts, mg_stats *stats) {
  using namespace mg;
  if (!g || !srcs || nsrc <= 0 || !depth) {
    mg_set_error("mg_bfs_noalloc: null argument or nsrc <= 0");
    return MG_ERR_ARG;
  }
  if (g->n > NOALLOC_MAX_N) {
    mg_set_error("mg_bfs_noalloc: graph has %lld vertices, the fixed scratch holds at most %lld (use mg_bfs)",
                 (long long)g->n, (long long)NOALLOC_MAX_N);
    return MG_ERR_ARG;
  }
  if (nsrc > NOALLOC_MAX_SRC) {
    mg_set_error("mg_bfs_noalloc: %d sources, the fixed scratch holds at most %lld", nsrc,
                 (long long)NOALLOC_MAX_SRC);
    return MG_ERR_ARG;
  }
  mg_opts o;
  std::memset(&o, 0, sizeof(o));
  o.directed = 1;
  if (opts) o = *opts;
  if (o.direction < MG_DIR_AUTO || o.direction > MG_DIR_PULL) {
    mg_set_error("mg_bfs_noalloc: invalid direction %d", o.direction);
    return MG_ERR_ARG;
  }
  for (int32_t i = 0; i < nsrc; i++) {
    if (srcs[i] < 0 || srcs[i] >= g->n) {
      mg_set_error("mg_bfs_noalloc: source %d out of range [0, %lld)", srcs[i], (long long)g->n);
      return MG_ERR_ARG;
    }
  }
  const bool symmetric = (g->flags & MG_GRAPH_SYMMETRIC) != 0;
  const bool undirected = o.directed == 0 && !symmetric;
  if (undirected && !g->has_csc) {
    mg_set_error("mg_bfs_noalloc: directed=0 needs the CSC (graph created with MG_GRAPH_NO_CSC)");
    return MG_ERR_UNSUPPORTED;
  }
  MG_TRY(graph_enter(g));
  MG_TRY(check_device_ptr(g, depth, "mg_bfs_noalloc", "depth"));
  char *scratch = nullptr;
  MG_TRY(noalloc_scratch_of(g->device, &scratch));
  const int64_t n = g->n;
  int64_t qcap64 = o.queue_sizing > 0 ? (int64_t)std::ceil(o.queue_sizing * (double)n) : n;
  qcap64 = std::max<int64_t>(1, std::min<int64_t>(qcap64, n));
  const int32_t qcap = (int32_t)qcap64;
  int32_t *dsrc = reinterpret_cast<int32_t *>(scratch + NOALLOC_SRC);
  cudaStream_t s = g->stream;

  BfsArgs a;
  std::memset(&a, 0, sizeof(a));  // the loop-graph signature compares its bytes
  bfs_tuning(a, g->tune);
  a.ro = g->ro;
  a.ci = g->ci;
  a.co = g->has_csc ? g->co : g->ro;
  a.ri = g->has_csc ? g->ri : g->ci;
  a.label = depth;
  a.vis = reinterpret_cast<uint32_t *>(scratch + NOALLOC_VIS);
  a.q0 = reinterpret_cast<int32_t *>(scratch + NOALLOC_Q0);
  a.q1 = reinterpret_cast<int32_t *>(scratch + NOALLOC_Q1);
  a.qcap = qcap;
  // AUTO on sparse graphs (mean out-degree <= 8: lattices, road networks) stays
  // top-down: a bottom-up level scans every unvisited vertex and, far from a thin
  // wavefront, finds no early exit (4096^2 lattice: 7.8 ms with Beamer's rule,
  // 6.7 ms top-down only).
  a.mode = (o.direction == MG_DIR_AUTO && g->m <= (int64_t)g->tune.bfs_sparse_degree * g->n) ? MG_DIR_PUSH
                                                                                           : o.direction;
  a.can_pull = g->has_csc && !undirected;
  a.both = undirected ? 1 : 0;
  a.n = n;
  a.m_total = g->m;
  a.big_v = reinterpret_cast<int32_t *>(scratch + NOALLOC_BIG);
  a.ctl = g->ctl;
  a.h = 0;
  a.use_cond = 0;
  a.bar_extra = (uint32_t)debug_barrier_extra();
  a.bar_limit = a.bar_extra ? debug_barrier_limit() : PERSIST_WAIT;

  const int32_t iter_cap = o.iter_num > 0 ? (int32_t)std::min<int64_t>(o.iter_num, n + 1) : (int32_t)(n + 1);
  // From the first queued copy on, every return (errors included) waits for the
  // stream: the queued work uses the shared scratch array, and a caller that
  // serialises its calls must find the array idle when a call returns.
  StreamDrain drain{s};
  MG_CUDA_TRY(cudaMemcpyAsync(dsrc, srcs, sizeof(int32_t) * nsrc, cudaMemcpyHostToDevice, s));
  MG_CUDA_TRY(cudaEventRecord(g->ev0, s));
  MG_CUDA_TRY(cudaMemsetAsync(g->ctl, 0, sizeof(DevCtl), s));
  bfs_clear_kernel<<<g->num_sms * 8, 256, 0, s>>>(depth, a.vis, n);
  bfs_seed_kernel<<<1, 1024, 0, s>>>(a, dsrc, nsrc, iter_cap, 0);
  MG_CUDA_TRY(cudaGetLastError());
  const int grid = g->num_sms * g->tune.bfs_ctas_per_sm;
  LoopBody body = [a, grid](cudaStream_t st, cudaGraphConditionalHandle, int) {
    bfs_push_kernel<<<grid, BFS_NT, 0, st>>>(a);
    bfs_push_big_kernel<<<grid, BFS_NT, 0, st>>>(a);
    bfs_pull_kernel<false><<<grid, BFS_NT, 0, st>>>(a);
  };
  MG_TRY(run_loop(g, SLOT_BFS, nullptr, 0, -1, body, n + 2));
  MG_CUDA_TRY(cudaEventRecord(g->ev1, s));
  MG_TRY(fetch_ctl(g));
  const DevCtl &hc = *g->ctl_host;
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->iterations = hc.level;
    stats->edges_traversed = hc.visited_deg;
    stats->edges_inspected = hc.edges_inspected;
    stats->bytes_compulsory = 4 * hc.edges_inspected + 16 * hc.vertices_expanded + 4 * n +
                              (int64_t)hc.levels_pull * ((n + 7) / 8);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    stats->kernel_ms = ms;
    stats->status_detail = hc.levels_pull;
    stats->launches = 2 + 3 * (int64_t)hc.level;
  }
  if (hc.status != 0) {
    mg_set_error("mg_bfs_noalloc: frontier exceeded queue capacity %d", qcap);
    return (mg_status)hc.status;
  }
  return MG_OK;
}

// ---- predecessors of a BFS result ------------------------------------------
// The reference's pred_extract (Algorithms/BFS/predextract.cuh:246-373): over the
// in-edges of every vertex v, the candidate of edge (u, v) is u when
// label[v] - label[u] == 1 and -1 otherwise (gather_edge, :143-155), reduced by max
// (ReduceFunctor, :211-219). Unreached vertices get -1; a source (label 0) gets
// its largest unreached in-neighbour, as in the reference, where the comment calls
// that value arbitrary (Algorithms/BFS/bfs.cu:461). Vertices without in-edges get
// -1. Each lane takes one vertex; in-degrees above 32 are scanned by the warp.
namespace mg {

__global__ void __launch_bounds__(256) bfs_pred_kernel(const int32_t *__restrict__ co, const int32_t *__restrict__ ri,
                                                       const int32_t *__restrict__ label, int64_t n,
                                                       int32_t *__restrict__ pred) {
  const int lane = lane_id();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    const int64_t v = base + threadIdx.x;
    const bool in = v < n;
    const int32_t lv = in ? label[v] : -1;
    const int32_t beg = in ? co[v] : 0, end = in ? co[v + 1] : 0;
    const bool scan = in && lv != -1;  // unreached vertices never match (label -2 does not exist)
    int32_t best = -1;
    const bool small = end - beg <= 32;
    if (scan && small)
      for (int32_t e = beg; e < end; e++) {
        const int32_t u = ri[e];
        if (lv - label[u] == 1) best = max(best, u);
      }
    unsigned pend = __ballot_sync(FULL, scan && !small);
    while (pend) {
      const int l = __ffs(pend) - 1;
      pend &= pend - 1;
      const int32_t b = __shfl_sync(FULL, beg, l), en = __shfl_sync(FULL, end, l), lbl = __shfl_sync(FULL, lv, l);
      int32_t m = -1;
      for (int32_t e = b + lane; e < en; e += 32) {
        const int32_t u = ri[e];
        if (lbl - label[u] == 1) m = max(m, u);
      }
      m = __reduce_max_sync(FULL, m);
      if (lane == l) best = m;
    }
    if (in) pred[v] = best;
  }
}

}  // namespace mg

extern "C" mg_status mg_bfs_predecessors(mg_graph *g, const int32_t *depth, int32_t *pred, const mg_opts *opts) {
  using namespace mg;
  if (!g || !depth || !pred) {
    mg_set_error("mg_bfs_predecessors: null argument");
    return MG_ERR_ARG;
  }
  const int dev_io = opts ? opts->device_output : 0;
  if (!g->has_csc) {
    mg_set_error("mg_bfs_predecessors: the gather over in-edges needs the CSC (graph created with MG_GRAPH_NO_CSC)");
    return MG_ERR_UNSUPPORTED;
  }
  MG_TRY(graph_enter(g));
  if (dev_io) {
    MG_TRY(check_device_ptr(g, depth, "mg_bfs_predecessors", "depth"));
    MG_TRY(check_device_ptr(g, pred, "mg_bfs_predecessors", "pred"));
  }
  const int64_t n = g->n;
  cudaStream_t s = g->stream;
  const int32_t *dlabel = depth;
  int32_t *dpred = pred;
  if (!dev_io) {
    MG_TRY(ws_reserve(g, g->ws_out, Carve::need({sizeof(int32_t) * (size_t)n, sizeof(int32_t) * (size_t)n})));
    Carve cv(g->ws_out.ptr);
    int32_t *l = cv.take<int32_t>(n);
    dpred = cv.take<int32_t>(n);
    MG_CUDA_TRY(cudaMemcpyAsync(l, depth, sizeof(int32_t) * n, cudaMemcpyHostToDevice, s));
    dlabel = l;
  }
  if (n > 0) bfs_pred_kernel<<<g->num_sms * 8, 256, 0, s>>>(g->co, g->ri, dlabel, n, dpred);
  MG_CUDA_TRY(cudaGetLastError());
  if (!dev_io) MG_CUDA_TRY(cudaMemcpyAsync(pred, dpred, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
  MG_CUDA_TRY(cudaStreamSynchronize(s));
  return MG_OK;
}
