// batch.cu -- batched traversals. No reference counterpart: the reference runs
// the whole engine once per source (Algorithms/BFS/bfs.cu:442-456), each run
// with its own context, allocations and per-level host round trips.
//
// mg_bfs_batch: bit-parallel multi-source BFS. Up to 64 sources share one pass
// over the graph. Every vertex carries 64-bit masks: `seen` (sources that have
// reached it), the frontier (sources that reached it in the last level) and, for
// top-down levels, an accumulator of sources arriving in this level. One edge
// read serves all the sources of the group. A level runs either
//   - top-down: the union frontier (vertices with a non-empty frontier mask) is
//     expanded with the degree-binned tile expansion and each edge ORs the
//     sender's frontier mask, minus the sources the receiver has already seen,
//     into the receiver's accumulator; a finishing pass commits the new bits, or
//   - bottom-up: every vertex still missing some source ORs its in-neighbours'
//     frontier masks and stops as soon as every missing source has arrived,
// chosen per level from the out-edges of the union frontier. Depth rows:
// depth[i * n + v] = level at which source i reached v, -1 if never. BFS levels
// are unique, so every row equals a single-source mg_bfs from srcs[i].
//
// mg_bfs_ragged: the members of a ragged batch are disjoint inside the union
// graph, so one multi-source BFS from every member's source (shifted by its
// vertex base) is every member's own BFS, in one device run.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "engine.cuh"
#include "expand.cuh"
#define MG_PRB_NO_PLAN_KERNELS
#include "pr_binned.cuh"

namespace mg {

constexpr int MS_NT = 256;
constexpr int MS_CTA_TH = 512;
constexpr int MS_WIDTH = 64;        // sources per bit-parallel group
constexpr int MS_PLANES = 5;         // digits of the depths kept by vertex
constexpr int MS_FV = 4;             // vertices a thread commits at a time
constexpr int64_t MS_ALPHA = 14;    // bottom-up when the union frontier's out-edges exceed m / MS_ALPHA

struct MsArgs {
  const int32_t *ro, *ci;  // out-edges (CSR)
  const int32_t *co, *ri;  // in-edges (CSC; the CSR itself for symmetric graphs)
  uint64_t *seen, *f0, *f1, *acc;
  int32_t *q0, *q1;
  int32_t qcap;
  int32_t *big_v;  // grid-strided bin (BIG_CAP vertices)
  int32_t *depth;  // the group's first depth row (k rows of n)
  uint64_t *plane[MS_PLANES];  // depths by their binary digits, while the level is below 1 << MS_PLANES
  int64_t n, m_total;
  uint64_t full;   // mask of the group's sources
  int32_t mode, can_pull, both;
  int32_t *grab;   // work counters of the bottom-up passes (reset at the level's end)
  DevCtl *ctl;
  cudaGraphConditionalHandle h;
  int32_t use_cond;
};

__device__ void ms_level_end(const MsArgs &a) {
  DevCtl *c = a.ctl;
  const int cur = vload(&c->cur);
  const int32_t nf = vload(&c->qlen[cur ^ 1]);
  const int64_t mf = vload(&c->mf_next);
  const int lvl = vload(&c->level) + 1;
  c->level = lvl;
  c->qlen[cur] = 0;
  c->cur = cur ^ 1;
  c->mf_front = mf;
  c->mf_next = 0;
  c->blocks_done = 0;
  c->big_len = 0;
  a.grab[0] = 0;
  a.grab[1] = 0;
  const bool over = vload(&c->overflow) != 0;
  const bool done = nf == 0 || lvl >= c->iter_cap || over;
  int dir = 0;
  if (a.mode == MG_DIR_PULL) dir = a.can_pull ? 1 : 0;
  else if (a.mode == MG_DIR_AUTO && a.can_pull) dir = mf * MS_ALPHA > a.m_total ? 1 : 0;
  if (dir == 1 && !done) c->levels_pull += 1;
  c->dir = dir;
  c->nf_next = nf;
  if (over) c->status = MG_ERR_QUEUE_OVERFLOW;
  __threadfence();
  c->done = done ? 1 : 0;
  loop_signal(a.ctl, a.h, a.use_cond, done);
}

// What a level kernel reads from the control block: by one thread per block, since
// every warp of the grid reading one L2 sector queues for microseconds.
struct MsEnter {
  int32_t skip, cur, nin, level;
  int64_t mf;
};

// Early exit of the level kernels: true if the run is over (then it makes sure the loop
// stops) or the level goes the other way (want_dir -1: either way is right). Every
// thread of the block calls it.
__device__ __forceinline__ bool ms_skip(const MsArgs &a, int want_dir, MsEnter &en) {
  DevCtl *c = a.ctl;
  if (threadIdx.x == 0) {
    const int32_t done = vload(&c->done), dir = vload(&c->dir), cur = vload(&c->cur);
    const int32_t q0 = vload(&c->qlen[0]), q1 = vload(&c->qlen[1]);
    en.level = vload(&c->level);
    en.mf = vload(&c->mf_front);
    en.cur = cur;
    en.nin = cur ? q1 : q0;
    en.skip = done || (want_dir >= 0 && dir != want_dir);
    if (done) loop_over(a.ctl, a.h, a.use_cond);
  }
  __syncthreads();
  return en.skip != 0;
}

// Depths while the levels are few (fewer than 1 << MS_PLANES). A level that stores
// its new depths writes each row in pieces, the sector of a row at several levels, and
// the rows had to be set to -1 first (R-MAT s20, 64 sources, 268 MB of rows: 43 us).
// Instead digit b of a vertex's 64 depths is kept in one word, plane[b][v]; a level
// ORs its new bits into the planes of its own digits, and the rows are written once,
// complete, at the end of the run (or at level 1 << MS_PLANES, from where on
// ms_write_depths stores them): 56 us.
__device__ __forceinline__ void ms_plane(const MsArgs &a, int64_t w, uint64_t nw, int32_t d) {
#pragma unroll
  for (int b = 0; b < MS_PLANES; b++) {
    if (d == 1 << b) a.plane[b][w] = nw;  // first level with this digit: no other bit yet
    else if (((d >> b) & 1) && nw) a.plane[b][w] |= nw;
  }
}

// The rows of vertex v, complete: reached (`seen`) sources' depths from the planes of
// levels up to `top`, 1 << MS_PLANES for those in `nw`, -1 for the others. Sources
// i, i + 8, i + 16, i + 24 are decoded at a time, a byte each.
__device__ __forceinline__ void ms_emit_rows(const MsArgs &a, int64_t v, uint64_t seen, uint64_t nw, int32_t top) {
  uint64_t pl[MS_PLANES];
#pragma unroll
  for (int b = 0; b < MS_PLANES; b++) pl[b] = top >> b ? __ldcs(a.plane[b] + v) : 0;
  seen |= nw;
  const int k = 64 - __clzll((long long)a.full);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const unsigned s = (unsigned)(seen >> (32 * h)), w = (unsigned)(nw >> (32 * h));
    unsigned p[MS_PLANES];
#pragma unroll
    for (int b = 0; b < MS_PLANES; b++) p[b] = (unsigned)(pl[b] >> (32 * h));
    const int kh = k - 32 * h;
    int32_t *row = a.depth + (int64_t)(32 * h) * a.n + v;
    for (int i = 0; i < 8 && i < kh; i++, row += a.n) {
      unsigned x = ((w >> i) & 0x01010101u) << MS_PLANES;
#pragma unroll
      for (int b = 0; b < MS_PLANES; b++) x |= ((p[b] >> i) & 0x01010101u) << b;
      x |= (~(s >> i) & 0x01010101u) * 0xffu;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (i + 8 * j < kh) __stcs(row + 8 * j * a.n, (int32_t)(x << (24 - 8 * j)) >> 24);
    }
  }
}

// After the last level: the rows, unless level 1 << MS_PLANES wrote them.
__global__ void __launch_bounds__(MS_NT) ms_rows_kernel(MsArgs a) {
  __shared__ int32_t s_top;
  if (threadIdx.x == 0) s_top = vload(&a.ctl->level);
  __syncthreads();
  const int32_t top = s_top;
  if (top >= 1 << MS_PLANES) return;
  for (int64_t v = (int64_t)blockIdx.x * MS_NT + threadIdx.x; v < a.n; v += (int64_t)gridDim.x * MS_NT)
    ms_emit_rows(a, v, a.seen[v], 0, top);
}

// Writes depth d of every lane's vertex v for each source bit in its `nw`.
// Called by the whole warp (lanes without a vertex pass nw = 0): the warp walks
// the union of its lanes' bits source by source, so the stores of one source go
// to consecutive vertices of one depth row.
__device__ __forceinline__ void ms_write_depths(int32_t *depth, int64_t n, int64_t v, uint64_t nw, int32_t d) {
  const unsigned lo = __reduce_or_sync(FULL, (unsigned)nw), hi = __reduce_or_sync(FULL, (unsigned)(nw >> 32));
  uint64_t any = ((uint64_t)hi << 32) | lo;
  while (any) {
    const int i = __ffsll((long long)any) - 1;
    any &= any - 1;
    if ((nw >> i) & 1) depth[(int64_t)i * n + v] = d;
  }
}

// Top-down expansion of the union frontier into the accumulators.
__global__ void __launch_bounds__(MS_NT) ms_push_kernel(MsArgs a) {
  __shared__ ExpandSmem<MS_NT, uint64_t> sm;
  __shared__ int64_t s_sum[MS_NT / 32 + 1];
  __shared__ MsEnter en;
  if (ms_skip(a, 0, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  const int32_t nin = en.nin;
  const int32_t *qin = cur ? a.q1 : a.q0;
  const uint64_t *fcur = cur ? a.f1 : a.f0;
  const uint64_t *seen = a.seen;
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc);
  const int32_t *ci = a.ci, *ri = a.ri;
  int64_t insp = 0, nexp = 0;
  const BigList big{a.big_v, &c->big_len, defer_threshold<MS_NT>(nin, MS_CTA_TH)};
  auto visit_to = [&](uint64_t f, int32_t w) {
    const uint64_t add = f & ~__ldg(seen + w);
    if (add) atomicOr(acc + w, (unsigned long long)add);
  };
  const int tl = tile_lanes<MS_NT>(nin, en.mf), tn = tl * (MS_NT / 32);
  for (int64_t tile = (int64_t)blockIdx.x * tn; tile < nin; tile += (int64_t)gridDim.x * tn) {
    const int64_t i = tile + warp_id() * tl + lane_id();
    const int32_t v = lane_id() < tl && i < nin ? qin[i] : -1;
    nexp += v >= 0;
    const uint64_t f = v >= 0 ? __ldg(fcur + v) : 0;  // the sender's frontier mask, once per vertex
    expand_tile_p<MS_NT, MS_CTA_TH>(sm, a.ro, v, f, insp,
                                    [&](int32_t, uint64_t fv, int32_t k) { visit_to(fv, ci[k]); }, &big);
    if (a.both)
      expand_tile_p<MS_NT, MS_CTA_TH>(sm, a.co, v, f, insp,
                                      [&](int32_t, uint64_t fv, int32_t k) { visit_to(fv, ri[k]); });
  }
  const int64_t bins = block_sum<MS_NT>(insp, s_sum);
  const int64_t bexp = block_sum<MS_NT>(nexp, s_sum);
  if (threadIdx.x == 0) {
    if (bins) atomicAdd((unsigned long long *)&c->edges_inspected, (unsigned long long)bins);
    if (bexp) atomicAdd((unsigned long long *)&c->vertices_expanded, (unsigned long long)bexp);
  }
}

// Grid-strided bin of a top-down level: the out-edges of the deferred hubs spread
// over every CTA.
__global__ void __launch_bounds__(MS_NT) ms_push_big_kernel(MsArgs a) {
  __shared__ BigSmem<MS_NT> sm;
  __shared__ MsEnter en;
  if (ms_skip(a, 0, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  const uint64_t *fcur = cur ? a.f1 : a.f0;
  const uint64_t *seen = a.seen;
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc);
  const int32_t *ci = a.ci;
  expand_big<MS_NT>(sm, a.ro, BigList{a.big_v, &c->big_len}, [&](int32_t sv, int32_t k) {
    const int32_t w = ci[k];
    const uint64_t add = __ldg(fcur + sv) & ~__ldg(seen + w);
    if (add) atomicOr(acc + w, (unsigned long long)add);
  });
}

// Commits a level: new bits = accumulated & ~seen; rewrites every vertex's
// next-frontier mask and clears the accumulators it read, in vertex order. Latency
// bounds it (three dependent loads per new vertex), so a thread has MS_FV vertices in
// flight and a warp stages its appends. R-MAT s20, 64 sources, the fullest level: 44 us
// with one vertex in flight and an atomic on the queue's length per 32 vertices, 34 us now.
__global__ void __launch_bounds__(MS_NT) ms_finish_kernel(MsArgs a) {
  __shared__ int64_t s_sum[MS_NT / 32 + 1];
  __shared__ int32_t s_stage[MS_NT / 32][WS_CAP];
  __shared__ MsEnter en;
  if (ms_skip(a, -1, en)) return;
  DevCtl *c = a.ctl;
  const int cur = en.cur;
  const int32_t d = en.level + 1;
  uint64_t *fnext = cur ? a.f0 : a.f1;
  int32_t *qout = cur ? a.q0 : a.q1;
  int32_t *qlen_out = &c->qlen[cur ^ 1];
  WarpStage st{s_stage[warp_id()], 0};
  int64_t mf = 0, vdeg = 0;
  const int64_t stride = (int64_t)gridDim.x * MS_NT;
  for (int64_t base = (int64_t)blockIdx.x * MS_NT; base < a.n; base += MS_FV * stride) {
    uint64_t ac[MS_FV], s[MS_FV];
    int32_t r0[MS_FV], r1[MS_FV];
#pragma unroll
    for (int j = 0; j < MS_FV; j++) {
      const int64_t w = base + j * stride + threadIdx.x;
      ac[j] = w < a.n ? a.acc[w] : 0;
    }
#pragma unroll
    for (int j = 0; j < MS_FV; j++) {
      const int64_t w = base + j * stride + threadIdx.x;
      s[j] = ac[j] || (d == 1 << MS_PLANES && w < a.n) ? a.seen[w] : 0;
      r0[j] = ac[j] ? __ldg(a.ro + w) : 0;
      r1[j] = ac[j] ? __ldg(a.ro + w + 1) : 0;
    }
#pragma unroll
    for (int j = 0; j < MS_FV; j++) {
      const int64_t w = base + j * stride + threadIdx.x;
      const uint64_t nw = ac[j] & ~s[j];
      if (w < a.n) {
        if (ac[j]) a.acc[w] = 0;
        if (nw) {
          a.seen[w] = s[j] | nw;
          mf += r1[j] - r0[j];
          vdeg += (int64_t)(r1[j] - r0[j]) * __popcll(nw);
        }
        fnext[w] = nw;
        if (d < 1 << MS_PLANES) ms_plane(a, w, nw, d);
        else if (d == 1 << MS_PLANES) ms_emit_rows(a, w, s[j], nw, d - 1);
      }
      if (d > 1 << MS_PLANES) ms_write_depths(a.depth, a.n, w, nw, d);
      ws_push(st, nw != 0, (int32_t)w, qout, qlen_out, a.qcap, &c->overflow);
    }
  }
  ws_flush(st, qout, qlen_out, a.qcap, &c->overflow);
  const int64_t bmf = block_sum<MS_NT>(mf, s_sum);
  const int64_t bvd = block_sum<MS_NT>(vdeg, s_sum);
  if (threadIdx.x == 0) {
    if (bmf) atomicAdd((unsigned long long *)&c->mf_next, (unsigned long long)bmf);
    if (bvd) atomicAdd((unsigned long long *)&c->visited_deg, (unsigned long long)bvd);
  }
  if (last_block(&c->blocks_done) && threadIdx.x == 0) ms_level_end(a);
}

// Bottom-up pass: every vertex still missing sources ORs its in-neighbours'
// frontier masks into its accumulator and stops once all of them have arrived.
// Vertices come in the degree bins of the gather plan `p` (a lane each up to 64
// in-edges, 8 index loads and 8 masks in flight per step; 4 lanes to 256; then a
// warp; hubs in chunks, which add to the accumulator by atomics). In vertex order,
// with a lane per vertex that calls its warp once it runs long, a few warps walked
// neighbouring hubs one after another, two dependent loads per 32 edges: R-MAT s20,
// 64 sources, 1.48 ms for the first bottom-up level, 0.12 ms with the bins. The
// random mask reads bound it.
// `second`: the out-edges' pass of an undirected run, on top of the first.
__global__ void __launch_bounds__(MS_NT) ms_pull_kernel(MsArgs a, PrbArgs p, int second) {
  __shared__ int64_t s_sum[MS_NT / 32 + 1];
  __shared__ MsEnter en;
  if (ms_skip(a, 1, en)) return;
  DevCtl *c = a.ctl;
  const uint64_t *__restrict__ fcur = en.cur ? a.f1 : a.f0;
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(a.acc);
  int64_t insp = 0, nexp = 0;
  prb_walk(p, [&](auto lanes, int32_t row, int32_t b, int32_t e, int sub, int64_t task, int64_t) {
    constexpr int L = decltype(lanes)::value > 0 ? decltype(lanes)::value : 1;
    uint64_t miss = 0;
    if (row >= 0) {
      miss = a.full & ~a.seen[row];
      // bits an earlier chunk or pass has brought already
      if (miss && (task >= 0 || second)) miss &= ~__ldcg(a.acc + row);
    }
    // The other chunks of a hub add to its accumulator meanwhile, so the lanes may have
    // read different words, and the loop below, which the warp leaves together, ends by it.
    if constexpr (L == 32) miss = __shfl_sync(FULL, miss, 0);
    if (sub == 0 && miss && task < 0 && !second) nexp++;
    if (!miss) e = b;
    uint64_t got = 0;
    for (int32_t k0 = (b & ~7) + 8 * sub; L == 32 ? k0 - 8 * sub < e : k0 < e; k0 += 8 * L) {
      int32_t u[8];
      uint64_t x[8];
      if (k0 < e) prb_load8(p.idx + k0, u);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] = k0 + j >= b && k0 + j < e ? __ldg(fcur + u[j]) : 0ull;
      insp += max(0, min(e, k0 + 8) - max(b, k0));
#pragma unroll
      for (int j = 0; j < 8; j++) got |= x[j];
      if constexpr (L == 32) {
        const unsigned lo = __reduce_or_sync(FULL, (unsigned)got), hi = __reduce_or_sync(FULL, (unsigned)(got >> 32));
        got = ((uint64_t)hi << 32) | lo;
      }
      if ((got & miss) == miss) break;
    }
    if constexpr (L == 4) {
      got |= __shfl_xor_sync(FULL, got, 1);
      got |= __shfl_xor_sync(FULL, got, 2);
    }
    got &= miss;
    if (sub == 0 && got) {
      if (task >= 0) atomicOr(acc + row, (unsigned long long)got);
      else a.acc[row] = second ? a.acc[row] | got : got;
    }
  });
  const int64_t bins = block_sum<MS_NT>(insp, s_sum);
  const int64_t bexp = block_sum<MS_NT>(nexp, s_sum);
  if (threadIdx.x == 0) {
    if (bins) atomicAdd((unsigned long long *)&c->edges_inspected, (unsigned long long)bins);
    if (bexp) atomicAdd((unsigned long long *)&c->vertices_expanded, (unsigned long long)bexp);
  }
}

// Masks := 0.
__global__ void ms_clear_kernel(MsArgs a) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += stride) {
    a.seen[i] = 0;
    a.f0[i] = 0;
    a.f1[i] = 0;
    a.acc[i] = 0;
  }
}

// Seeds the group's sources (bit i for srcs[i]; equal sources share a vertex).
__global__ void ms_seed_kernel(MsArgs a, const int32_t *srcs, int32_t k, int32_t iter_cap, int32_t dir0) {
  __shared__ int64_t s_sum[1024 / 32 + 1];
  DevCtl *c = a.ctl;
  int64_t mf = 0, vdeg = 0;
  unsigned long long *seen = reinterpret_cast<unsigned long long *>(a.seen);
  unsigned long long *f0 = reinterpret_cast<unsigned long long *>(a.f0);
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    const int32_t s = srcs[i];
    const unsigned long long bit = 1ull << i;
    const int64_t deg = a.ro[s + 1] - a.ro[s];
    atomicOr(seen + s, bit);
    vdeg += deg;
    if (atomicOr(f0 + s, bit) == 0ull) {
      mf += deg;
      const int pos = atomicAdd(&c->qlen[0], 1);
      if (pos < a.qcap) a.q0[pos] = s;
      else c->overflow = 1;
    }
  }
  const int64_t tm = block_sum<1024>(mf, s_sum);
  const int64_t tv = block_sum<1024>(vdeg, s_sum);
  if (threadIdx.x == 0) {
    c->visited_deg = tv;
    c->mf_front = tm;
    c->mf_next = 0;
    c->level = 0;
    c->cur = 0;
    int dir = dir0;
    if (a.mode == MG_DIR_AUTO && a.can_pull) dir = tm * MS_ALPHA > a.m_total ? 1 : 0;
    c->dir = dir;
    if (dir == 1) c->levels_pull = 1;
    c->iter_cap = iter_cap;
    c->done = (iter_cap <= 0 || c->overflow) ? 1 : 0;
    if (c->overflow) c->status = MG_ERR_QUEUE_OVERFLOW;
  }
}

}  // namespace mg

// Runs the bit-parallel BFS of every group of up to 64 sources into `depth`
// (device, nsrc x n).
static mg_status msbfs_run(mg_graph *g, const int32_t *srcs, int32_t nsrc, int32_t *depth, const mg_opts &o,
                           mg_stats *stats) {
  using namespace mg;
  const bool symmetric = (g->flags & MG_GRAPH_SYMMETRIC) != 0;
  const bool undirected = o.directed == 0 && !symmetric;
  if (undirected && !g->has_csc) {
    mg_set_error("mg_bfs_batch: directed=0 needs the CSC (graph created with MG_GRAPH_NO_CSC)");
    return MG_ERR_UNSUPPORTED;
  }
  const int64_t n = g->n;
  const size_t need = Carve::need({sizeof(uint64_t) * (size_t)n, sizeof(uint64_t) * (size_t)n,
                                   sizeof(uint64_t) * (size_t)n, sizeof(uint64_t) * (size_t)n,
                                   sizeof(int32_t) * (size_t)n, sizeof(int32_t) * (size_t)n,
                                   sizeof(int32_t) * (size_t)BIG_CAP, sizeof(int32_t) * (size_t)nsrc,
                                   sizeof(int32_t) * 2, sizeof(uint64_t) * (size_t)n * MS_PLANES});
  MG_TRY(ws_reserve(g, g->ws_main, need));
  Carve cv(g->ws_main.ptr);
  MsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.seen = cv.take<uint64_t>(n);
  a.f0 = cv.take<uint64_t>(n);
  a.f1 = cv.take<uint64_t>(n);
  a.acc = cv.take<uint64_t>(n);
  a.q0 = cv.take<int32_t>(n);
  a.q1 = cv.take<int32_t>(n);
  a.big_v = cv.take<int32_t>(BIG_CAP);
  int32_t *dsrc = cv.take<int32_t>(nsrc);
  a.grab = cv.take<int32_t>(2);
  uint64_t *planes = cv.take<uint64_t>(n * MS_PLANES);
  for (int b = 0; b < MS_PLANES; b++) a.plane[b] = planes + b * n;
  a.qcap = (int32_t)n;
  a.ro = g->ro;
  a.ci = g->ci;
  a.co = g->has_csc ? g->co : g->ro;
  a.ri = g->has_csc ? g->ri : g->ci;
  a.n = n;
  a.m_total = g->m;
  a.mode = o.direction;
  a.can_pull = g->has_csc || symmetric;
  a.both = undirected ? 1 : 0;
  // bottom-up levels walk the gather plan of the in-edges (then of the out-edges)
  const bool pull = a.can_pull && o.direction != MG_DIR_PUSH;
  PrbArgs pin, pout;
  std::memset(&pin, 0, sizeof(pin));
  std::memset(&pout, 0, sizeof(pout));
  if (pull) {
    MG_TRY(graph_bin_plan(g, !g->has_csc, &pin));
    pin.grab = a.grab;
    if (undirected) {
      MG_TRY(graph_bin_plan(g, true, &pout));
      pout.grab = a.grab + 1;
    }
  }
  a.ctl = g->ctl;
  cudaStream_t s = g->stream;
  const int32_t iter_cap = o.iter_num > 0 ? (int32_t)std::min<int64_t>(o.iter_num, n + 1) : (int32_t)(n + 1);
  const int32_t dir0 = (o.direction == MG_DIR_PULL && a.can_pull) ? 1 : 0;
  MG_CUDA_TRY(cudaMemcpyAsync(dsrc, srcs, sizeof(int32_t) * nsrc, cudaMemcpyHostToDevice, s));
  MG_CUDA_TRY(cudaMemsetAsync(a.grab, 0, sizeof(int32_t) * 2, s));
  const int grid = g->num_sms * 4;
  int64_t iters = 0, vdeg = 0, insp = 0, launches = 0, pulls = 0;
  float ms_total = 0.f;
  for (int32_t g0 = 0; g0 < nsrc; g0 += MS_WIDTH) {
    const int32_t k = std::min<int32_t>(MS_WIDTH, nsrc - g0);
    a.depth = depth + (int64_t)g0 * n;
    a.full = k == 64 ? ~0ull : ((1ull << k) - 1);
    MG_CUDA_TRY(cudaEventRecord(g->ev0, s));
    MG_CUDA_TRY(cudaMemsetAsync(g->ctl, 0, sizeof(DevCtl), s));
    ms_clear_kernel<<<g->num_sms * 8, 256, 0, s>>>(a);
    ms_seed_kernel<<<1, 1024, 0, s>>>(a, dsrc + g0, k, iter_cap, dir0);
    MG_CUDA_TRY(cudaGetLastError());
    struct Sig {
      MsArgs a;
      PrbArgs pin, pout;
      int grid;
    } sig;
    std::memset(&sig, 0, sizeof(sig));
    sig.a = a;
    sig.pin = pin;
    sig.pout = pout;
    sig.grid = grid;
    LoopBody body = [a, pin, pout, pull, grid](cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) {
      MsArgs b = a;
      b.h = h;
      b.use_cond = use_cond;
      ms_push_kernel<<<grid, MS_NT, 0, st>>>(b);
      ms_push_big_kernel<<<grid, MS_NT, 0, st>>>(b);
      if (pull) ms_pull_kernel<<<grid, MS_NT, 0, st>>>(b, pin, 0);
      if (pull && b.both) ms_pull_kernel<<<grid, MS_NT, 0, st>>>(b, pout, 1);
      ms_finish_kernel<<<grid, MS_NT, 0, st>>>(b);
    };
    MG_TRY(run_loop(g, SLOT_MSBFS, &sig, sizeof(sig), o.use_graph, body, n + 2));
    ms_rows_kernel<<<g->num_sms * 8, MS_NT, 0, s>>>(a);
    MG_CUDA_TRY(cudaGetLastError());
    MG_CUDA_TRY(cudaEventRecord(g->ev1, s));
    MG_TRY(fetch_ctl(g));
    const DevCtl &hc = *g->ctl_host;
    if (hc.status != 0) {
      mg_set_error("mg_bfs_batch: device status %d", hc.status);
      return (mg_status)hc.status;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    ms_total += ms;
    iters = std::max<int64_t>(iters, hc.level);
    vdeg += hc.visited_deg;
    insp += hc.edges_inspected;
    pulls += hc.levels_pull;
    const int64_t per = 3 + (pull ? 1 + a.both : 0);
    launches += 3 + loop_launches(g, per);
  }
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->iterations = iters;
    stats->edges_traversed = vdeg;
    stats->edges_inspected = insp;
    stats->bytes_compulsory = 12 * insp + 40 * n * iters + 4 * (int64_t)nsrc * n;
    stats->kernel_ms = ms_total;
    stats->status_detail = (int32_t)pulls;
    stats->launches = launches;
  }
  return MG_OK;
}

extern "C" mg_status mg_bfs_batch(mg_graph *g, const int32_t *srcs, int32_t nsrc, int32_t *depth,
                                  const mg_opts *opts, mg_stats *stats) {
  if (!g || !srcs || nsrc <= 0 || !depth) {
    mg_set_error("mg_bfs_batch: null argument or nsrc <= 0");
    return MG_ERR_ARG;
  }
  mg_opts o;
  std::memset(&o, 0, sizeof(o));
  o.directed = 1;
  if (opts) o = *opts;
  if (o.direction < MG_DIR_AUTO || o.direction > MG_DIR_PULL) {
    mg_set_error("mg_bfs_batch: invalid direction %d", o.direction);
    return MG_ERR_ARG;
  }
  for (int32_t i = 0; i < nsrc; i++) {
    if (srcs[i] < 0 || srcs[i] >= g->n) {
      mg_set_error("mg_bfs_batch: source %d out of range [0, %lld)", srcs[i], (long long)g->n);
      return MG_ERR_ARG;
    }
  }
  MG_TRY(graph_enter(g));
  if (o.device_output) MG_TRY(check_device_ptr(g, depth, "mg_bfs_batch", "depth"));
  const size_t bytes = sizeof(int32_t) * (size_t)nsrc * (size_t)g->n;
  int32_t *out = depth;
  if (!o.device_output) {
    MG_TRY(ws_reserve(g, g->ws_out, bytes + 256));
    out = (int32_t *)g->ws_out.ptr;
  }
  MG_TRY(msbfs_run(g, srcs, nsrc, out, o, stats));
  if (!o.device_output) {
    MG_TRY(copy_out(g, depth, out, bytes, 0));
    MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
  }
  return MG_OK;
}

extern "C" mg_status mg_bfs_ragged(mg_graph *g, const int32_t *srcs, int32_t *depth, const mg_opts *opts,
                                   mg_stats *stats) {
  if (!g || !srcs || !depth) {
    mg_set_error("mg_bfs_ragged: null argument");
    return MG_ERR_ARG;
  }
  if (g->vbase.size() < 2) {
    mg_set_error("mg_bfs_ragged: the graph is not a ragged batch (create it with mg_graph_create_ragged)");
    return MG_ERR_ARG;
  }
  const int32_t ng = (int32_t)g->vbase.size() - 1;
  std::vector<int32_t> global(ng);
  for (int32_t i = 0; i < ng; i++) {
    const int64_t ni = g->vbase[i + 1] - g->vbase[i];
    if (srcs[i] < 0 || srcs[i] >= ni) {
      mg_set_error("mg_bfs_ragged: source %d of member graph %d out of range [0, %lld)", srcs[i], i,
                   (long long)ni);
      return MG_ERR_ARG;
    }
    global[i] = (int32_t)(g->vbase[i] + srcs[i]);
  }
  return mg_bfs(g, global.data(), ng, depth, opts, stats);
}
