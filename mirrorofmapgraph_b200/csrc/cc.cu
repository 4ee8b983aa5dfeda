// cc.cu -- connected components (struct cc, Algorithms/CC/cc.h:32-349).
//
// The reference propagates minimum labels: every vertex starts with its own id
// (SequenceKernel, cc.h:118-120) and each iteration pushes a neighbour's smaller
// label through atomicMin, over CSR and CSC (the driver forces directed = 0,
// Algorithms/CC/cc.cu:289), until nothing changes. The fixed point labels every
// vertex with the smallest id in its weakly connected component.
//
// Here the same labels come from union-find, where hooking always links the
// larger root under the smaller one with atomicCAS: parent pointers only
// decrease, so every root is its component's minimum and the final labels equal
// the reference's bit for bit. The edge work follows the sampling scheme of
// Afforest (Sutton et al., IPDPS 2018): a cheap forest over a few edges of every
// vertex first, and only what lies outside its largest tree walks all its edges.
// The forest needs no union to succeed, so it is built without compare-and-swap:
//   1. every vertex points at the smallest of itself and its first CC_FIRST
//      neighbours, then the trees are compressed;
//   2. 1 + mg_tuning.cc_rounds passes (one more on sparse graphs) over CC_HOOK
//      neighbours each, from the row's start again (by default the first four, which
//      step 1 took the smallest of), hook the larger of the two roots under the
//      smaller one by a fire-and-forget minimum, each followed by a compression; a
//      root hooked twice keeps the smaller link;
//   3. one CTA samples 1024 vertices and takes the most frequent root c (on
//      power-law graphs, the giant component);
//   4. only vertices outside c unite all their edges (and, without a symmetric
//      adjacency, their in-edges too), by union-find; then compress.
// Any edge with both endpoints skipped joins two members of c's tree already, so
// the result does not depend on the sample or on the forest.
#include <algorithm>
#include <climits>
#include <cstring>

#include "common.cuh"
#include "engine.cuh"
#include "expand.cuh"

namespace mg {

constexpr int CC_NT = 256;
constexpr int CC_CTA_TH = 1024;
constexpr int CC_SAMPLES = 1024;
constexpr int CC_V = 4;      // vertices a thread holds in flight
constexpr int CC_FIRST = 4;  // neighbours the first forest looks at
constexpr int CC_HOOK = 2;   // neighbours a hooking pass looks at

// Root of x with path halving. Parent entries are read from L2 (ld.cg): they are
// rewritten concurrently, and every value ever stored is an ancestor, so a
// racing read is still a valid step towards the root.
__device__ __forceinline__ int32_t uf_find(int32_t *p, int32_t x) {
  int32_t par = __ldcg(p + x);
  while (par != x) {
    const int32_t gp = __ldcg(p + par);
    if (gp != par) __stcg(p + x, gp);
    x = par;
    par = gp;
  }
  return x;
}

// Unites the trees of a and b. Two vertices with the same parent are in one tree
// already: after a compression that is nearly every edge, and it costs two loads
// where two finds cost four.
__device__ __forceinline__ void uf_union(int32_t *p, int32_t a, int32_t b) {
  int32_t ra = __ldcg(p + a), rb = __ldcg(p + b);
  if (ra == rb) return;
  ra = uf_find(p, ra);
  rb = uf_find(p, rb);
  while (ra != rb) {
    const int32_t hi = max(ra, rb), lo = min(ra, rb);
    const int32_t old = atomicCAS(p + hi, hi, lo);
    if (old == hi) return;
    // hi was hooked meanwhile; continue from its new root.
    ra = uf_find(p, old);
    rb = uf_find(p, lo);
  }
}

__global__ void cc_init_kernel(int32_t *p, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = (int32_t)i;
}

// The first forest: p[v] = min(v, v's first CC_FIRST neighbours). Every vertex
// writes only its own entry and pointers decrease, so there is no atomic and no
// cycle. Counts the edges that it and the hooking passes (hook_reads of every vertex
// that has any) read.
__global__ void __launch_bounds__(CC_NT) cc_first_kernel(const int32_t *__restrict__ ro,
                                                         const int32_t *__restrict__ ci, int64_t n, int32_t *p,
                                                         int hook_reads, unsigned long long *insp_out) {
  __shared__ int32_t s_insp[CC_NT / 32];
  int32_t insp = 0;  // a block's share of the vertices keeps within 32 bits
  for (int64_t v = (int64_t)blockIdx.x * CC_NT + threadIdx.x; v < n; v += (int64_t)gridDim.x * CC_NT) {
    const int32_t b = ro[v], e = ro[v + 1];
    int32_t mn = (int32_t)v;
#pragma unroll
    for (int k = 0; k < CC_FIRST; k++)
      if (b + k < e) mn = min(mn, ci[b + k]);
    p[v] = mn;
    if (b < e) insp += min(e - b, CC_FIRST) + hook_reads;
  }
  insp = __reduce_add_sync(FULL, insp);
  if (lane_id() == 0) s_insp[warp_id()] = insp;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < CC_NT / 32; w++) insp += s_insp[w];
    if (insp) atomicAdd(insp_out, (unsigned long long)insp);
  }
}

// Hooking pass over neighbours r0 .. r0 + CC_HOOK - 1 of every vertex, counted round
// its row (a root keeps one of the links that a pass finds for it, so a short row's
// neighbours are worth a second look), on compressed trees. Bound by its random parent
// reads. With atomicCAS unions in its place (one neighbour each) the sampled roots are few and hot: R-MAT s22, rows in edge-list
// order, 466 us from singletons and 737 us from the first forest; two passes of
// this kernel and the whole run take 300 us.
// Rows whose first neighbours are arbitrary need the minimum to spread: from
// singletons one round leaves 42-58% of an R-MAT graph's edges outside the largest
// tree (every one walked by the last pass, 10 ms at s22), the first forest and one
// hooking pass 0.4%, two passes nothing but the small components.
__global__ void __launch_bounds__(CC_NT) cc_hook_kernel(const int32_t *__restrict__ ro,
                                                        const int32_t *__restrict__ ci, int64_t n, int32_t *p,
                                                        int r0) {
  for (int64_t v = (int64_t)blockIdx.x * CC_NT + threadIdx.x; v < n; v += (int64_t)gridDim.x * CC_NT) {
    const int32_t b = ro[v], len = ro[v + 1] - b;
    if (len == 0) continue;
    const int32_t pv = __ldcg(p + v);
    int32_t pu[CC_HOOK];
#pragma unroll
    for (int k = 0; k < CC_HOOK; k++) pu[k] = __ldca(p + ci[b + (r0 + k < len ? r0 + k : (r0 + k) % len)]);
#pragma unroll
    for (int k = 0; k < CC_HOOK; k++) {
      const int32_t hi = max(pv, pu[k]), lo = min(pv, pu[k]);
      if (lo < __ldca(p + hi) && lo < __ldcg(p + hi)) red_min(p + hi, lo);
    }
  }
}

// Points every vertex at its root (into p, or into label for the final pass).
// CC_V independent walks per thread, with path halving on the way: the first
// forest of a lattice is chains as long as a column. Parents are read through L1:
// a stale one is an older ancestor, roots do not change here, and nearly every
// walk ends at the same root, whose one L2 sector 130,000 warps would queue for
// (the last pass on R-MAT s22 43 us from L2).
__global__ void __launch_bounds__(CC_NT) cc_compress_kernel(int32_t *p, int32_t *label, int64_t n) {
  for (int64_t t0 = (int64_t)blockIdx.x * CC_NT * CC_V; t0 < n; t0 += (int64_t)gridDim.x * CC_NT * CC_V) {
    int32_t par[CC_V], gp[CC_V];
#pragma unroll
    for (int k = 0; k < CC_V; k++) {
      const int64_t i = t0 + k * CC_NT + threadIdx.x;
      par[k] = i < n ? __ldcg(p + i) : 0;
    }
#pragma unroll
    for (int k = 0; k < CC_V; k++) gp[k] = __ldca(p + par[k]);
#pragma unroll
    for (int k = 0; k < CC_V; k++) {
      const int64_t i = t0 + k * CC_NT + threadIdx.x;
      if (i >= n) continue;
      const int32_t r = gp[k] == par[k] ? par[k] : uf_find(p, gp[k]);
      if (label) label[i] = r;
      else if (r != par[k]) __stcg(p + i, r);
    }
  }
}

// Most frequent root among CC_SAMPLES hashed vertices (one CTA of CC_SAMPLES
// threads), counted in an open-addressed table in shared memory; writes it to *out.
__global__ void __launch_bounds__(CC_SAMPLES) cc_mode_kernel(const int32_t *p, int64_t n, int32_t *out) {
  __shared__ int32_t key[2 * CC_SAMPLES], cnt[2 * CC_SAMPLES];
  __shared__ unsigned long long best;
  const int t = threadIdx.x;
  for (int i = t; i < 2 * CC_SAMPLES; i += CC_SAMPLES) {
    key[i] = -1;
    cnt[i] = 0;
  }
  if (t == 0) best = 0ull;
  uint64_t h = (uint64_t)t * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
  h ^= h >> 31;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 29;
  const int32_t r = __ldcg(p + (int64_t)(h % (uint64_t)n));
  __syncthreads();
  // lanes with the same root add once
  const unsigned same = __match_any_sync(FULL, r);
  const bool lead = (same & lanemask_lt()) == 0;
  if (lead) {
    unsigned at = ((unsigned)r * 2654435761u) >> 21;  // 2048 slots for at most 1024 keys
    for (;;) {
      const int32_t k = atomicCAS(key + at, -1, r);
      if (k == -1 || k == r) break;
      at = (at + 1) & (2 * CC_SAMPLES - 1);
    }
    atomicAdd(cnt + at, __popc(same));
  }
  __syncthreads();
  for (int i = t; i < 2 * CC_SAMPLES; i += CC_SAMPLES)
    if (cnt[i] > 0)  // larger count first, then the smaller root
      atomicMax(&best, ((unsigned long long)cnt[i] << 32) | (unsigned)(INT_MAX - key[i]));
  __syncthreads();
  if (t == 0) *out = INT_MAX - (int32_t)(best & 0xffffffffu);
}

// Phase 4: every vertex whose root is not c unites all its edges (all in-edges
// too when `both`). A CTA looks at CC_NT x CC_V vertices at a time and gathers the
// few that are outside c and have edges before it expands them.
__global__ void __launch_bounds__(CC_NT) cc_finish_kernel(const int32_t *__restrict__ ro,
                                                          const int32_t *__restrict__ ci,
                                                          const int32_t *__restrict__ co,
                                                          const int32_t *__restrict__ ri, int64_t n, int32_t *p,
                                                          const int32_t *cptr, int both,
                                                          unsigned long long *insp_out) {
  __shared__ ExpandSmem<CC_NT> sm;
  __shared__ int64_t s_sum[CC_NT / 32 + 1];
  __shared__ int32_t s_list[CC_NT * CC_V], s_len;
  const int32_t c = *cptr;
  int64_t insp = 0;
  for (int64_t t0 = (int64_t)blockIdx.x * CC_NT * CC_V; t0 < n; t0 += (int64_t)gridDim.x * CC_NT * CC_V) {
    if (threadIdx.x == 0) s_len = 0;
    __syncthreads();
    int32_t par[CC_V];
#pragma unroll
    for (int k = 0; k < CC_V; k++) {
      const int64_t i = t0 + k * CC_NT + threadIdx.x;
      par[k] = i < n ? __ldcg(p + i) : c;
    }
#pragma unroll
    for (int k = 0; k < CC_V; k++) {
      const int64_t i = t0 + k * CC_NT + threadIdx.x;
      if (par[k] != c && (ro[i + 1] > ro[i] || (both && co[i + 1] > co[i])))
        s_list[atomicAdd(&s_len, 1)] = (int32_t)i;
    }
    __syncthreads();
    const int32_t len = s_len;
    for (int32_t l0 = 0; l0 < len; l0 += CC_NT) {
      const int32_t v = l0 + threadIdx.x < len ? s_list[l0 + threadIdx.x] : -1;
      expand_tile<CC_NT, CC_CTA_TH>(sm, ro, v, insp, [&](int32_t sv, int32_t k) {
        const int32_t u = ci[k];
        if (u != sv) uf_union(p, sv, u);
      });
      if (both)
        expand_tile<CC_NT, CC_CTA_TH>(sm, co, v, insp, [&](int32_t sv, int32_t k) {
          const int32_t u = ri[k];
          if (u != sv) uf_union(p, sv, u);
        });
    }
    __syncthreads();
  }
  const int64_t b = block_sum<CC_NT>(insp, s_sum);
  if (threadIdx.x == 0 && b) atomicAdd(insp_out, (unsigned long long)b);
}

// Without a usable transpose: every edge once.
__global__ void __launch_bounds__(CC_NT) cc_all_edges_kernel(const int32_t *__restrict__ ro,
                                                             const int32_t *__restrict__ ci, int64_t n, int32_t *p,
                                                             unsigned long long *insp_out) {
  __shared__ ExpandSmem<CC_NT> sm;
  __shared__ int64_t s_sum[CC_NT / 32 + 1];
  int64_t insp = 0;
  for (int64_t tile = (int64_t)blockIdx.x * CC_NT; tile < n; tile += (int64_t)gridDim.x * CC_NT) {
    const int64_t i = tile + threadIdx.x;
    const int32_t v = i < n ? (int32_t)i : -1;
    expand_tile<CC_NT, CC_CTA_TH>(sm, ro, v, insp, [&](int32_t sv, int32_t k) {
      const int32_t u = ci[k];
      if (u != sv) uf_union(p, sv, u);
    });
  }
  const int64_t b = block_sum<CC_NT>(insp, s_sum);
  if (threadIdx.x == 0 && b) atomicAdd(insp_out, (unsigned long long)b);
}

}  // namespace mg

extern "C" mg_status mg_cc(mg_graph *g, int32_t *label, const mg_opts *opts, mg_stats *stats) {
  using namespace mg;
  if (!g || !label) {
    mg_set_error("mg_cc: null argument");
    return MG_ERR_ARG;
  }
  mg_opts o;
  std::memset(&o, 0, sizeof(o));
  if (opts) o = *opts;
  MG_TRY(graph_enter(g));
  if (o.device_output) MG_TRY(check_device_ptr(g, label, "mg_cc", "label"));
  const int64_t n = g->n;
  const size_t need = Carve::need({sizeof(int32_t) * (size_t)n, sizeof(int32_t) * (size_t)n, 64});
  MG_TRY(ws_reserve(g, g->ws_main, need));
  Carve cv(g->ws_main.ptr);
  int32_t *parent = cv.take<int32_t>(n);
  int32_t *lab_ws = cv.take<int32_t>(n);
  int32_t *cmode = cv.take<int32_t>(16);
  int32_t *out = o.device_output ? label : lab_ws;
  cudaStream_t s = g->stream;
  const bool symmetric = (g->flags & MG_GRAPH_SYMMETRIC) != 0;
  const bool sampling = symmetric || g->has_csc;
  unsigned long long *insp = reinterpret_cast<unsigned long long *>(&g->ctl->edges_inspected);
  MG_CUDA_TRY(cudaMemsetAsync(g->ctl, 0, sizeof(DevCtl), s));
  MG_CUDA_TRY(cudaEventRecord(g->ev0, s));
  const int grid = g->num_sms * 8;
  int64_t launches = 0;
  // Hooking passes beyond the first before the giant component is picked; every
  // count gives the same labels.
  // With 4 neighbours or fewer on average two passes leave most vertices outside the
  // largest tree, and their edges to compare-and-swap unions (random graph, mean degree
  // 2: 97% of the vertices after two passes, 20% after three, nearly all of them in other
  // components; n = 912,385: 775 us with two passes and no second look, 220 us now).
  const int32_t rounds = g->tune.cc_rounds + (g->m <= 4 * n ? 1 : 0);
  const int64_t per = (int64_t)CC_NT * CC_V;
  const int gv = (int)std::min<int64_t>(std::max<int64_t>((n + per - 1) / per, 1), g->num_sms * 8);
  if (n > 0 && sampling) {
    cc_first_kernel<<<grid, CC_NT, 0, s>>>(g->ro, g->ci, n, parent, CC_HOOK * (rounds + 1), insp);
    cc_compress_kernel<<<gv, CC_NT, 0, s>>>(parent, nullptr, n);
    for (int r = 0; r <= rounds; r++) {
      cc_hook_kernel<<<grid, CC_NT, 0, s>>>(g->ro, g->ci, n, parent, r * CC_HOOK);
      cc_compress_kernel<<<gv, CC_NT, 0, s>>>(parent, nullptr, n);
    }
    cc_mode_kernel<<<1, CC_SAMPLES, 0, s>>>(parent, n, cmode);
    cc_finish_kernel<<<gv, CC_NT, 0, s>>>(g->ro, g->ci, g->co, g->ri, n, parent, cmode, symmetric ? 0 : 1, insp);
    launches += 2 * rounds + 6;
  } else if (n > 0) {
    cc_init_kernel<<<grid, 256, 0, s>>>(parent, n);
    cc_all_edges_kernel<<<g->num_sms * 4, CC_NT, 0, s>>>(g->ro, g->ci, n, parent, insp);
    launches += 2;
  }
  cc_compress_kernel<<<gv, CC_NT, 0, s>>>(parent, out, n);
  launches++;
  MG_CUDA_TRY(cudaGetLastError());
  MG_CUDA_TRY(cudaEventRecord(g->ev1, s));
  if (!o.device_output) MG_TRY(copy_out(g, label, out, sizeof(int32_t) * n, 0));
  MG_TRY(fetch_ctl(g));
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->iterations = 1;
    stats->edges_traversed = g->m;
    stats->edges_inspected = g->ctl_host->edges_inspected;
    // offsets and sampled neighbours, the remaining edges actually read, parent
    // init / compress passes
    stats->bytes_compulsory = 4 * (n + 1) + 4 * stats->edges_inspected + 16 * n;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    stats->kernel_ms = ms;
    stats->launches = launches;
  }
  return MG_OK;
}
