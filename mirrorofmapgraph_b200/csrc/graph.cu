// graph.cu -- device graph storage: upload, validation and the CSC build.
//
// Replaces CsrProblem::FromHostProblem (GASengine/csr_problem.cuh:401-621) and
// its thrust CSC build (util.cuh:55-126). Layout in HBM, all int32:
//   CSR  row_offsets[n+1], col_idx[m], values[m] (int32 or float)
//   CSC  col_offsets[n+1], row_idx[m], perm[m] (CSC slot -> CSR edge id),
//        cvals[m] (values already permuted, so in-edge kernels read them
//        sequentially instead of through perm)
// The CSC is built on the device by a stable radix sort of the edges by column,
// which makes it identical to the reference's stable sort by column (within a
// column, edges in CSR order) and therefore deterministic.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "mg_internal.h"

namespace {
thread_local char g_err[1024] = "";
}

void mg_set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

// Test hooks: host-side fault injection (no device fault is ever caused).
// g_fail_alloc: 0 off; k > 0: the k-th allocation from now and every later one
// fail (until the hook is disarmed), so no retry can mask the failure.
static std::atomic<int64_t> g_fail_alloc{0};
static std::atomic<int32_t> g_bar_extra{0};
static std::atomic<unsigned long long> g_bar_limit{1ull << 12};

cudaError_t mg_malloc_async(void **p, size_t bytes, cudaStream_t s) {
  int64_t k = g_fail_alloc.load();
  while (k > 1 && !g_fail_alloc.compare_exchange_weak(k, k - 1)) {
  }
  if (k == 1) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMallocAsync(p, bytes, s);
}

int32_t debug_barrier_extra() { return g_bar_extra.load(); }
unsigned long long debug_barrier_limit() { return g_bar_limit.load(); }

extern "C" mg_status mg_graph_sync(mg_graph *g) {
  if (!g) {
    mg_set_error("mg_graph_sync: null graph");
    return MG_ERR_ARG;
  }
  MG_TRY(graph_enter(g));
  MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
  return MG_OK;
}

extern "C" void mg_tuning_defaults(mg_tuning *t) {
  if (t) *t = tuning_defaults();
}

extern "C" mg_status mg_graph_get_tuning(mg_graph *g, mg_tuning *t) {
  if (!g || !t) {
    mg_set_error("mg_graph_get_tuning: null argument");
    return MG_ERR_ARG;
  }
  *t = g->tune;
  return MG_OK;
}

extern "C" mg_status mg_graph_set_tuning(mg_graph *g, const mg_tuning *t) {
  if (!g || !t) {
    mg_set_error("mg_graph_set_tuning: null argument");
    return MG_ERR_ARG;
  }
  struct Range {
    const char *name;
    int32_t v, lo, hi;
  } const r[] = {{"sssp_heavy", t->sssp_heavy, 1, 1 << 30},
                 {"sssp_heavy_small", t->sssp_heavy_small, 1, t->sssp_heavy},
                 {"sssp_ctas_per_sm", t->sssp_ctas_per_sm, 1, 8},
                 {"sssp_chunk_cap", t->sssp_chunk_cap, 0, 1 << 30},
                 {"sssp_batch_heavy", t->sssp_batch_heavy, 1, 1 << 30},
                 {"bfs_cta_th", t->bfs_cta_th, 32, 1 << 30},
                 {"bfs_grid_th", t->bfs_grid_th, 32, 1 << 30},
                 {"bfs_defer_warp", t->bfs_defer_warp, 0, 1},
                 {"bfs_persist_max", t->bfs_persist_max, 0, 1 << 30},
                 {"bfs_persist_edges", t->bfs_persist_edges, 0, 1 << 30},
                 {"bfs_alpha", t->bfs_alpha, 1, 1 << 20},
                 {"bfs_beta", t->bfs_beta, 1, 1 << 20},
                 {"bfs_sparse_degree", t->bfs_sparse_degree, 0, 1 << 20},
                 {"bfs_ctas_per_sm", t->bfs_ctas_per_sm, 1, 8},
                 {"bfs_tail_max", t->bfs_tail_max, 0, 1 << 30},
                 {"bfs_tail_edges", t->bfs_tail_edges, 0, 1 << 30},
                 {"cc_rounds", t->cc_rounds, 0, 8}};
  for (const Range &x : r) {
    if (x.v < x.lo || x.v > x.hi) {
      mg_set_error("mg_graph_set_tuning: %s = %d outside [%d, %d]", x.name, x.v, x.lo, x.hi);
      return MG_ERR_ARG;
    }
  }
  g->tune = *t;
  return MG_OK;
}

extern "C" mg_status mg_graph_trace(mg_graph *g, mg_level_record *out, int32_t cap, int32_t *count) {
  if (!g || !count || (cap > 0 && !out)) {
    mg_set_error("mg_graph_trace: null argument");
    return MG_ERR_ARG;
  }
  MG_TRY(graph_enter(g));
  int32_t len = 0;
  MG_CUDA_TRY(cudaMemcpyAsync(&len, &g->ctl->trace_len, sizeof(int32_t), cudaMemcpyDeviceToHost, g->stream));
  MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
  len = std::max(0, std::min(std::min(len, (int32_t)MG_TRACE_LEVELS), std::max(cap, 0)));
  if (len > 0)
    MG_CUDA_TRY(cudaMemcpyAsync(out, trace_of(g->ctl), sizeof(mg_level_record) * (size_t)len, cudaMemcpyDeviceToHost,
                                g->stream));
  MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
  *count = len;
  return MG_OK;
}

extern "C" mg_status mg_debug_fail_alloc(int64_t k) {
  if (k < 0) {
    mg_set_error("mg_debug_fail_alloc: k must be >= 0");
    return MG_ERR_ARG;
  }
  g_fail_alloc.store(k);
  return MG_OK;
}

extern "C" mg_status mg_debug_barrier_skew(int32_t extra, int64_t poll_limit) {
  if (extra < 0 || poll_limit <= 0) {
    mg_set_error("mg_debug_barrier_skew: extra must be >= 0 and poll_limit > 0");
    return MG_ERR_ARG;
  }
  g_bar_extra.store(extra);
  g_bar_limit.store((unsigned long long)poll_limit);
  return MG_OK;
}

mg_status dev_alloc(mg_graph *g, void **p, size_t bytes) {
  *p = nullptr;
  cudaError_t e = mg_malloc_async(p, std::max<size_t>(bytes, 1), g->stream);
  if (e == cudaErrorMemoryAllocation) {
    // Return the pool's idle blocks to the driver and try once more.
    cudaGetLastError();
    cudaMemPool_t pool;
    if (cudaStreamSynchronize(g->stream) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, g->device) == cudaSuccess)
      cudaMemPoolTrimTo(pool, 0);
    cudaGetLastError();
    e = mg_malloc_async(p, std::max<size_t>(bytes, 1), g->stream);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    mg_set_error("device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? MG_ERR_OOM : MG_ERR_CUDA;
  }
  return MG_OK;
}

void dev_free(mg_graph *g, void *p) {
  if (p) cudaFreeAsync(p, g->stream);
}

mg_status ws_reserve(mg_graph *g, Workspace &w, size_t bytes) {
  if (w.bytes >= bytes) return MG_OK;
  dev_free(g, w.ptr);
  w.ptr = nullptr;
  const size_t grown = std::max(bytes, w.bytes + w.bytes / 4);
  w.bytes = 0;
  if (dev_alloc(g, &w.ptr, grown) != MG_OK) {
    mg_status st = dev_alloc(g, &w.ptr, bytes);
    if (st != MG_OK) {
      mg_set_error("workspace allocation of %zu bytes failed", bytes);
      return st;
    }
    w.bytes = bytes;
    return MG_OK;
  }
  w.bytes = grown;
  return MG_OK;
}

mg_status graph_enter(mg_graph *g) {
  MG_CUDA_TRY(cudaSetDevice(g->device));
  if (g->pending_validation) {
    // an asynchronous upload: wait for it and read the validation flags before any
    // kernel touches the arrays
    int hbad = 0;
    const int *bad = reinterpret_cast<const int *>(reinterpret_cast<const char *>(g->ctl) + sizeof(DevCtl));
    MG_CUDA_TRY(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
    MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
    if (hbad) {
      mg_set_error("mg_graph_create (asynchronous upload): %s",
                   (hbad & 1) ? "row offsets are not a valid CSR (0..m, non-decreasing)"
                              : "column index out of range [0, n)");
      return MG_ERR_ARG;
    }
    g->pending_validation = false;
  }
  return MG_OK;
}

mg_status check_device_ptr(const mg_graph *g, const void *p, const char *fn, const char *what) {
  if (!p) return MG_OK;
  cudaPointerAttributes at;
  const cudaError_t e = cudaPointerGetAttributes(&at, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    mg_set_error("%s: cannot query %s (%s): it must be device memory", fn, what, cudaGetErrorString(e));
    return MG_ERR_ARG;
  }
  if (at.type == cudaMemoryTypeManaged) return MG_OK;
  if (at.type != cudaMemoryTypeDevice) {
    mg_set_error("%s: %s is %s memory; it must be device memory of device %d", fn, what,
                 at.type == cudaMemoryTypeHost ? "pinned host" : "pageable host", g->device);
    return MG_ERR_ARG;
  }
  if (at.device != g->device) {
    mg_set_error("%s: %s is memory of device %d, the graph lives on device %d", fn, what, at.device, g->device);
    return MG_ERR_ARG;
  }
  return MG_OK;
}

mg_status copy_out(mg_graph *g, void *dst, const void *src, size_t bytes, int device_output) {
  if (bytes == 0) return MG_OK;
  MG_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, device_output ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                              g->stream));
  return MG_OK;
}

namespace mg {

// ---------------------------------------------------------------------------
// Validation: row offsets non-decreasing from 0 to m, column indices in [0, n).
// Column indices are read with 16-byte vector loads.
__global__ void validate_kernel(const int32_t *__restrict__ ro, const int32_t *__restrict__ ci, int64_t n,
                                int64_t m, int *__restrict__ bad) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int b = 0;
  for (int64_t i = tid; i <= n; i += stride) {
    int32_t r = ro[i];
    if (i == 0 && r != 0) b |= 1;
    if (i == n && r != (int32_t)m) b |= 1;
    if (i < n && ro[i + 1] < r) b |= 1;
  }
  const int64_t m4 = m / 4;
  const int4 *ci4 = reinterpret_cast<const int4 *>(ci);
  const uint32_t un = (uint32_t)n;
  for (int64_t i = tid; i < m4; i += stride) {
    int4 c = __ldg(ci4 + i);
    if ((uint32_t)c.x >= un || (uint32_t)c.y >= un || (uint32_t)c.z >= un || (uint32_t)c.w >= un) b |= 2;
  }
  for (int64_t i = m4 * 4 + tid; i < m; i += stride)
    if ((uint32_t)ci[i] >= un) b |= 2;
  if (b) atomicOr(bad, b);
}

// ---------------------------------------------------------------------------
// Exclusive scan of int32 counts (n items) into int32 offsets (n + 1 items),
// three passes over tiles of 2048.
constexpr int SCAN_NT = 256, SCAN_VT = 8, SCAN_TILE = SCAN_NT * SCAN_VT;

__global__ void __launch_bounds__(SCAN_NT) scan_tile_sums(const int32_t *__restrict__ in, int64_t n,
                                                          int64_t *__restrict__ sums) {
  __shared__ int64_t sm[SCAN_NT / 32 + 1];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_VT; k++) {
    int64_t i = base + k * SCAN_NT + threadIdx.x;
    if (i < n) s += in[i];
  }
  s = block_sum<SCAN_NT>(s, sm);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

__global__ void __launch_bounds__(1024) scan_sums_single(int64_t *__restrict__ sums, int64_t nt) {
  __shared__ int64_t sm[1024 / 32 + 1];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b = 0; b < nt; b += 1024) {
    int64_t i = b + threadIdx.x;
    int64_t v = i < nt ? sums[i] : 0;
    int64_t tot;
    int64_t ex = block_exclusive_scan<1024>(v, sm, &tot);
    if (i < nt) sums[i] = ex + carry;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(SCAN_NT) scan_tiles(const int32_t *__restrict__ in, int64_t n,
                                                      const int64_t *__restrict__ sums, int32_t *__restrict__ out) {
  __shared__ int64_t sm[SCAN_NT / 32 + 1];
  __shared__ int32_t tile[SCAN_TILE];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
  for (int k = 0; k < SCAN_VT; k++) {
    int64_t i = base + k * SCAN_NT + threadIdx.x;
    tile[k * SCAN_NT + threadIdx.x] = i < n ? in[i] : 0;
  }
  __syncthreads();
  int64_t loc[SCAN_VT];
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_VT; k++) {
    loc[k] = s;
    s += tile[threadIdx.x * SCAN_VT + k];
  }
  int64_t tot;
  int64_t ex = block_exclusive_scan<SCAN_NT>(s, sm, &tot);
  int64_t off = sums[blockIdx.x] + ex;
#pragma unroll
  for (int k = 0; k < SCAN_VT; k++) {
    int64_t i = base + threadIdx.x * SCAN_VT + k;
    if (i < n) out[i] = (int32_t)(off + loc[k]);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == SCAN_NT - 1) out[n] = (int32_t)(off + s);
}

}  // namespace mg

// Exclusive scan of n int32 counts into n+1 offsets; tmp must hold
// ceil(n / 2048) int64 values.
mg_status device_exclusive_scan(const int32_t *in, int32_t *out, int64_t n, int64_t *tmp, cudaStream_t s) {
  using namespace mg;
  int64_t nt = std::max<int64_t>(1, (n + SCAN_TILE - 1) / SCAN_TILE);
  scan_tile_sums<<<(unsigned)nt, SCAN_NT, 0, s>>>(in, n, tmp);
  scan_sums_single<<<1, 1024, 0, s>>>(tmp, nt);
  scan_tiles<<<(unsigned)nt, SCAN_NT, 0, s>>>(in, n, tmp, out);
  MG_CUDA_TRY(cudaGetLastError());
  return MG_OK;
}

namespace mg {

// Pads of an offsets array (INT_MAX after entry n) and of its edge arrays (0).
__global__ void fill_pad_kernel(int32_t *off, int64_t n, int32_t *edges, void *vals, int64_t m) {
  const int t = threadIdx.x;
  if (t < MG_OFF_PAD) off[n + 1 + t] = INT_MAX;
  if (t < MG_EDGE_PAD) {
    edges[m + t] = 0;
    if (vals) reinterpret_cast<int32_t *>(vals)[m + t] = 0;
  }
}

// ---------------------------------------------------------------------------
// CSC build: least-significant-digit radix sort of (column, edge id), RS_BITS bits
// a pass. A tile of RS_TILE edges is counted per digit, the counts are scanned
// digit-major over the tiles, and the tile is ranked and written out.
//
// Memory traffic bounds it: 20 bytes per edge and pass. A counting sort by atomics
// (count, scatter, sort every column) queues on the hot columns of a skewed graph:
// R-MAT s20, 16.8 M edges, 0.34 ms for the counts, 3.2 ms for the scatter and 3.1
// ms for sorting the columns.
constexpr int RS_BITS = 8;
constexpr int RS_NT = 256;
constexpr int RS_WARPS = RS_NT / 32;
constexpr int RS_VT = 16;
constexpr int RS_TILE = RS_NT * RS_VT;

// Lanes of the warp whose digit equals this lane's (all lanes call it). A ballot per
// bit: match.any took 131 us per pass here against 97 (R-MAT s20, 16.8 M edges).
__device__ __forceinline__ unsigned rs_peers(unsigned d, int bits) {
  unsigned m = FULL;
  for (int b = 0; b < bits; b++) {
    const unsigned v = __ballot_sync(FULL, (d >> b) & 1);
    m &= (d >> b) & 1 ? v : ~v;
  }
  return m;
}

// Digit counts of a tile: cnt[digit * ntiles + tile].
__global__ void __launch_bounds__(RS_NT) rs_count_kernel(const int32_t *__restrict__ key, int64_t m, int shift,
                                                         int bits, int32_t ntiles, int32_t *__restrict__ cnt) {
  // a copy per warp: a skewed graph's hot column is in most warps
  __shared__ int32_t s_cnt[RS_WARPS][1 << RS_BITS];
  const unsigned mask = (1u << bits) - 1;
  for (int i = threadIdx.x; i < RS_WARPS << RS_BITS; i += RS_NT) (&s_cnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t t0 = (int64_t)blockIdx.x * RS_TILE;
  int32_t k[RS_VT];
#pragma unroll
  for (int r = 0; r < RS_VT; r++) {
    const int64_t i = t0 + r * RS_NT + threadIdx.x;
    k[r] = i < m ? __ldcs(key + i) : -1;
  }
#pragma unroll
  for (int r = 0; r < RS_VT; r++)
    if (k[r] >= 0) atomicAdd(&s_cnt[warp_id()][((unsigned)k[r] >> shift) & mask], 1);
  __syncthreads();
  for (int i = threadIdx.x; i <= (int)mask; i += RS_NT) {
    int32_t t = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) t += s_cnt[w][i];
    cnt[(int64_t)i * ntiles + blockIdx.x] = t;
  }
}

// Stable scatter of a tile: warp w ranks its RS_VT x 32 consecutive edges in order
// (32 at a time, per-warp digit counters), the tile is put in digit order in shared
// memory and leaves it in runs. val_in == nullptr: the payload is the edge id.
__global__ void __launch_bounds__(RS_NT, 3) rs_scatter_kernel(const int32_t *__restrict__ key_in,
                                                           const int32_t *__restrict__ val_in, int64_t m, int shift,
                                                           int bits, int32_t ntiles,
                                                           const int32_t *__restrict__ ofs,
                                                           int32_t *__restrict__ key_out,
                                                           int32_t *__restrict__ val_out) {
  __shared__ int32_t s_key[RS_TILE], s_val[RS_TILE];
  __shared__ uint16_t s_cnt[RS_WARPS][1 << RS_BITS];  // per warp: digit counts, then exclusive tile positions
  __shared__ int32_t s_base[1 << RS_BITS];            // global position of a digit minus its tile position
  __shared__ int32_t s_red[RS_WARPS + 1];
  const unsigned mask = (1u << bits) - 1;
  const int lane = lane_id(), w = warp_id();
  for (int i = threadIdx.x; i < RS_WARPS << RS_BITS; i += RS_NT) (&s_cnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t t0 = (int64_t)blockIdx.x * RS_TILE;
  const int64_t w0 = t0 + w * (RS_VT * 32) + lane;
  int32_t k[RS_VT], v[RS_VT];
  uint16_t rank[RS_VT];
#pragma unroll
  for (int r = 0; r < RS_VT; r++) {
    const int64_t i = w0 + r * 32;
    k[r] = i < m ? __ldcs(key_in + i) : -1;
    v[r] = i < m ? (val_in ? __ldcs(val_in + i) : (int32_t)i) : 0;
  }
#pragma unroll
  for (int r = 0; r < RS_VT; r++) {
    const unsigned d = k[r] < 0 ? (1u << bits) : ((unsigned)k[r] >> shift) & mask;
    const unsigned peers = rs_peers(d, bits + 1);
    const int before = __popc(peers & lanemask_lt());
    int32_t c = 0;
    if (k[r] >= 0) c = s_cnt[w][d];
    __syncwarp();
    if (k[r] >= 0 && before == 0) s_cnt[w][d] = (uint16_t)(c + __popc(peers));
    __syncwarp();
    rank[r] = (uint16_t)(c + before);
  }
  __syncthreads();
  // digit d (one per thread): the warps' counts become tile positions
  int32_t tot = 0;
  const int d0 = threadIdx.x;
  if (d0 <= (int)mask)
    for (int q = 0; q < RS_WARPS; q++) tot += s_cnt[q][d0];
  int32_t all;
  int32_t pos = block_exclusive_scan<RS_NT>(tot, s_red, &all);
  if (d0 <= (int)mask) {
    s_base[d0] = ofs[(int64_t)d0 * ntiles + blockIdx.x] - pos;
    for (int q = 0; q < RS_WARPS; q++) {
      const int32_t c = s_cnt[q][d0];
      s_cnt[q][d0] = (uint16_t)pos;
      pos += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_VT; r++) {
    if (k[r] < 0) continue;
    const int32_t at = s_cnt[w][((unsigned)k[r] >> shift) & mask] + rank[r];
    s_key[at] = k[r];
    s_val[at] = v[r];
  }
  __syncthreads();
  const int32_t n_here = (int32_t)min((int64_t)RS_TILE, m - t0);
  for (int32_t i = threadIdx.x; i < n_here; i += RS_NT) {
    const int32_t key = s_key[i];
    const int32_t at = s_base[((unsigned)key >> shift) & mask] + i;
    key_out[at] = key;
    val_out[at] = s_val[i];
  }
}

// First position in [lo, hi) of the ascending a whose value is >= x (hi if none).
__device__ __forceinline__ int64_t lower_bound_i32(const int32_t *__restrict__ a, int64_t lo, int64_t hi, int32_t x) {
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(a + mid) < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Column offsets from the sorted columns: a CTA brackets its 256 columns first (2,048
// columns per CTA: 68 us against 35, R-MAT s20).
__global__ void __launch_bounds__(256) csc_offsets_kernel(const int32_t *__restrict__ key, int64_t m, int64_t n,
                                                          int32_t *__restrict__ co) {
  __shared__ int64_t s_lo, s_hi;
  const int64_t c0 = (int64_t)blockIdx.x * 256, c1 = c0 + 256;
  if (threadIdx.x == 0) s_lo = lower_bound_i32(key, 0, m, (int32_t)c0);
  if (threadIdx.x == 32) s_hi = c1 <= n ? lower_bound_i32(key, 0, m, (int32_t)(c1 - 1)) : m;
  __syncthreads();
  for (int64_t c = c0 + threadIdx.x; c < min(c1, n + 1); c += 256)
    co[c] = c == n ? (int32_t)m : (int32_t)lower_bound_i32(key, s_lo, s_hi, (int32_t)c);
}

// Row of every CSR edge beside its value, {row, value bits} (val == nullptr: the
// row alone): a CTA brackets the rows of its EP_VT x 256 edges, a thread then
// searches between them (8,192 edges per CTA: 181 us for 16.8 M edges, 1,024: 130).
// The pair is one random read per edge for csc_gather_kernel.
constexpr int EP_VT = 4;
template <bool PAIR>
__global__ void __launch_bounds__(256) edge_rows_kernel(const int32_t *__restrict__ ro, int64_t n, int64_t m,
                                                        const int32_t *__restrict__ val, int32_t *__restrict__ out) {
  __shared__ int64_t s_row[2];
  const int64_t k0 = (int64_t)blockIdx.x * 256 * EP_VT;
  if ((threadIdx.x & 31) == 0 && threadIdx.x < 64) {
    // last row that starts at or before the tile's first / last edge
    const int64_t k = threadIdx.x == 0 ? k0 : min(k0 + 256 * EP_VT, m) - 1;
    s_row[threadIdx.x >> 5] = lower_bound_i32(ro, 0, n + 1, (int32_t)k + 1) - 1;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < EP_VT; j++) {
    const int64_t k = k0 + j * 256 + threadIdx.x;
    if (k >= m) break;
    const int32_t row = (int32_t)(lower_bound_i32(ro, s_row[0], s_row[1] + 1, (int32_t)k + 1) - 1);
    if (PAIR) reinterpret_cast<int2 *>(out)[k] = make_int2(row, val[k]);
    else out[k] = row;
  }
}

// Row index and value of every CSC slot, through its edge id.
template <bool PAIR>
__global__ void __launch_bounds__(256) csc_gather_kernel(const int32_t *__restrict__ perm,
                                                         const int32_t *__restrict__ rows, int64_t m,
                                                         int32_t *__restrict__ ri, int32_t *__restrict__ cval) {
  const int64_t stride = (int64_t)gridDim.x * 256;
  for (int64_t i0 = (int64_t)blockIdx.x * 256 + threadIdx.x; i0 < m; i0 += 4 * stride) {
    int32_t k[4];
    int2 p[4];
#pragma unroll
    for (int j = 0; j < 4; j++) k[j] = i0 + j * stride < m ? __ldcs(perm + i0 + j * stride) : 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (PAIR) p[j] = __ldg(reinterpret_cast<const int2 *>(rows) + k[j]);
      else p[j].x = __ldg(rows + k[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t i = i0 + j * stride;
      if (i >= m) continue;
      ri[i] = p[j].x;
      if (PAIR) cval[i] = p[j].y;
    }
  }
}

}  // namespace mg

// Builds the CSC of g (co, ri, perm, cvals). Scratch is taken from ws_aux.
static mg_status build_csc(mg_graph *g) {
  using namespace mg;
  const int64_t n = g->n, m = g->m;
  cudaStream_t s = g->stream;
  const size_t vbytes = g->vtype == MG_DTYPE_NONE ? 0 : 4;
  g->csc_owned = true;  // set first: a failure below frees what was allocated
  MG_CUDA_TRY(mg_malloc_async((void **)&g->co, sizeof(int32_t) * (n + 1 + MG_OFF_PAD), s));
  MG_CUDA_TRY(mg_malloc_async((void **)&g->ri, sizeof(int32_t) * (m + MG_EDGE_PAD), s));
  MG_CUDA_TRY(mg_malloc_async((void **)&g->perm, sizeof(int32_t) * (m + MG_EDGE_PAD), s));
  if (vbytes) MG_CUDA_TRY(mg_malloc_async(&g->cvals, vbytes * (m + MG_EDGE_PAD), s));
  mg::fill_pad_kernel<<<1, 32, 0, s>>>(g->co, n, g->ri, g->cvals, m);
  g->has_csc = true;
  if (m == 0) {
    MG_CUDA_TRY(cudaMemsetAsync(g->co, 0, sizeof(int32_t) * (n + 1), s));
    return MG_OK;
  }
  int bits = 1;
  while (bits < 31 && ((int64_t)1 << bits) < n) bits++;
  const int passes = (bits + RS_BITS - 1) / RS_BITS;
  const int32_t tiles = (int32_t)((m + RS_TILE - 1) / RS_TILE);
  const int64_t ncnt = (int64_t)tiles << RS_BITS;
  const size_t em = sizeof(int32_t) * (size_t)m;
  // keys ping-pong side by side (afterwards the {row, value} pairs), the payload's
  // other buffer (one of the two is perm itself), tile counts and their offsets
  MG_TRY(ws_reserve(g, g->ws_aux, Carve::need({2 * em + 256, em, sizeof(int32_t) * (size_t)ncnt,
                                               sizeof(int32_t) * (size_t)(ncnt + 1),
                                               sizeof(int64_t) * (size_t)(ncnt / SCAN_TILE + 2)})));
  Carve cv(g->ws_aux.ptr);
  int32_t *keys = cv.take<int32_t>(2 * (size_t)m + 64);
  int32_t *vtmp = cv.take<int32_t>(m);
  int32_t *cnt = cv.take<int32_t>(ncnt);
  int32_t *ofs = cv.take<int32_t>(ncnt + 1);
  int64_t *tmp = cv.take<int64_t>(ncnt / SCAN_TILE + 2);
  int32_t *kbuf[2] = {keys, keys + m};
  const int32_t *kin = g->ci, *vin = nullptr;
  int shift = 0;
  for (int p = 0; p < passes; p++) {
    const int b = (bits - shift + (passes - p) - 1) / (passes - p);  // digits of equal width
    int32_t *ko = kbuf[p & 1], *vo = (passes - 1 - p) & 1 ? vtmp : g->perm;
    rs_count_kernel<<<tiles, RS_NT, 0, s>>>(kin, m, shift, b, tiles, cnt);
    MG_TRY(device_exclusive_scan(cnt, ofs, (int64_t)tiles << b, tmp, s));
    rs_scatter_kernel<<<tiles, RS_NT, 0, s>>>(kin, vin, m, shift, b, tiles, ofs, ko, vo);
    kin = ko;
    vin = vo;
    shift += b;
  }
  csc_offsets_kernel<<<(unsigned)(n / 256 + 1), 256, 0, s>>>(kin, m, n, g->co);
  // the sorted keys are done with: the pairs take their place
  const unsigned et = (unsigned)((m + 256 * EP_VT - 1) / (256 * EP_VT));
  const int grid = g->num_sms * 8;
  if (vbytes) {
    edge_rows_kernel<true><<<et, 256, 0, s>>>(g->ro, n, m, (const int32_t *)g->vals, keys);
    csc_gather_kernel<true><<<grid, 256, 0, s>>>(g->perm, keys, m, g->ri, (int32_t *)g->cvals);
  } else {
    edge_rows_kernel<false><<<et, 256, 0, s>>>(g->ro, n, m, nullptr, keys);
    csc_gather_kernel<false><<<grid, 256, 0, s>>>(g->perm, keys, m, g->ri, nullptr);
  }
  MG_CUDA_TRY(cudaGetLastError());
  return MG_OK;
}

// Pinned host mirrors of the control blocks, recycled across graphs: pinning
// and unpinning host memory costs a driver round trip each time.
static std::mutex g_pinned_mu;
static std::vector<void *> g_pinned_free;

static DevCtl *pinned_ctl_get() {
  {
    std::lock_guard<std::mutex> lk(g_pinned_mu);
    if (!g_pinned_free.empty()) {
      void *p = g_pinned_free.back();
      g_pinned_free.pop_back();
      return static_cast<DevCtl *>(p);
    }
  }
  void *p = nullptr;
  if (cudaHostAlloc(&p, sizeof(DevCtl) + 64, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<DevCtl *>(p);
}

static void pinned_ctl_put(DevCtl *p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  g_pinned_free.push_back(p);
}

static void graph_free_device(mg_graph *g) {
  cudaStream_t s = g->stream;
  auto fr = [&](void *p) {
    if (p) cudaFreeAsync(p, s);
  };
  fr(g->ro);
  fr(g->ci);
  fr(g->vals);
  if (g->csc_owned) {
    fr(g->co);
    fr(g->ri);
    fr(g->perm);
    fr(g->cvals);
  }
  fr(g->ws_main.ptr);
  fr(g->ws_aux.ptr);
  fr(g->ws_out.ptr);
  fr(g->ctl);
  if (s) cudaStreamSynchronize(s);
  pinned_ctl_put(g->ctl_host);
  g->ctl_host = nullptr;
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (s) cudaStreamDestroy(s);
  cudaGetLastError();
}

void engine_release_cached(mg_graph *g);  // defined with the iteration drivers
void pr_release_plans(mg_graph *g);       // defined with PageRank

extern "C" {

const char *mg_status_string(mg_status s) {
  switch (s) {
    case MG_OK: return "MG_OK";
    case MG_ERR_ARG: return "MG_ERR_ARG: invalid argument";
    case MG_ERR_OOM: return "MG_ERR_OOM: out of memory";
    case MG_ERR_QUEUE_OVERFLOW: return "MG_ERR_QUEUE_OVERFLOW: frontier queue overflow, increase queue_sizing";
    case MG_ERR_TIMEOUT: return "MG_ERR_TIMEOUT: a bounded device wait ran out";
    case MG_ERR_CUDA: return "MG_ERR_CUDA: CUDA runtime error";
    case MG_ERR_NO_DEVICE: return "MG_ERR_NO_DEVICE: no usable CUDA device";
    case MG_ERR_UNSUPPORTED: return "MG_ERR_UNSUPPORTED: unsupported option combination";
  }
  return "unknown mg_status";
}

const char *mg_last_error(void) { return g_err; }

const char *mg_version(void) { return "mapgraph_b200 0.1.0 (sm_100a)"; }

int32_t mg_device_count(void) {
  int c = 0;
  if (cudaGetDeviceCount(&c) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return c;
}

static mg_status create_impl(const int32_t *row_offsets, const int32_t *col_idx, const void *edge_vals,
                             mg_dtype vals_t, int64_t n, int64_t m, uint32_t flags, mg_graph **out) {
  if (!out) {
    mg_set_error("mg_graph_create: out is NULL");
    return MG_ERR_ARG;
  }
  *out = nullptr;
  if (n < 0 || m < 0 || n > INT32_MAX - 1 || m > INT32_MAX || !row_offsets || (m > 0 && !col_idx) ||
      (vals_t != MG_DTYPE_NONE && m > 0 && !edge_vals) || vals_t < MG_DTYPE_NONE || vals_t > MG_DTYPE_F32) {
    mg_set_error("mg_graph_create: invalid sizes or null arrays (n=%lld m=%lld)", (long long)n, (long long)m);
    return MG_ERR_ARG;
  }
  if (mg_device_count() <= 0) {
    mg_set_error("mg_graph_create: no CUDA device");
    return MG_ERR_NO_DEVICE;
  }
  mg_graph *g = new mg_graph();
  g->n = n;
  g->m = m;
  g->flags = flags;
  g->vtype = vals_t;
  auto fail = [&](mg_status st) {
    graph_free_device(g);
    delete g;
    return st;
  };
  if (cudaGetDevice(&g->device) != cudaSuccess) return fail(MG_ERR_CUDA);
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  g->num_sms = sms > 0 ? sms : 148;
  if (cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking) != cudaSuccess) {
    mg_set_error("mg_graph_create: stream creation failed");
    return fail(MG_ERR_CUDA);
  }
  {
    // Keep freed graph memory in the stream-ordered pool so that repeated
    // create/destroy cycles reuse it instead of returning it to the driver.
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, g->device) == cudaSuccess) {
      uint64_t thr = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    cudaGetLastError();
  }
  cudaStream_t s = g->stream;
  const size_t vb = vals_t == MG_DTYPE_NONE ? 0 : 4;
  const cudaMemcpyKind kind = (flags & MG_GRAPH_DEVICE_INPUT) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
#define CREATE_TRY(expr)                                                                        \
  do {                                                                                          \
    cudaError_t _e = (expr);                                                                    \
    if (_e != cudaSuccess) {                                                                    \
      mg_set_error("mg_graph_create: %s failed: %s", #expr, cudaGetErrorString(_e));           \
      cudaGetLastError();                                                                       \
      return fail(_e == cudaErrorMemoryAllocation ? MG_ERR_OOM : MG_ERR_CUDA);                  \
    }                                                                                           \
  } while (0)
  CREATE_TRY(mg_malloc_async((void **)&g->ro, sizeof(int32_t) * (n + 1 + MG_OFF_PAD), s));
  CREATE_TRY(mg_malloc_async((void **)&g->ci, sizeof(int32_t) * (m + MG_EDGE_PAD), s));
  if (vb) CREATE_TRY(mg_malloc_async(&g->vals, vb * (m + MG_EDGE_PAD), s));
  mg::fill_pad_kernel<<<1, 32, 0, s>>>(g->ro, n, g->ci, g->vals, m);
  CREATE_TRY(cudaMemcpyAsync(g->ro, row_offsets, sizeof(int32_t) * (n + 1), kind, s));
  if (m > 0) CREATE_TRY(cudaMemcpyAsync(g->ci, col_idx, sizeof(int32_t) * m, kind, s));
  if (vb && m > 0) CREATE_TRY(cudaMemcpyAsync(g->vals, edge_vals, vb * m, kind, s));
  if (dev_alloc(g, (void **)&g->ctl, MG_TRACE_OFF + sizeof(mg_level_record) * MG_TRACE_LEVELS) != MG_OK)
    return fail(MG_ERR_OOM);
  g->ctl_host = pinned_ctl_get();
  if (!g->ctl_host) {
    mg_set_error("mg_graph_create: pinned host allocation failed");
    return fail(MG_ERR_OOM);
  }
  {
    unsigned long long *box = const_cast<unsigned long long *>(graph_mailbox(g));
    CREATE_TRY(cudaMemcpyAsync(loop_mailbox(g->ctl), &box, sizeof(box), cudaMemcpyHostToDevice, s));
  }
  CREATE_TRY(cudaEventCreate(&g->ev0));
  CREATE_TRY(cudaEventCreate(&g->ev1));
  // Validate on the device.
  int *bad = reinterpret_cast<int *>(reinterpret_cast<char *>(g->ctl) + sizeof(DevCtl));
  CREATE_TRY(cudaMemsetAsync(bad, 0, sizeof(int) * 2, s));
  mg::validate_kernel<<<g->num_sms * 8, 256, 0, s>>>(g->ro, g->ci, n, m, bad);
  CREATE_TRY(cudaGetLastError());
  if ((flags & MG_GRAPH_ASYNC_UPLOAD) && (flags & (MG_GRAPH_SYMMETRIC | MG_GRAPH_NO_CSC))) {
    // no CSC to build from unvalidated arrays: return now, check on first use
    g->pending_validation = true;
    if (flags & MG_GRAPH_SYMMETRIC) {
      g->co = g->ro;
      g->ri = g->ci;
      g->perm = nullptr;
      g->cvals = g->vals;
      g->has_csc = true;
      g->csc_owned = false;
    }
    *out = g;
    return MG_OK;
  }
  int hbad[2] = {0, 0};
  CREATE_TRY(cudaMemcpyAsync(hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  CREATE_TRY(cudaStreamSynchronize(s));
  if (hbad[0]) {
    mg_set_error("mg_graph_create: %s", (hbad[0] & 1) ? "row offsets are not a valid CSR (0..m, non-decreasing)"
                                                      : "column index out of range [0, n)");
    return fail(MG_ERR_ARG);
  }
  if (flags & MG_GRAPH_SYMMETRIC) {
    g->co = g->ro;
    g->ri = g->ci;
    g->perm = nullptr;
    g->cvals = g->vals;
    g->has_csc = true;
    g->csc_owned = false;
  } else if (!(flags & MG_GRAPH_NO_CSC)) {
    mg_status st = build_csc(g);
    if (st != MG_OK) return fail(st);
  }
  if (cudaStreamSynchronize(s) != cudaSuccess) {
    mg_set_error("mg_graph_create: %s", cudaGetErrorString(cudaGetLastError()));
    return fail(MG_ERR_CUDA);
  }
#undef CREATE_TRY
  *out = g;
  return MG_OK;
}

mg_status mg_graph_create(const int32_t *row_offsets, const int32_t *col_idx, const void *edge_vals,
                          mg_dtype vals_t, int64_t n, int64_t m, uint32_t flags, mg_graph **out) {
  return create_impl(row_offsets, col_idx, edge_vals, vals_t, n, m, flags, out);
}

mg_status mg_graph_destroy(mg_graph *g) {
  if (!g) return MG_OK;
  cudaSetDevice(g->device);
  engine_release_cached(g);
  pr_release_plans(g);
  graph_free_device(g);
  delete g;
  return MG_OK;
}

mg_status mg_graph_stream(const mg_graph *g, void **stream) {
  if (!g || !stream) {
    mg_set_error("mg_graph_stream: null argument");
    return MG_ERR_ARG;
  }
  *stream = (void *)g->stream;
  return MG_OK;
}

mg_status mg_graph_info(const mg_graph *g, int64_t *n, int64_t *m, uint32_t *flags, int32_t *device) {
  if (!g) {
    mg_set_error("mg_graph_info: graph is NULL");
    return MG_ERR_ARG;
  }
  if (n) *n = g->n;
  if (m) *m = g->m;
  if (flags) *flags = g->flags;
  if (device) *device = g->device;
  return MG_OK;
}

namespace {
// out[0] = max out-degree, out[1] = vertices without out-edges.
__global__ void degree_stats_kernel(const int32_t *__restrict__ ro, int64_t n, unsigned long long *out) {
  int32_t mx = 0;
  unsigned long long zero = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t d = ro[i + 1] - ro[i];
    mx = max(mx, d);
    zero += d == 0;
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  for (int o = 16; o > 0; o >>= 1) zero += __shfl_xor_sync(0xffffffffu, zero, o);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, (unsigned long long)mx);
    if (zero) atomicAdd(out + 1, zero);
  }
}
}  // namespace

mg_status mg_graph_degree_stats(mg_graph *g, int64_t *max_out_degree, int64_t *no_out_edges) {
  if (!g) {
    mg_set_error("mg_graph_degree_stats: graph is NULL");
    return MG_ERR_ARG;
  }
  MG_TRY(graph_enter(g));
  // two counters in the control block's spare bytes behind the DevCtl
  unsigned long long *d = reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(g->ctl) + sizeof(DevCtl));
  unsigned long long h[2] = {0, 0};
  MG_CUDA_TRY(cudaMemcpyAsync(d, h, sizeof(h), cudaMemcpyHostToDevice, g->stream));
  if (g->n > 0) degree_stats_kernel<<<g->num_sms * 4, 256, 0, g->stream>>>(g->ro, g->n, d);
  MG_CUDA_TRY(cudaGetLastError());
  MG_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
  MG_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (max_out_degree) *max_out_degree = (int64_t)h[0];
  if (no_out_edges) *no_out_edges = (int64_t)h[1];
  return MG_OK;
}

mg_status mg_graph_device_arrays(const mg_graph *g, const int32_t **row_offsets, const int32_t **col_idx,
                                 const void **edge_vals, const int32_t **col_offsets, const int32_t **row_idx,
                                 const int32_t **csc_perm) {
  if (!g) {
    mg_set_error("mg_graph_device_arrays: graph is NULL");
    return MG_ERR_ARG;
  }
  if (row_offsets) *row_offsets = g->ro;
  if (col_idx) *col_idx = g->ci;
  if (edge_vals) *edge_vals = g->vals;
  if (col_offsets) *col_offsets = g->has_csc ? g->co : nullptr;
  if (row_idx) *row_idx = g->has_csc ? g->ri : nullptr;
  if (csc_perm) *csc_perm = g->perm;
  return MG_OK;
}

mg_status mg_graph_create_ragged(int32_t ngraphs, const int32_t *const *row_offsets, const int32_t *const *col_idx,
                                 const int64_t *n, const int64_t *m, uint32_t flags, mg_graph **out) {
  if (!out || ngraphs <= 0 || !row_offsets || !col_idx || !n || !m || (flags & MG_GRAPH_DEVICE_INPUT)) {
    mg_set_error("mg_graph_create_ragged: invalid arguments");
    return MG_ERR_ARG;
  }
  int64_t N = 0, M = 0;
  std::vector<int64_t> vbase(ngraphs + 1, 0);
  for (int32_t i = 0; i < ngraphs; i++) {
    if (n[i] < 0 || m[i] < 0 || !row_offsets[i] || (m[i] > 0 && !col_idx[i])) {
      mg_set_error("mg_graph_create_ragged: member %d invalid", i);
      return MG_ERR_ARG;
    }
    vbase[i] = N;
    N += n[i];
    M += m[i];
  }
  vbase[ngraphs] = N;
  if (N > INT32_MAX - 1 || M > INT32_MAX) {
    mg_set_error("mg_graph_create_ragged: union exceeds int32");
    return MG_ERR_ARG;
  }
  std::vector<int32_t> ro(N + 1), ci(std::max<int64_t>(M, 1));
  int64_t eo = 0;
  for (int32_t i = 0; i < ngraphs; i++) {
    const int32_t *r = row_offsets[i];
    if (r[0] != 0 || r[n[i]] != m[i]) {
      mg_set_error("mg_graph_create_ragged: member %d row offsets do not span 0..m", i);
      return MG_ERR_ARG;
    }
    for (int64_t v = 0; v < n[i]; v++) ro[vbase[i] + v] = (int32_t)(eo + r[v]);
    for (int64_t e = 0; e < m[i]; e++) {
      int32_t c = col_idx[i][e];
      if (c < 0 || c >= n[i]) {
        mg_set_error("mg_graph_create_ragged: member %d column index out of range", i);
        return MG_ERR_ARG;
      }
      ci[eo + e] = (int32_t)(vbase[i] + c);
    }
    eo += m[i];
  }
  ro[N] = (int32_t)M;
  mg_status st = create_impl(ro.data(), ci.data(), nullptr, MG_DTYPE_NONE, N, M, flags, out);
  if (st == MG_OK) (*out)->vbase = vbase;
  return st;
}

mg_status mg_graph_ragged_bases(const mg_graph *g, int64_t *vertex_base) {
  if (!g || !vertex_base || g->vbase.empty()) {
    mg_set_error("mg_graph_ragged_bases: not a ragged graph");
    return MG_ERR_ARG;
  }
  std::memcpy(vertex_base, g->vbase.data(), sizeof(int64_t) * g->vbase.size());
  return MG_OK;
}

}  // extern "C"
