// pr_binned.cuh -- degree-binned gather over a CSR-shaped adjacency, the default
// PageRank / adjoint gather.
//
// Rows are binned once per adjacency by degree, and each bin gets the lane count
// that keeps a warp's loads in flight without idle lanes:
//   bin 0       no edges: only the row update;
//   bin 1       1 or 2 edges: one lane per row, plain loads;
//   bins 2..9   up to 64 edges: one lane per row, classes narrow enough that the
//               32 rows of a warp end together. A lane reads its row's indices a
//               sector at a time and gathers 8 values before its first add, so a
//               warp keeps up to 256 gathers in flight, with no shuffles;
//   bin 10      65..256 edges: 4 lanes per row, 8 rows per warp;
//   bin 11      up to PRB_HEAVY: one warp per row, 256 edges per step;
//   bin 12      degree >= PRB_HEAVY (hubs): split into chunks of PRB_CHUNK edges; a
//               warp reduces one chunk into a partial; the warp that completes a
//               hub's last chunk (per-row arrival counter) adds the partials in
//               chunk order and finishes the row.
// The random gathers bound it, and before them the number in flight: with a warp
// per row above 16 edges and 32 such rows per work item, a warp waited for two
// round trips per row and the items of the heaviest rows ran last and alone
// (R-MAT s22 directed, weighted, 67 M edges: 451 us per iteration, 380 with these
// bins; symmetric, unweighted, 134 M edges: 542 and 530).
// Warps are independent (no CTA barriers while gathering). The per-row sums are
// compensated (TwoSum per addend, FMA-based TwoProduct for weights) and every
// row's sum has a fixed order, so the result does not depend on scheduling. A
// persistent grid takes the assignments from a counter (or with a fixed stride);
// hub rows keep their FP64 contributions in a per-hub array.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "pr_gather.cuh"

namespace mg {

constexpr int PRB_NT = 256;
constexpr int PRB_BINS = 13;
constexpr int PRB_QUAD = 10;  // first bin of more than one lane per row (4 lanes)
constexpr int PRB_WARP = 11;  // a warp per row
constexpr int PRB_HUB = 12;   // hub rows
// Rows of one warp assignment of a bin.
__host__ __device__ constexpr int prb_rows_per(int bin) { return bin < PRB_QUAD ? 32 : bin == PRB_QUAD ? 8 : 2; }
// Resident CTAs per SM the iteration kernel is compiled for.
#ifndef PRB_MIN_BLOCKS
#define PRB_MIN_BLOCKS 5
#endif
// Index (and weight) streams are read once per iteration: they do not displace the
// gathered vector in L1.
#ifndef PRB_STREAM_LOADS
#define PRB_STREAM_LOADS 1
#endif
__device__ __forceinline__ int32_t prb_stream(const int32_t *p) {
#if PRB_STREAM_LOADS
  int32_t v;
  asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
#else
  return __ldcs(p);
#endif
}
__device__ __forceinline__ uint32_t prb_stream(const uint32_t *p) {
  return (uint32_t)prb_stream(reinterpret_cast<const int32_t *>(p));
}
__device__ __forceinline__ float prb_stream(const float *p) {
  return __int_as_float(prb_stream(reinterpret_cast<const int32_t *>(p)));
}
#ifndef PRB_HEAVY_EDGES
#define PRB_HEAVY_EDGES 2048
#endif
// Solve kernels take their work items from a shared counter (1) or by a fixed
// grid stride (0).
#ifndef PRB_DYNAMIC
#define PRB_DYNAMIC 1
#endif
constexpr int32_t PRB_HEAVY = PRB_HEAVY_EDGES;
constexpr int32_t PRB_CHUNK = 2048;

// Plan of one adjacency.
struct BinPlan {
  int32_t *rows = nullptr;      // rows grouped by bin (hubs apart), bin b at rows[boff[b]..]
  int32_t *hrows = nullptr;     // hub rows
  int32_t *hbase = nullptr;     // first chunk task of each hub, nheavy + 1 entries
  int32_t *hcount = nullptr;    // arrival counters of the hubs (reset by the finishing warp)
  Comp *hpart = nullptr;        // partial sums of the hub chunks
  double *hcontrib = nullptr;   // per-hub FP64 contributions (residual, second reduction)
  int32_t *grab = nullptr;      // work-item counter of the dynamic schedule (zero between launches)
  int64_t boff[PRB_BINS + 1] = {0};  // bin offsets into rows
  int64_t nheavy = 0, ntasks = 0;
  int64_t wstart[PRB_BINS + 1] = {0};  // first warp assignment of each bin
};

}  // namespace mg

// Host side (pagerank.cu): builds / releases a plan over `off` (n + 1 entries);
// rows of at least `heavy` edges become hubs.
mg_status bin_plan_build(cudaStream_t s, const int32_t *off, int64_t n, mg::BinPlan &bp,
                         int32_t heavy = mg::PRB_HEAVY);
void bin_plan_release(cudaStream_t s, mg::BinPlan &bp);
namespace mg {
struct PrbArgs;
}
// Arguments of the graph's cached plan of its CSC (or CSR) rows, without weights.
mg_status graph_bin_plan(mg_graph *g, bool csr, mg::PrbArgs *out);

namespace mg {

// Bin of a row of `deg` edges; rows of at least `heavy` edges are hubs.
__device__ __forceinline__ int prb_bin_of(int32_t deg, int32_t heavy = PRB_HEAVY) {
  if (deg >= heavy) return PRB_HUB;
  if (deg <= 8) return deg <= 2 ? (deg + 1) >> 1 : deg <= 4 ? 2 : 3;
  if (deg <= 16) return deg <= 12 ? 4 : 5;
  if (deg <= 32) return deg <= 24 ? 6 : 7;
  if (deg <= 64) return deg <= 48 ? 8 : 9;
  return deg <= 256 ? PRB_QUAD : PRB_WARP;
}

// Ordered binning. Rows are cut into chunks of PRB_NT * PRB_RPT rows, one per
// CTA; pass 1 counts every bin per chunk, a single CTA turns the counts into
// output offsets (bin-major, chunk order), and pass 2 writes each chunk's rows in
// row order with an in-CTA exclusive scan per bin. Bins therefore list rows in
// ascending order and the plan is deterministic.
constexpr int PRB_RPT = 8;
constexpr int PRB_CHUNK_ROWS = PRB_NT * PRB_RPT;

#ifndef MG_PRB_NO_PLAN_KERNELS  // plan building runs in pagerank.cu only
// Bins of a thread's PRB_RPT consecutive rows from r0 (-1 past the end).
__device__ __forceinline__ void prb_bins_of(const int32_t *__restrict__ off, int64_t n, int64_t r0, int32_t heavy,
                                            int (&bins)[PRB_RPT], int32_t &chunks) {
  int32_t o[PRB_RPT + 1];
#pragma unroll
  for (int k = 0; k <= PRB_RPT; k++) o[k] = off[min(r0 + k, n)];
  chunks = 0;
#pragma unroll
  for (int k = 0; k < PRB_RPT; k++) {
    const int32_t d = o[k + 1] - o[k];
    bins[k] = r0 + k < n ? prb_bin_of(d, heavy) : -1;
    if (bins[k] == PRB_HUB) chunks += (d + PRB_CHUNK - 1) / PRB_CHUNK;
  }
}

// Counts are summed over a warp packed seven to a word (9 bits each: a warp has
// 256 rows), then added to the CTA's counters by one lane per warp and bin.
__global__ void __launch_bounds__(PRB_NT) prb_count_kernel(const int32_t *__restrict__ off, int64_t n,
                                                           int64_t *__restrict__ counts /* [chunk][BINS+1] */,
                                                           int32_t heavy) {
  __shared__ int32_t s[PRB_BINS + 1];
  if (threadIdx.x <= PRB_BINS) s[threadIdx.x] = 0;
  __syncthreads();
  int bins[PRB_RPT];
  int32_t chunks;
  prb_bins_of(off, n, (int64_t)blockIdx.x * PRB_CHUNK_ROWS + (int64_t)threadIdx.x * PRB_RPT, heavy, bins, chunks);
  unsigned long long w0 = 0, w1 = 0;
#pragma unroll
  for (int k = 0; k < PRB_RPT; k++) {
    if (bins[k] >= 7) w1 += 1ull << (9 * (bins[k] - 7));
    else if (bins[k] >= 0) w0 += 1ull << (9 * bins[k]);
  }
  w0 = warp_sum(w0);
  w1 = warp_sum(w1);
  const int lane = lane_id();
  if (lane < PRB_BINS) {
    const int32_t v = (int32_t)((lane < 7 ? w0 >> (9 * lane) : w1 >> (9 * (lane - 7))) & 511);
    if (v) atomicAdd(s + lane, v);
  }
  if (chunks) atomicAdd(s + PRB_BINS, chunks);
  __syncthreads();
  if (threadIdx.x <= PRB_BINS) counts[(int64_t)blockIdx.x * (PRB_BINS + 1) + threadIdx.x] = s[threadIdx.x];
}

// Exclusive prefix over chunks of every bin, in place (a warp per bin);
// totals[b] = bin sizes.
__global__ void __launch_bounds__(32 * (PRB_BINS + 1)) prb_offsets_kernel(int64_t *counts, int64_t nchunks,
                                                                          int64_t *totals) {
  const int b = warp_id(), lane = lane_id();
  int64_t acc = 0;
  for (int64_t c0 = 0; c0 < nchunks; c0 += 32) {
    const int64_t c = c0 + lane;
    const int64_t v = c < nchunks ? counts[c * (PRB_BINS + 1) + b] : 0;
    const int64_t inc = warp_inclusive_scan(v);
    if (c < nchunks) counts[c * (PRB_BINS + 1) + b] = acc + inc - v;
    acc += __shfl_sync(FULL, inc, 31);
  }
  if (lane == 0) totals[b] = acc;
}

__global__ void __launch_bounds__(PRB_NT) prb_scatter_kernel(const int32_t *__restrict__ off, int64_t n,
                                                             const int64_t *__restrict__ offsets,
                                                             const int64_t *__restrict__ boff, int32_t *rows,
                                                             int32_t *hrows, int32_t heavy) {
  // a CTA has 2048 rows: four bins to a 64-bit word, 16 bits each
  constexpr int NW = (PRB_BINS + 3) / 4;
  __shared__ unsigned long long red[PRB_NT / 32 + 1];
  const int64_t r0 = (int64_t)blockIdx.x * PRB_CHUNK_ROWS + (int64_t)threadIdx.x * PRB_RPT;
  int bins[PRB_RPT];
  int32_t chunks;
  prb_bins_of(off, n, r0, heavy, bins, chunks);
  unsigned long long pos[NW];
#pragma unroll
  for (int w = 0; w < NW; w++) {
    unsigned long long c = 0, tot;
#pragma unroll
    for (int k = 0; k < PRB_RPT; k++)
      if (bins[k] >= 0 && (bins[k] >> 2) == w) c += 1ull << (16 * (bins[k] & 3));
    pos[w] = block_exclusive_scan<PRB_NT>(c, red, &tot);
  }
#pragma unroll
  for (int k = 0; k < PRB_RPT; k++) {
    const int b = bins[k];
    if (b < 0) continue;
    int32_t at = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
      if ((b >> 2) == w) {
        at = (int32_t)((pos[w] >> (16 * (b & 3))) & 0xffff);
        pos[w] += 1ull << (16 * (b & 3));
      }
    }
    const int64_t o = offsets[(int64_t)blockIdx.x * (PRB_BINS + 1) + b] + at;
    if (b == PRB_HUB) hrows[o] = (int32_t)(r0 + k);
    else rows[boff[b] + o] = (int32_t)(r0 + k);
  }
}

// Chunk bases of the hubs (listed in ascending order): one CTA, exclusive scan of
// their chunk counts PRB_NT at a time.
__global__ void __launch_bounds__(PRB_NT) prb_hubs_kernel(const int32_t *__restrict__ off, const int32_t *hrows,
                                                          int64_t nheavy, int32_t *hbase) {
  __shared__ int32_t red[PRB_NT / 32 + 1];
  int32_t carry = 0;
  for (int64_t b0 = 0; b0 < nheavy; b0 += PRB_NT) {
    const int64_t i = b0 + threadIdx.x;
    int32_t c = 0;
    if (i < nheavy) {
      const int32_t d = off[hrows[i] + 1] - off[hrows[i]];
      c = (d + PRB_CHUNK - 1) / PRB_CHUNK;
    }
    int32_t tot;
    const int32_t ex = block_exclusive_scan<PRB_NT>(c, red, &tot);
    if (i < nheavy) hbase[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) hbase[nheavy] = carry;
}
#endif  // MG_PRB_NO_PLAN_KERNELS

struct PrbArgs {
  const int32_t *off, *idx;
  const float *wts;
  const int32_t *rows, *hrows, *hbase;
  int32_t *hcount;
  Comp *hpart;
  double *hcontrib;
  // Dynamic schedule: warps take one work item at a time from this counter
  // (heaviest first) instead of a fixed grid stride; the launch's last CTA
  // resets it. nullptr: fixed stride.
  int32_t *grab;
  int64_t boff[PRB_BINS + 1];
  int64_t wstart[PRB_BINS + 1];
  int64_t nheavy;
};

template <int G>
__device__ __forceinline__ void group_comp_reduce(Comp &c) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    Comp d{__shfl_xor_sync(0xffffffffu, c.hi, o), __shfl_xor_sync(0xffffffffu, c.lo, o)};
    // Fixed pairing: the lower lane of each pair adds the upper one's value.
    if ((threadIdx.x & o) == 0) comp_add(c, d);
    else {
      comp_add(d, c);
      c = d;
    }
  }
}

// 32 bytes of an index or weight stream (256-bit load, sm_100): read once, so not
// kept in L1.
__device__ __forceinline__ void prb_load8(const int32_t *p, int32_t (&c)[8]) {
  asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
      : "l"(p));
}
__device__ __forceinline__ void prb_load8(const float *p, float (&c)[8]) {
  asm("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]), "=f"(c[4]), "=f"(c[5]), "=f"(c[6]), "=f"(c[7])
      : "l"(p));
}

// Shared-memory address of a column cache that is complete: taken behind the barrier
// that ends its filling, so that no gather through it moves ahead of that.
__device__ __forceinline__ uint32_t cache_addr(const float *s) {
  uint32_t a = smem_u32(s);
  asm volatile("" : "+r"(a)::"memory");
  return a;
}

// Value of column entry c with a shared-memory column cache: c < 0 is a cached
// column's slot | 0x80000000, or -1 for no column, which reads the zero behind the
// cache (`zero`: its byte offset from `cache`, a shared-memory address). One
// predicated load either way, no branch.
__device__ __forceinline__ float cached_gather(uint32_t cache, uint32_t zero, const float *__restrict__ g, int32_t c) {
  float x;
  asm("{\n\t.reg .pred h;\n\t.reg .u32 s;\n\t.reg .s64 a;\n\tsetp.lt.s32 h, %1, 0;\n\t"
      "shl.b32 s, %1, 2;\n\tmin.u32 s, s, %3;\n\tadd.u32 s, s, %2;\n\tmad.wide.s32 a, %1, 4, %4;\n\t"
      "@h ld.shared.f32 %0, [s];\n\t@!h ld.global.nc.f32 %0, [a];\n\t}"
      : "=f"(x)
      : "r"(c), "r"(cache), "r"(zero), "l"(g));
  return x;
}

// Compensated sum of edges [b, e) by the L lanes of a group (sub: the lane's place
// in it), 8 edges per lane and step: one 32-byte index load (the lanes of a group
// side by side) from the row's start rounded down to a sector, 8 gathers, then the
// adds. Slots outside the row gather column -1, which is 0, and +0 leaves a
// compensated sum as it is. Index and weight arrays are padded by 8 entries, so the
// last sector may run over the row's (or the array's) end. Lanes of other groups
// may end earlier.
//
// A warp's load of 32 rows' sectors costs the L1 32 tag lookups, one per clock, like
// a load of 32 random columns, and lookups bound this kernel: 32-byte loads make it
// an eighth of a lookup per index against a quarter with 16-byte loads (weighted
// R-MAT s22 iteration 380 us with those, 338 with these).
template <int L, bool WEIGHTED, bool COMP, typename Gather>
__device__ __forceinline__ Comp prb_group_range(const PrbArgs &p, int32_t b, int32_t e, int sub, Gather &gather) {
  Comp acc{0.f, 0.f};
  for (int32_t k0 = (b & ~7) + 8 * sub; k0 < e; k0 += 8 * L) {
    int32_t c[8];
    float x[8], w[8];
    prb_load8(p.idx + k0, c);
    if (WEIGHTED) prb_load8(p.wts + k0, w);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const bool in = k0 + j >= b && k0 + j < e;
      x[j] = gather(in ? c[j] : -1);
      if (WEIGHTED) w[j] = in ? w[j] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (WEIGHTED) {
        const float pr = w[j] * x[j];
        two_sum_add(acc, pr);
        acc.lo += __fmaf_rn(w[j], x[j], -pr);
      } else if (COMP) {
        two_sum_add(acc, x[j]);
      } else {
        acc.hi += x[j];
      }
    }
  }
  if (L > 1) group_comp_reduce<L>(acc);
  return acc;
}

// Rows of up to 2 edges, one lane each, plain index loads.
template <bool WEIGHTED, bool COMP, typename Gather>
__device__ __forceinline__ Comp prb_short_range(const PrbArgs &p, int32_t b, int32_t e, Gather &gather) {
  Comp acc{0.f, 0.f};
  int32_t c[2];
  float x[2], w[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    c[j] = b + j < e ? prb_stream(p.idx + b + j) : -1;
    w[j] = WEIGHTED && b + j < e ? prb_stream(p.wts + b + j) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < 2; j++) x[j] = gather(c[j]);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    if (WEIGHTED) {
      const float pr = w[j] * x[j];
      two_sum_add(acc, pr);
      acc.lo += __fmaf_rn(w[j], x[j], -pr);
    } else if (COMP) {
      two_sum_add(acc, x[j]);
    } else {
      acc.hi += x[j];
    }
  }
  return acc;
}

// Hands the plan's warp assignments to item(bin, wa), hub chunks first and the
// lightest rows last (long items first shortens the tail), over a persistent grid.
template <typename Item>
__device__ __forceinline__ void prb_items(const PrbArgs &p, Item &&item) {
  const int64_t total = p.wstart[PRB_BINS];
  auto at = [&](int64_t wi) {
    const int64_t w = total - 1 - wi;
    int bin = 0;
#pragma unroll
    for (int q = 1; q < PRB_BINS; q++)
      if (w >= p.wstart[q]) bin = q;
    item(bin, w - p.wstart[bin]);
  };
  if (p.grab) {
    for (;;) {
      int64_t wi = 0;
      if (lane_id() == 0) wi = atomicAdd(p.grab, 1);
      wi = __shfl_sync(FULL, wi, 0);
      if (wi >= total) break;
      at(wi);
    }
  } else {
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t wi = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wi < total; wi += nwarps) at(wi);
  }
}

// Walks the plan's rows: body(L, row, b, e, sub, task) with L the lanes (an
// integral constant) that share edges [b, e) of `row`, sub the lane's place among
// them and task the chunk's number if they are a chunk of a hub (else -1). Every
// lane of the warp calls it: a group past the bin's end has row -1 and no edges.
template <typename Body>
__device__ __forceinline__ void prb_walk(const PrbArgs &p, Body &&body) {
  const int lane = threadIdx.x & 31;
  prb_items(p, [&](int bin, int64_t wa) {
    if (bin == PRB_HUB) {
      // its hub by binary search over the chunk bases
      int64_t lo = 0, hi = p.nheavy;
      while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (p.hbase[mid] <= wa) lo = mid;
        else hi = mid;
      }
      const int32_t row = p.hrows[lo];
      const int32_t b = __ldg(p.off + row) + (int32_t)(wa - p.hbase[lo]) * PRB_CHUNK;
      body(std::integral_constant<int, 32>(), row, b, min(b + PRB_CHUNK, __ldg(p.off + row + 1)), lane, wa, lo);
      return;
    }
    const int lg = bin < PRB_QUAD ? 0 : bin == PRB_QUAD ? 2 : 5;  // log2 of the lanes per row
    const int sub = lane & ((1 << lg) - 1);
    const int nrow = bin == PRB_WARP ? prb_rows_per(PRB_WARP) : 1;
    for (int q = 0; q < nrow; q++) {
      const int64_t slot = p.boff[bin] + (bin == PRB_WARP ? wa * nrow + q : wa * (32 >> lg) + (lane >> lg));
      const int32_t row = slot < p.boff[bin + 1] ? p.rows[slot] : -1;
      const int32_t b = row >= 0 ? __ldg(p.off + row) : 0;
      const int32_t e = row >= 0 ? __ldg(p.off + row + 1) : 0;
      const int64_t whole = -1;
      if (bin == PRB_WARP) body(std::integral_constant<int, 32>(), row, b, e, sub, whole, whole);
      else if (bin == PRB_QUAD) body(std::integral_constant<int, 4>(), row, b, e, sub, whole, whole);
      else if (bin > 1) body(std::integral_constant<int, 1>(), row, b, e, sub, whole, whole);
      else body(std::integral_constant<int, 0>(), row, b, e, sub, whole, whole);  // at most 2 edges
    }
  });
}

// A lane's share (prb_walk's L and sub) of the compensated sum of edges [b, e); COMP
// false: its own additions are plain FP32 (unweighted sums only).
template <int L, bool WEIGHTED, bool COMP = true, typename Gather>
__device__ __forceinline__ Comp prb_range(const PrbArgs &p, int32_t b, int32_t e, int sub, Gather &gather) {
  if constexpr (L == 0) return prb_short_range<WEIGHTED, COMP>(p, b, e, gather);
  else return prb_group_range<L, WEIGHTED, COMP>(p, b, e, sub, gather);
}

// A hub chunk's partial: stored, and the lane that stores the last one of hub h
// gets the sum of all of them in chunk order (true). Lane 0 calls it.
__device__ __forceinline__ bool prb_hub_done(const PrbArgs &p, int64_t task, int64_t h, const Comp &part, Comp &tot) {
  p.hpart[task] = part;
  __threadfence();
  const int32_t nch = p.hbase[h + 1] - p.hbase[h];
  if (atomicAdd(p.hcount + h, 1) != nch - 1) return false;
  __threadfence();
  tot = Comp{0.f, 0.f};
  const float2 *parts = reinterpret_cast<const float2 *>(p.hpart) + p.hbase[h];
  for (int32_t c = 0; c < nch; c++) {
    const float2 v = __ldcg(parts + c);  // written by other SMs: read from L2
    comp_add(tot, Comp{v.x, v.y});
  }
  p.hcount[h] = 0;
  return true;
}

// Sums every row of the plan, gather(-1) being 0: finish(row, Comp) consumes a row sum,
// finish_hub(h, row, Comp) a hub's.
template <bool WEIGHTED, typename Gather, typename Finish, typename FinishHub>
__device__ __forceinline__ void prb_run(const PrbArgs &p, Gather &&gather, Finish &&finish, FinishHub &&finish_hub) {
  prb_walk(p, [&](auto lanes, int32_t row, int32_t b, int32_t e, int sub, int64_t task, int64_t h) {
    const Comp acc = prb_range<decltype(lanes)::value, WEIGHTED>(p, b, e, sub, gather);
    if (task >= 0) {
      Comp tot;
      if (sub == 0 && prb_hub_done(p, task, h, acc, tot)) finish_hub(h, row, tot);
    } else if (row >= 0 && sub == 0) {
      finish(row, acc);
    }
  });
}

}  // namespace mg
