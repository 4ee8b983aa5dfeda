// engine.cuh -- the iteration-loop driver shared by the vertex programs.
//
// The reference drives every GAS iteration from the host and reads the frontier
// size back after each one (GASengine/enactor_vertex_centric.cuh:2526-2872,
// cudaMemcpy at :2866-2869). Here the kernel that finishes an iteration (last CTA
// to arrive) decides on the device whether another one runs, and nothing waits for
// the host to hear of it. mg_opts.use_graph picks how the next iteration gets there:
//    1  the iteration's kernels are captured once into the body of a CUDA-graph
//       WHILE node: one graph launch per run and an idle host, for a few microseconds
//       per iteration (the conditional node and a loop guard) and the instantiation
//       on a first call.
//    0  (default) as 1 for the traversals, whose iterations are several kernels of a
//       few microseconds each (launching them one by one is slower: BFS R-MAT s22 488
//       us in the graph, 571 launched ahead). The PageRank loops, one or two kernels
//       of tens of microseconds, are launched ahead: up to LOOP_AHEAD iterations are
//       queued behind the running one, the device reports every finished iteration
//       and the end by a store to a word of pinned host memory, and iterations
//       queued past the end return at once. The gap between two iterations is that
//       of two kernels, and a first call builds no graph (reference-compatible
//       PageRank, 48 sweeps: 1.85 -> 1.56 ms; a one-shot solve 3.19 -> 2.79 ms).
//   -1  host-driven, one control-block read per iteration, for comparison and
//       debugging.
#pragma once

#include <cuda_runtime.h>
#include <cstring>
#include <functional>
#include <vector>

#include "mg_internal.h"

// Body enqueuer: launches one iteration's kernels on `s`. The CTA that ends the
// iteration passes h and `use_cond` to loop_signal, a kernel that finds the run over
// to loop_over.
using LoopBody = std::function<void(cudaStream_t s, cudaGraphConditionalHandle h, int use_cond)>;

// Runs `body` until DevCtl::done is set on the device, as `mode` (mg_opts.use_graph)
// says; `ahead`: mode 0 launches ahead. `slot` and `sig` identify a cached executable
// graph (reused while the signature matches). `max_iters` bounds the host's launches.
mg_status run_loop(mg_graph *g, int slot, const void *sig, size_t sig_len, int mode, const LoopBody &body,
                   int64_t max_iters, bool ahead = false);

// Kernels the last run's loop launched, `per` of them per iteration (host_iters 0: a
// graph, whose guard adds one; ctl_host is the control block after the run).
inline int64_t loop_launches(const mg_graph *g, int64_t per) {
  return g->host_iters ? per * g->host_iters : (per + 1) * (int64_t)g->ctl_host->body_iters;
}

// use_cond of a body: who hears that an iteration ended.
enum { LOOP_NONE = 0, LOOP_GRAPH = 1, LOOP_MAIL = 2 };

#ifdef __CUDACC__
// The host's mailbox: one word per run, reports << 1 | over.
__device__ __forceinline__ void loop_mail(DevCtl *c, bool over) {
  volatile unsigned long long *box = *loop_mailbox(c);
  *box = ((unsigned long long)c->reports << 1) | (over ? 1ull : 0ull);
}

// Called by one thread when an iteration ends.
__device__ __forceinline__ void loop_signal(DevCtl *c, cudaGraphConditionalHandle h, int use_cond, bool over) {
  if (use_cond == LOOP_GRAPH) {
    cudaGraphSetConditional(h, over ? 0u : 1u);
  } else if (use_cond == LOOP_MAIL) {
    c->reports += 1;
    loop_mail(c, over);
  }
}

// Called by every thread of a kernel that finds the run over.
__device__ __forceinline__ void loop_over(DevCtl *c, cudaGraphConditionalHandle h, int use_cond) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  if (use_cond == LOOP_GRAPH) cudaGraphSetConditional(h, 0u);
  else if (use_cond == LOOP_MAIL) loop_mail(c, true);
}
#endif

// Copies the control block back to the pinned host mirror (synchronises the stream).
mg_status fetch_ctl(mg_graph *g);

// Cache slots.
enum LoopSlot { SLOT_BFS = 0, SLOT_SSSP, SLOT_CC, SLOT_PR, SLOT_PR_REF, SLOT_ADJ, SLOT_MSBFS, SLOT_BSSSP, SLOT_PPR,
                SLOT_MSSSP, SLOT_COUNT };
