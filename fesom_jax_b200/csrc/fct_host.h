// Host-side helpers shared by the libfesom_fct translation units.
#pragma once

#include <algorithm>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>

#include <cuda_runtime.h>

#include "fct_internal.cuh"

namespace fct {

// Record the calling thread's last error and return ``status``.
int set_error(int status, const char* fmt, ...);

inline int cuda_error(cudaError_t e, const char* what) {
  return set_error(FCT_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define FCT_CUDA(call)                                   \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return ::fct::cuda_error(e_, #call); \
  } while (0)

// most blocks of the one launch of a small instance's first stages: eight waves of two blocks on
// every SM. Measured up to 6 waves it gains (pi, T and S: 46.5 us a step against 50.9 with a
// launch per stage; 600 nodes 33.8 against 46.1), at 44 there is no difference (20,000 nodes x 3
// tracers); where between them the gain ends was not measured.
constexpr int64_t kFirstBlocks = 8 * 2 * 148;

// fused stages with their own thread mapping: LO, edge, limiter, final
constexpr int kFusedStages = 4;
enum { kStageLo = 0, kStageEdge = 1, kStageLimit = 2, kStageFinal = 3 };

// Launch the forward kernel sequence for ``n`` instances. ``single`` is used when
// ``tab`` is null (n == 1), otherwise ``tab`` is a device array of ``n`` instances
// whose lane counts are bounded by the ``max_*`` arguments.
struct LaunchDims {
  int64_t max_iface, max_layer, max_edge, max_elem, max_dense, max_nodes;
  int64_t max_dry = 0;   // dry node levels (kept from T)
  int max_levels = 0;    // nl
  int ntr;           // tracers per instance (every instance of a launch has the same)
  int chunk = 0;     // tracers whose intermediates share the workspace (0 = all ntr);
                     // stages run chunk by chunk
  bool any_wi;      // launch the implicit w_i stage
  bool copy_dry;    // launch the dry-level copy
  bool pairs = true;  // the instances' interleaved tracer buffers start on 16-byte boundaries
  bool any_vdiff = false;  // launch the implicit vertical diffusion after each chunk
  bool any_derive_w = false;  // derive w_e from uv (compute_w) before the step
  bool skip_vflux = false;    // the workspace already holds this step's volume fluxes (and
                              // w_derived its w)
  bool fused = true;  // fused stages (lean workspace); false: every stage kernel writes its
                      // intermediates (what the reverse pass reads)
  // fused (segment) stages: per stage (LO, edge, limiter, final) the most tracers and the
  // levels a thread takes (tuning knobs), and the largest segment counts over the launch's
  // instances
  int smap_tracers[kFusedStages] = {2, 2, 2, 2};
  int smap_levels[kFusedStages] = {1, 1, 1, 1};
  void set_map(int tracers, int levels) {
    for (int i = 0; i < kFusedStages; ++i) {
      smap_tracers[i] = tracers;
      smap_levels[i] = levels;
    }
  }
  // The mapping of a plan or batch that was given none. Tracer-major: two tracers and one level
  // per thread everywhere (the stream kernels; runs of two or more levels per thread spread a
  // warp's loads over twice the lines or more). Interleaved, from sweeps over 8 tracers of two
  // CORE2-size members: the final stage's run kernel at two levels (1.08 ms, stream 1.14); 4
  // tracers per thread in the others where ``threads`` (wet node layers x tracers of the launch
  // / 4) leaves two blocks for every SM (LO 0.76 ms against 0.90 at 2 tracers, edge 0.66 / 0.80,
  // limiter 1.25 / 1.37); odd tracer counts, whose loads are single values, the run kernels at
  // two levels except in the edge stage (LO 1.21 against 1.54, limiter 1.68 / 1.75).
  void auto_map(bool interleaved, bool even, int64_t threads) {
    set_map(2, 1);
    if (!interleaved) return;
    smap_levels[kStageFinal] = 2;
    if (!even) {
      smap_levels[kStageLo] = smap_levels[kStageLimit] = 2;
    } else if (ntr >= 4 && threads >= int64_t(148) * 2 * 256) {
      for (int i : {kStageLo, kStageEdge, kStageLimit}) smap_tracers[i] = 4;
    }
  }
  int64_t max_nseg[kSegVariants] = {0, 0, 0, 0};
  int64_t max_eseg[kSegVariants] = {0, 0, 0, 0};
  int64_t max_efix = 0;
  // fused path: run the edge stage on fork->side beside the LO stage (null: one stream)
  const Fork* fork = nullptr;
};

// Create / release a Fork on the current device.
int fork_create(Fork& f);
void fork_destroy(Fork& f);

// Grow ``d``'s lane and segment counts to cover a plan's mesh.
inline void dims_cover(LaunchDims& d, const FctPlan* P) {
  const DevMesh& m = P->hm;
  d.max_iface = std::max(d.max_iface, m.n_iface);
  d.max_layer = std::max(d.max_layer, m.n_layer);
  d.max_edge = std::max(d.max_edge, m.n_edge);
  d.max_elem = std::max(d.max_elem, m.n_elem);
  d.max_dense = std::max(d.max_dense, int64_t(P->N) * P->L);
  d.max_dry = std::max(d.max_dry, P->hm.n_dry);
  d.max_nodes = std::max(d.max_nodes, int64_t(P->N));
  d.max_levels = std::max(d.max_levels, P->L);
  for (int v = 0; v < kSegVariants; ++v) {
    d.max_nseg[v] = std::max(d.max_nseg[v], m.n_nseg[v]);
    d.max_eseg[v] = std::max(d.max_eseg[v], m.n_eseg[v]);
  }
  d.max_efix = std::max(d.max_efix, m.n_efix);
}

// The mapping of a single-plan launch: the plan's own, or the rule's.
inline void dims_map(LaunchDims& d, const FctPlan* P) {
  if (P->per_thread > 0) d.set_map(P->per_thread, P->lpt);
  else d.auto_map(false, true, 0);
}

// Grid of a kernel whose threads walk its lanes, for ``n`` instances of at most ``need`` blocks
// when ``full`` blocks are resident at once. Large instances go one after the other, so that
// the gathers of all blocks stay within a few columns of each other; where one gives a thread
// fewer than kWalk lanes they go side by side (grid.y), with about as many blocks each as fill
// the chip together (16 pi-size members x 30 steps: 17.3 ms one after the other, 14.8 with every
// block of every instance in the grid and no walk, 12.8 so): full / n blocks each, rounded to
// the side with fewer waves per block. Rounded up always, a few blocks ran in a wave of their
// own (volume fluxes of 64 pi members, 768 blocks on 740 places: 202 us against 130; two and
// eight tracers of 24 pi members, all stages: 733 and 2,420 us a step against 627 and 2,054).
constexpr int kWalk = 4;
inline dim3 stream_grid(int64_t need, int64_t full, int n) {
  if (need >= kWalk * full) return dim3(unsigned(full), 1);
  auto waves = [&](int64_t x) { return (x * n + full - 1) / full; };
  const int64_t lo = std::max<int64_t>(1, full / n), hi = (full + n - 1) / n;
  const int64_t x = waves(hi) * lo <= waves(lo) * hi ? hi : lo;
  return dim3(unsigned(std::max<int64_t>(1, std::min(need, x))), unsigned(n));
}

// Tracers per thread and tracer slices of one segment launch over ``rem`` tracers: the
// largest compiled count (1, 2 or 4 interleaved, 1 when pairs are not 16-byte aligned; 1 or 2
// tracer-major) of at most ``per_thread``, and as many slices as whole counts fit (at most 8
// interleaved). Three tracer-major tracers go one per thread, in one launch instead of two.
struct SegSplit {
  int tracers, slices;
};
inline SegSplit seg_split(int rem, int per_thread, bool interleaved, bool even) {
  const int lim = std::min(rem, per_thread);
  int P = lim >= 2 ? 2 : 1;
  if (interleaved) {
    if (lim >= 4) P = 4;
    if (!even) P = 1;
    int S = std::min(8, rem / P);
    // three single tracers keep two launches per stage, two slices and one, as the launch count
    // of test_derived_w_equals_compute_w_then_fct has it; in one launch of three slices two
    // CORE2-size members took 2.86 ms a step against 3.83, 16 pi members 0.80 against 1.01, one
    // pi member 63 us against 85
    if (P == 1 && rem == 3) S = 2;
    return {P, S};
  }
  if (rem == 3) P = 1;
  return {P, rem / P};
}
// tracer pairs are 16-byte aligned: the interleaved tracer and workspace strides are even and
// the tracer buffers start on such a boundary
inline bool seg_even(const LaunchDims& d) {
  const int chunk = d.chunk > 0 ? d.chunk : d.ntr;
  return d.pairs && d.ntr % 2 == 0 && chunk % 2 == 0;
}
inline bool buffers_paired(const FctInstance& q) {
  for (const double* b : q.buf)
    if (reinterpret_cast<uintptr_t>(b) % 16 != 0) return false;
  return true;
}

// The fused stages over the tracers [c0, c1) of a workspace chunk (fct_seg_*.cu).
int launch_seg_lo(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                  int c1, cudaStream_t s);
int launch_seg_edge(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                    int c1, cudaStream_t s);
int launch_edge_fix(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                    int c1, cudaStream_t s);
int launch_seg_limit(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                     int c1, cudaStream_t s);
int launch_seg_final(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                     int c1, cudaStream_t s);
// The LO stage, the edge stage with its remaining lanes and (``dry``) the dry-level copy of a
// single instance in one launch, where their blocks make at most kFirstBlocks (seg_first_fits):
// they depend only on the volume fluxes, not on one another, and on a small mesh each of them is
// shorter than the gap between two launches (fct_seg_first.cu).
int launch_seg_first(const Inst& single, const LaunchDims& d, int c0, int c1, bool dry,
                     cudaStream_t s);
inline int64_t seg_first_blocks(const LaunchDims& d, int tracers_per_thread, int rem) {
  const int64_t slices = rem / tracers_per_thread;
  auto blocks = [](int64_t threads) { return (threads + 255) / 256; };
  return (blocks(d.max_nseg[0]) + blocks(d.max_eseg[0]) + blocks(d.max_efix * 2)) * slices;
}
inline bool seg_first_fits(const LaunchDims& d, int c0, int c1) {
  const SegSplit sp = seg_split(c1 - c0, d.smap_tracers[kStageLo], false, false);
  return d.smap_levels[kStageLo] == 1 && d.smap_levels[kStageEdge] == 1 &&
         d.smap_tracers[kStageEdge] == d.smap_tracers[kStageLo] &&
         seg_first_blocks(d, sp.tracers, c1 - c0) <= kFirstBlocks;
}
int launch_forward(const Inst& single, const Inst* tab, int n, const LaunchDims& d,
                   cudaStream_t s);
// Same, recording ``after[i]`` on ``s`` after stage i of a chunk (skipped stages record
// too); ``chunk_sel >= 0`` launches only that workspace chunk.
constexpr int kNumStages = 10;
extern const char* const kStageNames[kNumStages];
int launch_forward_events(const Inst& single, const Inst* tab, int n, const LaunchDims& d,
                          cudaStream_t s, cudaEvent_t* after, bool stop_before_final = false,
                          int chunk_sel = -1);
// Single-instance forward stages; ``through_factors`` stops after the limiter factors
// (everything the reverse pass reads), without writing T_new.
int launch_forward_stages(const Inst& single, const LaunchDims& d, cudaStream_t s,
                          bool through_factors);
// fct_plan_reserve (declared in the public header) is used by the adjoint reservation.

// Copy T's dry levels into T_new for ``n`` instances of ``tab`` (ignores Inst::copy_dry).
int launch_copy_dry(const Inst* tab, int n, int64_t max_dry, cudaStream_t s);
// compute_w of every table instance with w_derived set (fct_producers.cu).
int launch_compute_w_tab(const Inst* tab, int n, int64_t max_nodes, cudaStream_t s);
// Implicit vertical diffusion alone (fct_vert_diff): single instance, tracer-major.
int launch_vdiff(const Inst& single, const LaunchDims& d, cudaStream_t s);

// Workspace of `ntr` tracers: every stage field (the unfused stages, which the reverse
// pass recomputes and reads), or with `fused` only the fields the fused forward keeps.
Workspace carve_workspace(double* base, int64_t N, int64_t E, int64_t Ed, int64_t L, int ntr,
                          bool fused = false);
int64_t workspace_doubles(int64_t N, int64_t E, int64_t Ed, int64_t L, int ntr);
int64_t workspace_doubles_fused(int64_t N, int64_t Ed, int64_t L, int ntr);
// Grow the plan workspace to `ntr` tracers; `full` also makes it hold every stage field.
int plan_reserve_ws(FctPlan* P, int ntr, bool full);
// A plan created by fct_plan_create in this process and not destroyed yet.
bool plan_alive(const FctPlan* P);

// Ordering of the calls that use a plan's workspace: hold ``P->mu`` (PlanUse does), wait
// on stream ``s`` for the previous user, launch, then record the release on ``s``. Both
// are skipped while ``s`` is being captured into a CUDA graph (an event from outside a
// capture cannot be waited on inside it): captured calls are ordered by their graph.
class PlanUse {
 public:
  PlanUse(FctPlan* P, cudaStream_t s);
  // record the release event (call after the launches; returns a status)
  int release();
  int status() const { return st_; }

 private:
  std::lock_guard<std::mutex> lk_;
  FctPlan* P_;
  cudaStream_t s_;
  bool capturing_ = false;
  int st_ = 0;
};

// Copy a device counter to the host on ``s``, wait, zero it, and return FCT_ERR_NONFINITE
// when it was non-zero (``out`` receives the count when not NULL).
int read_health(unsigned long long* d_counter, int n, cudaStream_t s, int64_t* out);

// The volume-flux kernel reads u and v of an element level with one 16-byte load: a uv that it
// cannot read is refused before the launch.
inline int check_uv(const double* uv) {
  if (reinterpret_cast<uintptr_t>(uv) % 16 != 0)
    return set_error(FCT_ERR_INVALID, "uv must start on a 16-byte boundary");
  return FCT_OK;
}

// Launches one fused stage takes for `csz` tracers of a workspace chunk with at most
// `per_thread` tracers per thread.
inline int stage_launches(int csz, int per_thread, bool even) {
  int count = 0;
  for (int t = 0; t < csz; ++count) {
    const SegSplit sp = seg_split(csz - t, per_thread, true, even);
    t += sp.tracers * sp.slices;
  }
  return count;
}

}  // namespace fct
