// Segment kernels: adf_h on edge level runs (fill_up_dn_grad, adv_flux_hor_ho), plus the lane kernel of the remaining edge lanes. The bodies are in fct_segments.cuh; one translation
// unit per stage keeps the template instantiations of each stage compiling in parallel.
#include "fct_segments.cuh"

namespace fct {
namespace {

FCT_SEG_KERNEL(k_seg_edge, seg_edge_adf, kStageEdge)

// the remaining edge lanes: kFixThreads threads per lane (and slice of NTR tracers)
template <int NTR>
__global__ void __launch_bounds__(256) k_edge_fix_1(const __grid_constant__ Inst in, int t0,
                                                    int w0) {
  const int sub = int(blockIdx.y) * NTR;
  body_edge_fix<NTR, false>(in, lane_index() / kFixThreads, int(threadIdx.x) % kFixThreads,
                            t0 + sub, w0 + sub);
}
template <int NTR>
__global__ void __launch_bounds__(256) k_edge_fix_n(const Inst* __restrict__ tab, int t0, int w0,
                                                    int S) {
  const unsigned q = unsigned(lane_index() / kFixThreads), lane = q / unsigned(S);
  const int sub = int(q - lane * unsigned(S)) * NTR;
  body_edge_fix<NTR, true>(tab[blockIdx.y], lane, int(threadIdx.x) % kFixThreads, t0 + sub,
                           w0 + sub);
}

}  // namespace

int launch_edge_fix(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0,
                    int c1, cudaStream_t s) {
  if (d.max_efix == 0) return FCT_OK;
  for (int t0 = c0; t0 < c1;) {
    // two tracers per thread at most: the lanes are few, and a thread's chain is what counts
    const SegSplit sp = seg_split(c1 - t0, std::min(2, d.smap_tracers[kStageEdge]),
                                  tab != nullptr, seg_even(d));
    const int P = sp.tracers, S = sp.slices, w0 = t0 - c0;
    if (tab) {
      const dim3 g(seg_blocks(d.max_efix * S, 256 / kFixThreads), unsigned(n));
      if (P == 2) k_edge_fix_n<2><<<g, 256, 0, s>>>(tab, t0, w0, S);
      else k_edge_fix_n<1><<<g, 256, 0, s>>>(tab, t0, w0, S);
    } else {
      const dim3 g(seg_blocks(d.max_efix, 256 / kFixThreads), unsigned(S));
      if (P == 2) k_edge_fix_1<2><<<g, 256, 0, s>>>(single, t0, w0);
      else k_edge_fix_1<1><<<g, 256, 0, s>>>(single, t0, w0);
    }
    t0 += P * S;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "launch_edge_fix");
}

namespace {

__host__ __device__ constexpr int edge_blocks(int ntr, bool) {
  return ntr == 1 ? 5 : ntr == 2 ? 3 : 2;
}
#define FCT_BODY(NTR, IL) stream_edge_adf<NTR, IL>
FCT_STREAM_KERNEL(k_edge_stream, FCT_BODY, edge_blocks)
#undef FCT_BODY

#define FCT_COUNT(V) d.max_eseg[V]
FCT_STREAM_LAUNCHER(launch_stream, k_edge_stream, FCT_COUNT, FCT_GRID, kStageEdge, edge_blocks)
FCT_SEG_LAUNCHER(launch_impl, k_seg_edge, FCT_COUNT, FCT_GRID, kStageEdge)
#undef FCT_COUNT

}  // namespace

int launch_seg_edge(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1,
                    cudaStream_t s) {
  if (d.smap_levels[kStageEdge] == 1) return launch_stream(single, tab, n, d, c0, c1, s);
  return launch_impl(single, tab, n, d, c0, c1, s);
}

}  // namespace fct
