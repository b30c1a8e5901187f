// The first stages of a small single instance in one launch: the remaining edge lanes (the
// longest chain, so their blocks come first), the LO stage, the edge stage and the dry-level
// copy. Each depends only on the volume fluxes; on a small mesh a stage of its own takes less
// time than the gap between two launches and, on two streams, than the events between them.
#include "fct_segments.cuh"

namespace fct {
namespace {

template <int NTR>
__global__ void __launch_bounds__(256, 2) k_seg_first_1(const __grid_constant__ Inst in, int t0,
                                                        int w0, int nfix, int nlo, int nedge) {
  const int tid = threadIdx.x, sub = int(blockIdx.y) * NTR;
  int b = blockIdx.x;
  if (b < nfix) {
    const int64_t i = int64_t(b) * 256 + tid;
    body_edge_fix<NTR, false>(in, i / kFixThreads, tid % kFixThreads, t0 + sub, w0 + sub);
  } else if ((b -= nfix) < nlo) {
    stream_node_lo<NTR, false, 3>(in, int64_t(b) * 256 + tid, int64_t(nlo) * 256, t0 + sub,
                                  w0 + sub);
  } else if ((b -= nlo) < nedge) {
    stream_edge_adf<NTR, false>(in, int64_t(b) * 256 + tid, int64_t(nedge) * 256, t0 + sub,
                                   w0 + sub);
  } else if (blockIdx.y == 0) {
    body_copy_dry<false>(in, int64_t(b - nedge) * 256 + tid);
  }
}

}  // namespace

int launch_seg_first(const Inst& single, const LaunchDims& d, int c0, int c1, bool dry,
                     cudaStream_t s) {
  const unsigned nlo = seg_blocks(d.max_nseg[0], 256);
  const unsigned nedge = d.max_eseg[0] > 0 ? seg_blocks(d.max_eseg[0], 256) : 0;
  const unsigned nfix = d.max_efix > 0 ? seg_blocks(d.max_efix, 256 / kFixThreads) : 0;
  for (int t0 = c0; t0 < c1;) {
    const SegSplit sp = seg_split(c1 - t0, d.smap_tracers[kStageLo], false, false);
    const int w0 = t0 - c0;
    const unsigned ndry = dry && t0 == c0 && d.max_dry > 0 ? seg_blocks(d.max_dry, 256) : 0;
    const dim3 g(nfix + nlo + nedge + ndry, unsigned(sp.slices));
    if (sp.tracers == 2)
      k_seg_first_1<2><<<g, 256, 0, s>>>(single, t0, w0, int(nfix), int(nlo), int(nedge));
    else
      k_seg_first_1<1><<<g, 256, 0, s>>>(single, t0, w0, int(nfix), int(nlo), int(nedge));
    t0 += sp.tracers * sp.slices;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "launch_seg_first");
}

}  // namespace fct
