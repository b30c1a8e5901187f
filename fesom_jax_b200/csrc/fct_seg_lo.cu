// Segment kernels: LO and adf_v on node layer runs (compute_fct_lo, adv_flux_ver_ho). The bodies are in fct_segments.cuh; one translation
// unit per stage keeps the template instantiations of each stage compiling in parallel.
#include "fct_segments.cuh"

namespace fct {
namespace {

FCT_SEG_KERNEL(k_seg_lo, seg_node_lo, kStageLo)

// Blocks per SM and slots per batch by tracers per thread, against the run kernel at its best
// mapping: 1 tracer 84 us against 106, T and S 126 against 147 (CORE2-size mesh); 8 tracers of
// two members, 4 per thread, 0.76 ms against 0.90.
__host__ __device__ constexpr int stream_blocks(int ntr, bool il) {
  return ntr == 1 ? 4 : ntr == 2 ? (il ? 2 : 3) : 2;
}
__host__ __device__ constexpr int slot_batch(int ntr, bool il) {
  return ntr == 2 && !il ? 2 : 3;
}
#define FCT_BODY(NTR, IL) stream_node_lo<NTR, IL, slot_batch(NTR, IL)>
FCT_STREAM_KERNEL(k_stream_lo, FCT_BODY, stream_blocks)
#undef FCT_BODY

#define FCT_COUNT(V) d.max_nseg[V]
FCT_STREAM_LAUNCHER(launch_stream, k_stream_lo, FCT_COUNT, FCT_GRID, kStageLo, stream_blocks)
FCT_SEG_LAUNCHER(launch_impl, k_seg_lo, FCT_COUNT, FCT_GRID, kStageLo)
#undef FCT_COUNT

}  // namespace

int launch_seg_lo(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1,
                  cudaStream_t s) {
  if (d.smap_levels[kStageLo] == 1) return launch_stream(single, tab, n, d, c0, c1, s);
  return launch_impl(single, tab, n, d, c0, c1, s);
}

}  // namespace fct
