// Segment kernels: T_new on node layer runs (zalesak_limit b3, flux2dtracer_fct, ale_reconstruct). The bodies are in fct_segments.cuh; one translation
// unit per stage keeps the template instantiations of each stage compiling in parallel.
#include "fct_segments.cuh"

namespace fct {
namespace {

FCT_SEG_KERNEL(k_seg_final, seg_node_final, kStageFinal)

// Blocks per SM and slots per batch by tracers per thread, against the run kernel at its best
// mapping: 1 tracer 90 us against 102, T and S 155 against 179 (CORE2-size mesh); 8 tracers of
// two members 1.15 ms against 1.08 of the run kernel at 2 x 2, which interleaved instances of 4
// tracers or more therefore keep.
__host__ __device__ constexpr int stream_blocks(int ntr, bool) {
  return ntr == 1 ? 4 : ntr == 2 ? 2 : 1;
}
__host__ __device__ constexpr int slot_batch(int, bool) {
  return 3;
}
#define FCT_BODY(NTR, IL) stream_node_final<NTR, IL, slot_batch(NTR, IL)>
FCT_STREAM_KERNEL(k_stream_final, FCT_BODY, stream_blocks)
#undef FCT_BODY

#define FCT_COUNT(V) d.max_nseg[V]
FCT_STREAM_LAUNCHER(launch_stream, k_stream_final, FCT_COUNT, FCT_GRID, kStageFinal, stream_blocks)
FCT_SEG_LAUNCHER(launch_impl, k_seg_final, FCT_COUNT, FCT_GRID, kStageFinal)
#undef FCT_COUNT

}  // namespace

int launch_seg_final(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1,
                     cudaStream_t s) {
  if (d.smap_levels[kStageFinal] == 1) return launch_stream(single, tab, n, d, c0, c1, s);
  return launch_impl(single, tab, n, d, c0, c1, s);
}

}  // namespace fct
