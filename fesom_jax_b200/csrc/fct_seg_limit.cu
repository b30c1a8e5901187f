// Segment kernels: limiter factors on node layer runs (zalesak_limit a1-a4, b1, b2). The bodies are in fct_segments.cuh; one translation
// unit per stage keeps the template instantiations of each stage compiling in parallel.
#include "fct_segments.cuh"

namespace fct {
namespace {

FCT_SEG_LIMIT_KERNEL(k_seg_limit)

// Blocks per SM and slots per batch by tracers per thread, against the run kernel at its best
// mapping: 1 tracer 123 us against 131, T and S 194 against 198 (CORE2-size mesh); 8 tracers of
// two members, 4 per thread, 1.25 ms against 1.46.
__host__ __device__ constexpr int stream_blocks(int ntr, bool il) {
  return ntr == 1 ? (il ? 5 : 3) : ntr == 2 ? 4 : 2;
}
__host__ __device__ constexpr int slot_batch(int ntr, bool il) {
  return ntr == 1 ? (il ? 1 : 3) : ntr == 2 ? (il ? 2 : 1) : 3;
}
FCT_STREAM_LIMIT_KERNEL(k_stream_limit, stream_blocks, slot_batch)

#define FCT_COUNT(V) d.max_nseg[V]
FCT_STREAM_LAUNCHER(launch_stream, k_stream_limit, FCT_COUNT, FCT_LIMIT_GRID, kStageLimit, stream_blocks)
FCT_SEG_LAUNCHER(launch_impl, k_seg_limit, FCT_COUNT, FCT_LIMIT_GRID, kStageLimit)
#undef FCT_COUNT

}  // namespace

int launch_seg_limit(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1,
                     cudaStream_t s) {
  if (d.smap_levels[kStageLimit] == 1) return launch_stream(single, tab, n, d, c0, c1, s);
  return launch_impl(single, tab, n, d, c0, c1, s);
}

}  // namespace fct
