// Input producer on the GPU: vertical velocity from continuity, fesom_jax/ale.py:309-365
// (``compute_w(mesh, uv, helem)``), the function the reference's step calls right before
// the FCT (fesom_jax/step.py:367) to produce ``w_e``.
//
// For each node level, the edge->node antisymmetric divergence is gathered over the
// node's incident edges in ascending edge id (the order in which the reference's
// segment_sum over the flattened [edge, 2] contributions adds them), then a bottom-to-top
// running sum gives w, divided by ``area`` (safe where 0) and masked to the node's
// interfaces.
#include <algorithm>
#include <cstdint>

#include "fct_div.cuh"
#include "fct_host.h"

using namespace fct;

namespace {

// A block takes kWColumns node columns: all threads gather the divergence of the columns' wet
// levels (levels adjacent), one thread per column adds them bottom to top in shared memory (in
// the sequential order, so the sum is the reference's), and all threads write w. (With a warp
// per column and the running sum through shuffles the kernel executed 1,700 warp-instructions
// per column, half of them shuffles and idle levels, and was issue-bound: 340 us on the
// CORE2-size mesh.)
constexpr int kWColumns = 16, kWThreads = 256;

// u and v of element level q: one 16-byte load, or two of 8 bytes where the caller's uv starts
// at an odd double.
template <bool Pairs>
__device__ __forceinline__ double2 uv_at(const double* __restrict__ uv, uint32_t q) {
  if constexpr (Pairs) return __ldg(reinterpret_cast<const double2*>(uv) + q);
  return make_double2(__ldg(uv + 2 * size_t(q)), __ldg(uv + 2 * size_t(q) + 1));
}

template <bool Pairs>
__device__ __forceinline__ void compute_w_columns(const DevMesh& m, const double* __restrict__ uv,
                                                  const double* __restrict__ helem,
                                                  double* __restrict__ w, int n0, double* sh) {
  if (n0 >= m.N) return;   // block-uniform
  const int L = m.L, stride = L | 1;
  for (int i = threadIdx.x; i < kWColumns * L; i += kWThreads) {
    const int col = i / L, k = i - col * L, n = n0 + col;
    if (n >= m.N) break;
    const int4 rec = __ldg(m.nrec + n);
    const unsigned pk = unsigned(rec.z);
    if (!m.edges_outside && (k < int(pk & 255u) || k >= int((pk >> 8) & 255u)))
      continue;   // no edge has the level
    const int e1 = rec.x + int((pk >> 16) & 255u);
    double div = 0.0;
#pragma unroll 2
    for (int j = rec.x; j < e1; ++j) {
      const int4 sl = __ldg(m.nw4 + j);
      const unsigned tr = unsigned(sl.z);
      const bool on1 = k >= int(tr & 255u) && k < int((tr >> 8) & 255u);
      const bool on2 = ((tr >> 16) & 255u) != kNoCell && k >= int((tr >> 16) & 255u) &&
                       k < int(tr >> 24);
      const double2* cr = reinterpret_cast<const double2*>(m.cross + 4 * int64_t(sl.w >> 1));
      const double2 x1 = __ldg(cr), x2 = __ldg(cr + 1);
      double2 U1 = make_double2(0.0, 0.0), U2 = U1;
      double h1 = 0.0, h2 = 0.0;
      if (on1) {
        U1 = uv_at<Pairs>(uv, uint32_t(sl.x) + uint32_t(k));
        h1 = __ldg(helem + (uint32_t(sl.x) + uint32_t(k)));
      }
      if (on2) {
        U2 = uv_at<Pairs>(uv, uint32_t(sl.y) + uint32_t(k));
        h2 = __ldg(helem + (uint32_t(sl.y) + uint32_t(k)));
      }
      const double t1 = on1 ? (U1.y * x1.x - U1.x * x1.y) * h1 : 0.0;
      const double t2 = on2 ? (U2.y * x2.x - U2.x * x2.y) * h2 : 0.0;
      const double c = t1 - t2;
      if (on1 || on2) div += (sl.w & 1) ? -c : c;
    }
    sh[col * stride + k] = div;
  }
  __syncthreads();
  if (threadIdx.x < kWColumns && n0 + int(threadIdx.x) < m.N) {
    const int n = n0 + threadIdx.x;
    const int lo = m.edges_outside ? 0 : __ldg(m.nzmin + n);
    const int hi = m.edges_outside ? L : __ldg(m.nzmax + n);
    double* s = sh + threadIdx.x * stride;
    double acc = 0.0;
    for (int k = hi - 1; k >= lo; --k) s[k] = acc += s[k];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kWColumns * L; i += kWThreads) {
    const int col = i / L, k = i - col * L, n = n0 + col;
    if (n >= m.N) break;
    const int nzmin = __ldg(m.nzmin + n), nzmax = __ldg(m.nzmax + n);
    const int64_t q = int64_t(n) * L + k;
    const double a = __ldg(m.area + q);
    // the bottom interface nzmax carries 0 unless an edge reaches below it
    w[q] = (k >= nzmin && (k < nzmax || (m.edges_outside && k == nzmax))) ? sh[col * stride + k] / (a > 0.0 ? a : 1.0) : 0.0;
  }
}

template <bool Pairs>
__global__ void __launch_bounds__(kWThreads) k_compute_w(const DevMesh* __restrict__ mp,
                                                         const double* __restrict__ uv,
                                                         const double* __restrict__ helem,
                                                         double* __restrict__ w) {
  __shared__ double sh[kWColumns * (kMaxLevels + 1)];
  compute_w_columns<Pairs>(*mp, uv, helem, w, int(blockIdx.x) * kWColumns, sh);
}

// batched: instance blockIdx.y of a device table derives its w into w_derived
__global__ void __launch_bounds__(kWThreads) k_compute_w_n(const Inst* __restrict__ tab) {
  __shared__ double sh[kWColumns * (kMaxLevels + 1)];
  const Inst& in = tab[blockIdx.y];
  if (!in.w_derived) return;
  compute_w_columns<true>(in.m, in.uv, in.helem, in.w_derived, int(blockIdx.x) * kWColumns, sh);
}

}  // namespace

namespace fct {

int launch_compute_w_tab(const Inst* tab, int n, int64_t max_nodes, cudaStream_t s) {
  const dim3 g(unsigned(std::max<int64_t>(1, (max_nodes + kWColumns - 1) / kWColumns)),
               unsigned(n), 1);
  k_compute_w_n<<<g, kWThreads, 0, s>>>(tab);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "compute_w (batched) launch");
}

}  // namespace fct

extern "C" int fct_compute_w(FctPlan* P, const double* uv, const double* helem, double* w,
                             fct_stream_t stream) {
  if (!P || !uv || !helem || !w) return set_error(FCT_ERR_INVALID, "NULL argument");
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != P->device) cudaSetDevice(P->device);
  const int blocks = (P->N + kWColumns - 1) / kWColumns;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // uv may start at any double; the pair loads need a 16-byte boundary
  if (reinterpret_cast<uintptr_t>(uv) % 16 == 0)
    k_compute_w<true><<<blocks, kWThreads, 0, s>>>(P->d_mesh, uv, helem, w);
  else
    k_compute_w<false><<<blocks, kWThreads, 0, s>>>(P->d_mesh, uv, helem, w);
  cudaError_t e = cudaGetLastError();
  if (prev >= 0 && prev != P->device) cudaSetDevice(prev);
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "compute_w launch");
}

namespace {

// divr (shared-reciprocal division) against the native IEEE division, bit for bit
__global__ void __launch_bounds__(256) k_div_check(const double* __restrict__ x,
                                                   const double* __restrict__ y, int64_t n,
                                                   unsigned long long* result) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const double a = x[i] / y[i];
    const double b = fct::divr(x[i], fct::rcp(y[i]));
    if (__double_as_longlong(a) != __double_as_longlong(b)) {
      atomicAdd(result, 1ull);
      atomicMin(result + 1, static_cast<unsigned long long>(i));
    }
  }
}

}  // namespace

extern "C" int fct_div_check(const double* x, const double* y, int64_t n,
                             unsigned long long* result, fct_stream_t stream) {
  if (!x || !y || !result || n < 0) return set_error(FCT_ERR_INVALID, "invalid argument");
  if (n == 0) return FCT_OK;
  const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 16);
  k_div_check<<<unsigned(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, y, n, result);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "div_check launch");
}
