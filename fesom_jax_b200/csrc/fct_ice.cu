// Sea-ice FCT advection (fesom_jax/ice_adv.py:37-194, fesom_ice_fct.c): one step of the
// three ice tracers (a_ice, m_ice, m_snow) on the surface mesh.
//
// The reference scatters element contributions to nodes; here every node gathers over
// its cells (node->element CSR in the reference's nod_in_elem2D order, the node's vertex
// index packed in the slot) so sums are deterministic and no atomics are needed. A thread
// takes a node and one tracer (blockIdx.y); the right-hand side, whose matrix row is the same
// for all tracers, a node and all three. The kernels wait on their gathers: with all three
// tracers in one thread the CORE2-size mesh filled a third of the warp slots, and every flux
// divided by 12 through the full division sequence. Now the mesh's quotients come from the
// plan, quotients by 12 and 9 are correctly rounded products (fct_div.cuh), and a cell's slot
// is loaded one ahead.
//
//   k_ice_rhs    _tg_rhs (:47-75), _mm_times (:37-44), _solve_low_order (:78-89),
//                first high-order approximation (:103)
//   k_ice_hi     one high-order residual correction (:104-107), launched twice
//   k_ice_limit  _fem_fct antidiffusive fluxes, cluster bounds, clipping ratios (:126-160)
//   k_ice_apply  _fem_fct limited flux application (:162-172)
#include <algorithm>

#include "fct_div.cuh"
#include "fct_host.h"

using namespace fct;

namespace {

constexpr double kIceFluxEps = 1.0e-12;   // ice_adv.py:34
constexpr int B = 128;

struct IceArgs {
  DevMesh m;
  const double* X[3];   // a_ice, m_ice, m_snow
  const double *u, *v;
  double* out[3];
  double *rhs, *xl, *d0, *d1, *pp, *pm;   // workspace, each [3][nod2D]
  double dt, gamma, diff;
};

__device__ __forceinline__ int64_t node_index() {
  return int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
}
// x / 12 and x / 9, correctly rounded
__device__ __forceinline__ double div12(double x) { return divr(x, Rcp{12.0, 1.0 / 12.0, true}); }
__device__ __forceinline__ double div9(double x) { return divr(x, Rcp{9.0, 1.0 / 9.0, true}); }

// A node's cells in order, the slot records one ahead: ``sl`` {cell, its vertices}, ``p`` the
// node's place among them, ``on`` not a cavity cell.
#define ICE_FOR_CELLS(c0, c1)                                                     \
  int4 sl_nx = (c0) < (c1) ? __ldg(m.nel4 + (c0)) : make_int4(0, 0, 0, 0);        \
  int r_nx = (c0) < (c1) ? __ldg(m.nelr + (c0)) : 0;                              \
  for (int j = (c0); j < (c1); ++j)
#define ICE_CELL(c1)                                                              \
  const int4 sl = sl_nx;                                                          \
  const int p = (r_nx >> 16) & 3;                                                 \
  const bool on = (r_nx & 255) == 0;                                              \
  if (j + 1 < (c1)) {                                                             \
    sl_nx = __ldg(m.nel4 + j + 1);                                                \
    r_nx = __ldg(m.nelr + j + 1);                                                 \
  }                                                                               \
  const int vq[3] = {sl.y, sl.z, sl.w};

__device__ __forceinline__ double pick(const double (&x)[3], int p) {
  return p == 0 ? x[0] : (p == 1 ? x[1] : x[2]);
}

__global__ void __launch_bounds__(B) k_ice_rhs(const __grid_constant__ IceArgs A) {
  const DevMesh& m = A.m;
  const int64_t n = node_index();
  if (n >= m.N) return;
  const int N = m.N;
  double rhs[3] = {0.0, 0.0, 0.0}, mmx[3] = {0.0, 0.0, 0.0};
  const int c0 = __ldg(m.nel_off + n), c1 = __ldg(m.nel_off + n + 1);
  ICE_FOR_CELLS(c0, c1) {
    ICE_CELL(c1)
    if (!on) continue;   // cavity cells contribute 0
    const double2* gs = reinterpret_cast<const double2*>(m.gsca + 6 * int64_t(sl.x));
    const double2 g0 = __ldg(gs), g1 = __ldg(gs + 1), g2 = __ldg(gs + 2);
    const double dx[3] = {g0.x, g0.y, g1.x}, dy[3] = {g1.y, g2.x, g2.y};
    const double vol = __ldg(m.earea + sl.x), vol12 = __ldg(m.earea12 + sl.x);
    double U[3], V[3], x[3][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      U[q] = __ldg(A.u + vq[q]);
      V[q] = __ldg(A.v + vq[q]);
#pragma unroll
      for (int t = 0; t < 3; ++t) x[t][q] = __ldg(A.X[t] + vq[q]);
    }
    const double um = U[0] + U[1] + U[2], vm = V[0] + V[1] + V[2];
    const double diff = A.diff * __ldg(m.ediff + sl.x);
    const double dxp = pick(dx, p), dyp = pick(dy, p);
    const double udnp = um * dxp + vm * dyp;
    double E[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double a = div12(dxp * (um + U[q]) + dyp * (vm + V[q]));
      const double b = diff * (dxp * dx[q] + dyp * dy[q]);
      const double udnq = um * dx[q] + vm * dy[q];
      const double c = div9(0.5 * A.dt * (udnp * udnq));
      E[q] = vol * A.dt * (a - b - c);
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      rhs[t] += E[0] * x[t][0] + E[1] * x[t][1] + E[2] * x[t][2];
      mmx[t] += vol12 * (pick(x[t], p) + (x[t][0] + x[t][1] + x[t][2]));
    }
  }
  const bool nc = __ldg(m.nzmin + n) <= 0;   // ulevels_nod2D <= 1
  const double ia = __ldg(m.iarea0 + n);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const double X = __ldg(A.X[t] + n);
    A.rhs[t * N + n] = rhs[t];
    A.d0[t * N + n] = nc ? rhs[t] * ia : 0.0;
    A.xl[t * N + n] = nc ? (rhs[t] + A.gamma * mmx[t]) * ia + (1.0 - A.gamma) * X : X;
  }
}

// d_out = d_in + (rhs - mm d_in) / area on open-water/ice nodes
__global__ void __launch_bounds__(B) k_ice_hi(const __grid_constant__ IceArgs A,
                                              const double* __restrict__ din_,
                                              double* __restrict__ dout) {
  const DevMesh& m = A.m;
  const int64_t n = node_index();
  if (n >= m.N) return;
  const int64_t o = int64_t(blockIdx.y) * m.N;
  const double* __restrict__ din = din_ + o;
  double mmd = 0.0;
  const int c0 = __ldg(m.nel_off + n), c1 = __ldg(m.nel_off + n + 1);
  ICE_FOR_CELLS(c0, c1) {
    ICE_CELL(c1)
    const double x[3] = {__ldg(din + vq[0]), __ldg(din + vq[1]), __ldg(din + vq[2])};
    const double s = __ldg(m.earea12 + sl.x) * (pick(x, p) + (x[0] + x[1] + x[2]));
    mmd = on ? mmd + s : mmd;
  }
  const bool nc = __ldg(m.nzmin + n) <= 0;
  const double ia = __ldg(m.iarea0 + n), d = din[n];
  dout[o + n] = nc ? d + (A.rhs[o + n] - mmd) * ia : d;
}

// the cell's antidiffusive flux at vertex q: -s_q (vol / area_q) / 12, s_q = sum w - 3 w_q
__device__ __forceinline__ double ice_flux(double sw, double wq, double vol, double iaq) {
  return div12(-(sw - 3.0 * wq) * (vol * iaq));
}

__global__ void __launch_bounds__(B) k_ice_limit(const __grid_constant__ IceArgs A,
                                                 const double* __restrict__ dv_) {
  const DevMesh& m = A.m;
  const int64_t n = node_index();
  if (n >= m.N) return;
  const int64_t o = int64_t(blockIdx.y) * m.N;
  const double* __restrict__ X = A.X[blockIdx.y];
  const double* __restrict__ dv = dv_ + o;
  const double* __restrict__ XL = A.xl + o;
  const double ia_n = __ldg(m.iarea0 + n);
  double fp = 0.0, fm = 0.0, hi = -INFINITY, lo = INFINITY;
  const int c0 = __ldg(m.nel_off + n), c1 = __ldg(m.nel_off + n + 1);
  ICE_FOR_CELLS(c0, c1) {
    ICE_CELL(c1)
    const double vol = __ldg(m.earea + sl.x);
    double w[3], xl[3], xv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      xv[q] = __ldg(X + vq[q]);
      w[q] = A.gamma * xv[q] + __ldg(dv + vq[q]);
      xl[q] = __ldg(XL + vq[q]);
    }
    if (!on) continue;
    const double sw = w[0] + w[1] + w[2];
    const double f = ice_flux(sw, pick(w, p), vol, ia_n);
    fp += fmax(f, 0.0);
    fm += fmin(f, 0.0);
    const double ehi = fmax(fmax(fmax(xl[0], xl[1]), xl[2]), fmax(fmax(xv[0], xv[1]), xv[2]));
    const double elo = fmin(fmin(fmin(xl[0], xl[1]), xl[2]), fmin(fmin(xv[0], xv[1]), xv[2]));
    hi = fmax(hi, ehi);
    lo = fmin(lo, elo);
  }
  const bool nc = __ldg(m.nzmin + n) <= 0;
  const double h = isfinite(hi) ? hi : 0.0, l = isfinite(lo) ? lo : 0.0;
  const double xl = XL[n];
  const double tmax = h - xl, tmin = l - xl;
  const double pp = fp > 0.0 ? fmin(tmax / (fp > kIceFluxEps ? fp : kIceFluxEps), 1.0) : 0.0;
  const double pm = fm < 0.0 ? fmin(tmin / (fm < -kIceFluxEps ? fm : -kIceFluxEps), 1.0) : 0.0;
  A.pp[o + n] = nc ? pp : 0.0;
  A.pm[o + n] = nc ? pm : 0.0;
}

__global__ void __launch_bounds__(B) k_ice_apply(const __grid_constant__ IceArgs A,
                                                 const double* __restrict__ dv_) {
  const DevMesh& m = A.m;
  const int64_t n = node_index();
  if (n >= m.N) return;
  const int64_t o = int64_t(blockIdx.y) * m.N;
  const double* __restrict__ X = A.X[blockIdx.y];
  const double* __restrict__ dv = dv_ + o;
  const double* __restrict__ pp = A.pp + o;
  const double* __restrict__ pm = A.pm + o;
  double acc = 0.0;
  const int c0 = __ldg(m.nel_off + n), c1 = __ldg(m.nel_off + n + 1);
  ICE_FOR_CELLS(c0, c1) {
    ICE_CELL(c1)
    const double vol = __ldg(m.earea + sl.x);
    double w[3], f[3], cand[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) w[q] = A.gamma * __ldg(X + vq[q]) + __ldg(dv + vq[q]);
    const double sw = w[0] + w[1] + w[2];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double a = __ldg(pp + vq[q]), b = __ldg(pm + vq[q]);
      f[q] = ice_flux(sw, w[q], vol, __ldg(m.iarea0 + vq[q]));
      cand[q] = f[q] >= 0.0 ? a : b;
    }
    const double ae = fmin(fmin(cand[0], cand[1]), cand[2]);
    acc = on ? acc + pick(f, p) * ae : acc;   // limited fluxes of cavity cells are 0
  }
  A.out[blockIdx.y][n] = A.xl[o + n] + acc;
}

}  // namespace

extern "C" int fct_ice_solve(FctPlan* P, const FctIceFields* f, const FctIceConfig* cfg,
                             fct_stream_t stream) {
  if (!P || !f || !cfg) return set_error(FCT_ERR_INVALID, "NULL argument");
  for (int t = 0; t < 3; ++t)
    if (!f->tracer[t] || !f->tracer_new[t])
      return set_error(FCT_ERR_INVALID, "ice tracer %d pointer is NULL", t);
  if (!f->u_ice || !f->v_ice) return set_error(FCT_ERR_INVALID, "ice velocity is NULL");
  if (!(cfg->dt > 0.0)) return set_error(FCT_ERR_INVALID, "dt must be positive");
  const int64_t N = P->N;
  // scratch: 6 fields of 3 x nod2D doubles, carved from the plan workspace's node fields
  // (LO onwards: at least kFusedNodeFields x nod2D x nl doubles per tracer, contiguous in
  // both workspace layouts)
  if (18 * N > kFusedNodeFields * N * P->L * int64_t(P->max_tracers))
    return set_error(FCT_ERR_CAPACITY, "plan workspace too small for the ice step");
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != P->device) cudaSetDevice(P->device);
  IceArgs A{};
  A.m = P->hm;
  for (int t = 0; t < 3; ++t) { A.X[t] = f->tracer[t]; A.out[t] = f->tracer_new[t]; }
  A.u = f->u_ice;
  A.v = f->v_ice;
  double* w = P->ws.lo;
  A.rhs = w; A.xl = w + 3 * N; A.d0 = w + 6 * N; A.d1 = w + 9 * N;
  A.pp = w + 12 * N; A.pm = w + 15 * N;
  A.dt = cfg->dt; A.gamma = cfg->gamma; A.diff = cfg->diff;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned g = unsigned((N + B - 1) / B);
  int st;
  {
    PlanUse use(P, s);
    st = use.status();
    if (!st) {
      k_ice_rhs<<<g, B, 0, s>>>(A);
      const dim3 g3(g, 3);
      k_ice_hi<<<g3, B, 0, s>>>(A, A.d0, A.d1);   // two residual corrections (ice_adv.py:104)
      k_ice_hi<<<g3, B, 0, s>>>(A, A.d1, A.d0);
      k_ice_limit<<<g3, B, 0, s>>>(A, A.d0);
      k_ice_apply<<<g3, B, 0, s>>>(A, A.d0);
      const cudaError_t e = cudaGetLastError();
      st = e == cudaSuccess ? use.release() : cuda_error(e, "ice FCT launch");
    }
  }
  if (prev >= 0 && prev != P->device) cudaSetDevice(prev);
  return st;
}
