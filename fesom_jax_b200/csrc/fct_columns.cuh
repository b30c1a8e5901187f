// Column solves staged through shared memory: the implicit vertical diffusion and the
// implicit part of the split vertical velocity. A tridiagonal recursion is sequential in the
// level, so one thread walks a column; read straight from memory every step of that walk
// waits for a strided load (T of 60,000 columns x 48 levels: 212 us per tracer at 32% of the
// memory rate with 11% of the issue slots used). Here a block takes a few columns:
//   1. all threads form the rows' coefficients and right-hand sides, levels adjacent (whole
//      lines), into shared memory;
//   2. one lane per column, or with several tracers two or four of a warp, eliminate and
//      substitute back in shared memory (rows padded to an odd length, so that neighbouring
//      columns use different banks), the block's tracers divided among them, in registers: the
//      walk's chain is the matrix recursion's, and the tracers' and the next row's loads fit
//      beside it;
//   3. all threads write the result, levels adjacent.
// What bounds it is that chain (about 20 dependent operations a level), so the blocks are
// small and many: 3 + (tracers) values per row and column.
#pragma once

#include "fct_device.cuh"

namespace fct {
namespace {

constexpr int kColThreads = 256;
constexpr int kColMaxTracers = 8;        // right-hand sides of a block
constexpr int kColMaxSmem = 227 << 10;   // opt-in shared memory of a block

// Shared rows of a block: a, b, c (then cp) of the matrix and one right-hand side per tracer,
// each [columns][stride].
struct ColRows {
  double *a, *b, *c, *r;
  int stride, columns;
  __device__ __forceinline__ ColRows(double* sh, int columns_, int L)
      : stride(L | 1), columns(columns_) {
    const int n = columns * stride;
    a = sh;
    b = sh + n;
    c = sh + 2 * n;
    r = sh + 3 * n;
  }
  __device__ __forceinline__ int at(int col, int k) const { return col * stride + k; }
  __device__ __forceinline__ double* rhs(int t) const { return r + t * columns * stride; }
};

inline size_t col_smem(int columns, int L, int nt) {
  return size_t(columns) * size_t(L | 1) * size_t(3 + nt) * sizeof(double);
}
// Columns per block: 16, or 8 where 16 would leave fewer than four blocks on an SM.
inline int col_columns(int L, int nt) { return col_smem(16, L, nt) <= size_t(56) << 10 ? 16 : 8; }

// x / y for the NT + 1 dividends of a row, correctly rounded (fct_div.cuh) and without a branch
// per quotient; operands outside the products' range take the native division.
__device__ __noinline__ double col_div_slow(double x, double y) { return x / y; }
__device__ __forceinline__ bool col_div_ok(double x) { return x == 0.0 || div_exp_ok(x); }
__device__ __forceinline__ double col_div(double x, double y, double r) {
  const double q0 = x * r;
  const double q1 = fma(fma(-y, q0, x), r, q0);
  const double q2 = fma(fma(-y, q1, x), r, q1);
  return x == 0.0 ? q0 : q2;
}

// Thomas algorithm over the rows [nzmin, nzmax) of every column of the block (fesom_jax/
// ops.py:121-168; the padded rows above and below solve to exactly 0). The solutions replace
// the right-hand sides. Every thread of the block calls one of the two forms, after a barrier;
// lanes of the first warp work.
//
// One tracer: one lane per column (more lanes would only add traffic: 201 us against 253 for
// 127,000 nodes x 48 levels).
__device__ __forceinline__ void col_solve_one(const DevMesh& m, const ColRows& s, int n0) {
  const int col = threadIdx.x, n = n0 + col;
  if (col < s.columns && n < m.N) {
    const int nzmin = ld(m.nzmin + n), nzmax = ld(m.nzmax + n);
    double cp = 0.0, dp = 0.0, an = 0.0, bn = 1.0, cn = 0.0, rn = 0.0;
    int i = s.at(col, nzmin);
    if (nzmin < nzmax) {
      an = s.a[i]; bn = s.b[i]; cn = s.c[i]; rn = s.r[i];
    }
    for (int k = nzmin; k < nzmax; ++k, ++i) {
      const double a = an, c = cn, y = bn - a * cp, x = rn - a * dp;
      if (k + 1 < nzmax) {   // the next row beside this one's chain
        an = s.a[i + 1]; bn = s.b[i + 1]; cn = s.c[i + 1]; rn = s.r[i + 1];
      }
      const double r = __drcp_rn(y);
      cp = col_div(c, y, r);
      dp = col_div(x, y, r);
      if (!(div_exp_ok(y) && col_div_ok(c) && col_div_ok(x))) {
        cp = col_div_slow(c, y);
        dp = col_div_slow(x, y);
      }
      s.c[i] = cp;
      s.r[i] = dp;
    }
    double v = 0.0;
    for (int k = nzmax - 1; k >= nzmin; --k) {
      --i;
      v = s.r[i] - s.c[i] * v;
      s.r[i] = v;
    }
  }
  __syncthreads();
}

// Several tracers: G = 32 / C lanes share a column (C columns in the block), each carries the
// matrix recursion and TPL of the tracers, because a row's instructions bound the walk (one
// lane per column with 8 tracers in its registers: 786 us for 30,000 nodes x 70 levels, 2,195
// for 127,000 x 48; so 428 and 1,215; two tracers 146 and 318, so 141 and 306).
// The lanes step through their rows together, for the longest column of the warp: a column's
// first lane writes cp over c, after the others of the column have read it.
template <int NT, int C>
__device__ __forceinline__ void col_solve(const DevMesh& m, const ColRows& s, int n0) {
  constexpr int G = 32 / C, TPL = (NT + G - 1) / G;
  if (threadIdx.x < 32) {
    const int col = int(threadIdx.x) % C, g = int(threadIdx.x) / C, n = n0 + col;
    const bool in_mesh = n < m.N;
    const int nzmin = in_mesh ? ld(m.nzmin + n) : 0;
    const int len = in_mesh ? max(0, ld(m.nzmax + n) - nzmin) : 0;   // rows of the column
    const int rows = __reduce_max_sync(0xffffffffu, len);
    const int first = s.at(col, nzmin);
    double* rt[TPL];   // the lane's right-hand sides; past the last tracer, the last again
    bool own[TPL];     //   (read, not written)
#pragma unroll
    for (int t = 0; t < TPL; ++t) {
      own[t] = g * TPL + t < NT;
      rt[t] = s.rhs(own[t] ? g * TPL + t : NT - 1) + first;
    }
    double cp = 0.0, dp[TPL], an = 0.0, bn = 1.0, cn = 0.0, rn[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) dp[t] = rn[t] = 0.0;
    if (len > 0) {
      an = s.a[first]; bn = s.b[first]; cn = s.c[first];
#pragma unroll
      for (int t = 0; t < TPL; ++t) rn[t] = rt[t][0];
    }
    for (int i = 0; i < rows; ++i) {
      const double a = an, c = cn, y = bn - a * cp;
      double x[TPL];
#pragma unroll
      for (int t = 0; t < TPL; ++t) x[t] = rn[t] - a * dp[t];
      if (i + 1 < len) {   // the next row beside this one's chain
        an = s.a[first + i + 1]; bn = s.b[first + i + 1]; cn = s.c[first + i + 1];
#pragma unroll
        for (int t = 0; t < TPL; ++t) rn[t] = rt[t][i + 1];
      }
      if (i < len) {
        bool ok = div_exp_ok(y) && col_div_ok(c);
#pragma unroll
        for (int t = 0; t < TPL; ++t) ok = ok && col_div_ok(x[t]);
        const double r = __drcp_rn(y);
        cp = col_div(c, y, r);
#pragma unroll
        for (int t = 0; t < TPL; ++t) dp[t] = col_div(x[t], y, r);
        if (!ok) {
          cp = col_div_slow(c, y);
#pragma unroll
          for (int t = 0; t < TPL; ++t) dp[t] = col_div_slow(x[t], y);
        }
      }
      __syncwarp();
      if (i < len) {
        if (g == 0) s.c[first + i] = cp;
#pragma unroll
        for (int t = 0; t < TPL; ++t)
          if (own[t]) rt[t][i] = dp[t];
      }
    }
    __syncwarp();
    double v[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) v[t] = 0.0;
    for (int i = len - 1; i >= 0; --i) {
      const double q = s.c[first + i];
#pragma unroll
      for (int t = 0; t < TPL; ++t)
        if (own[t]) rt[t][i] = v[t] = rt[t][i] - q * v[t];
    }
  }
  __syncthreads();
}

template <int NT>
__device__ __forceinline__ void col_solve_block(const DevMesh& m, const ColRows& s, int n0) {
  if constexpr (NT == 1) col_solve_one(m, s, n0);
  else if (s.columns == 16) col_solve<NT, 16>(m, s, n0);
  else col_solve<NT, 8>(m, s, n0);
}

// ------------- implicit vertical diffusion (tracer_diff.py:68-123, ops.py:121-168) of the
// tracers [t0, t0 + nt) of the columns [n0, n0 + columns)
template <int nt, bool IL>
__device__ __forceinline__ void block_vdiff(const Inst& in, int n0, int columns, int t0,
                                            double* sh) {
  const DevMesh& m = in.m;
  if (!in.Kv || n0 >= m.N) return;   // block-uniform
  const int L = m.L;
  const ColRows s(sh, columns, L);
  const int64_t ts = in.tstride;
  const int tg = in.tg;
  const double* Tin = in.vd_T;
  const double dt = in.dt;
  for (int i = threadIdx.x; i < columns * L; i += kColThreads) {
    const int col = i / L, k = i - col * L, n = n0 + col;
    if (n >= m.N) break;
    const int nzmin = ld(m.nzmin + n), nzmax = ld(m.nzmax + n);
    if (k < nzmin || k >= nzmax) continue;
    const uint32_t base = lq(n, L, 0), q = base + uint32_t(k);
    const double* Zc = in.vd_Z3d ? in.vd_Z3d + base : m.Zp;
    const bool last = k + 1 >= L;
    double dzu = k == 0 ? 0.0 : ld(Zc + k - 1) - ld(Zc + k);
    double dzd = ld(Zc + k) - (last ? 0.0 : ld(Zc + k + 1));
    dzu = dzu == 0.0 ? 1.0 : dzu;
    dzd = dzd == 0.0 ? 1.0 : dzd;
    const double av = ld(m.areasvol + q);
    const double sav = av > 0.0 ? av : 1.0;
    const double ar = ld(m.area + q), arp = last ? 0.0 : ld(m.area + q + 1);
    const double kv = ld(in.Kv + q), kvp = last ? 0.0 : ld(in.Kv + q + 1);
    const double a_full = -kv * dt / dzu * (ar / sav);
    const double c_full = -kvp * dt / dzd * (arp / sav);
    const double a = k == nzmin ? 0.0 : a_full;
    const double c = k == nzmax - 1 ? 0.0 : c_full;
    const int j = s.at(col, k);
    s.a[j] = a;
    s.c[j] = c;
    s.b[j] = -a - c + ld(in.hnode_new + q);
    double swd = 0.0;
    if (in.sw_3d) {
      const double sw = ld(in.sw_3d + q), swp = last ? 0.0 : ld(in.sw_3d + q + 1);
      swd = (sw - swp * (arp / sav)) * dt;
    }
    for (int t = 0; t < nt; ++t) {
      const double Tc = Tin[tix<IL>(q, t0 + t, ts, tg)];
      const double Tm = Tin[tix<IL>(k > 0 ? q - 1 : q, t0 + t, ts, tg)];
      const double Tp = last ? 0.0 : Tin[tix<IL>(q + 1, t0 + t, ts, tg)];
      double rhs = a * (Tc - Tm) + c * (Tc - Tp);
      if (in.bc_surf)
        rhs = rhs + (k == nzmin ? ld(in.bc_surf + (t0 + t) * in.bc_stride + n) : 0.0);
      if (in.sw_3d && t0 + t == in.sw_tracer) rhs = rhs + swd;
      s.rhs(t)[j] = rhs;
    }
  }
  __syncthreads();
  col_solve_block<nt>(m, s, n0);
  const bool copy = Tin != in.T_new;   // out of place: dry levels keep T
  if constexpr (IL) {
    for (int i = threadIdx.x; i < columns * L * nt; i += kColThreads) {
      const int e = i / nt, t = i - e * nt, col = e / L, k = e - col * L, n = n0 + col;
      if (n >= m.N) break;
      const int64_t o = tix<IL>(lq(n, L, k), t0 + t, ts, tg);
      if (k >= ld(m.nzmin + n) && k < ld(m.nzmax + n)) in.T_new[o] = Tin[o] + s.rhs(t)[s.at(col, k)];
      else if (copy) in.T_new[o] = Tin[o];
    }
  } else {
    for (int t = 0; t < nt; ++t)
      for (int i = threadIdx.x; i < columns * L; i += kColThreads) {
        const int col = i / L, k = i - col * L, n = n0 + col;
        if (n >= m.N) break;
        const int64_t o = tix<IL>(lq(n, L, k), t0 + t, ts, tg);
        if (k >= ld(m.nzmin + n) && k < ld(m.nzmax + n))
          in.T_new[o] = Tin[o] + s.rhs(t)[s.at(col, k)];
        else if (copy) in.T_new[o] = Tin[o];
      }
  }
}

// The same for eight interleaved tracers of many columns, in place, straight from memory: a
// thread walks a column with a tracer pair, the four pairs of a column are adjacent, so each
// level is one whole line, and many walks hide each other's loads. It needs the threads: above
// half of the resident ones (kPairColumns) it wins (us a step, walks / shared memory: 127,000
// nodes x 48 levels 499 / 793, four such members 1,953 / 3,126, 16 pi members 290 / 352, 8
// 151 / 183, 30,000 x 70 levels 232 / 288; 20,000 columns the same, 4 pi members 133 / 100).
// With four tracers, half a line, the two are equal on large members and shared memory wins on
// the others. cp and dp wait in the workspace's adfv and lo, which the step has finished with; a
// batch has no surface flux and no shortwave.
constexpr int kPairTracers = 8, kPairBlocks = 5;
constexpr int64_t kPairColumns = int64_t(148) * kPairBlocks * 256 / 2 / (kPairTracers / 2);
__device__ __forceinline__ void pair_vdiff(const Inst& in, int64_t n, int t0, int w0) {
  const DevMesh& m = in.m;
  if (n >= m.N || !in.Kv) return;
  const int L = m.L;
  const int nzmin = ld(m.nzmin + n), nzmax = ld(m.nzmax + n);
  const uint32_t base = lq(int(n), L, 0);
  const int tg = in.tg;
  double* __restrict__ T = in.T_new;
  double* __restrict__ lo = in.ws.lo;
  double* __restrict__ cps = in.ws.adfv;
  auto get = [](const double* p, uint32_t q, int t, int g, double (&v)[2]) {
    const double2 x = *reinterpret_cast<const double2*>(p + (q * uint32_t(g) + uint32_t(t)));
    v[0] = x.x;
    v[1] = x.y;
  };
  auto put = [](double* p, uint32_t q, int t, int g, const double (&v)[2]) {
    *reinterpret_cast<double2*>(p + (q * uint32_t(g) + uint32_t(t))) = make_double2(v[0], v[1]);
  };
  const int wtg = in.wtg;
  if (nzmax <= nzmin) return;
  const double dt = in.dt;
  const double* Zc = in.vd_Z3d ? in.vd_Z3d + base : m.Zp;
  double cprev = 0.0, dprev[2] = {0.0, 0.0}, Tm[2], Tc[2], Tp[2];
  get(T, base + uint32_t(nzmin), t0, tg, Tc);
  get(T, base + uint32_t(nzmin > 0 ? nzmin - 1 : 0), t0, tg, Tm);
  for (int k = nzmin; k < nzmax; ++k) {
    const uint32_t q = base + uint32_t(k);
    const bool last = k + 1 >= L;
    Tp[0] = Tp[1] = 0.0;
    if (!last) get(T, q + 1, t0, tg, Tp);
    double dzu = k == 0 ? 0.0 : ld(Zc + k - 1) - ld(Zc + k);
    double dzd = ld(Zc + k) - (last ? 0.0 : ld(Zc + k + 1));
    dzu = dzu == 0.0 ? 1.0 : dzu;
    dzd = dzd == 0.0 ? 1.0 : dzd;
    const double av = ld(m.areasvol + q);
    const double sav = av > 0.0 ? av : 1.0;
    const double ar = ld(m.area + q), arp = last ? 0.0 : ld(m.area + q + 1);
    const double kv = ld(in.Kv + q), kvp = last ? 0.0 : ld(in.Kv + q + 1);
    const double a_full = -kv * dt / dzu * (ar / sav);
    const double c_full = -kvp * dt / dzd * (arp / sav);
    const double a = k == nzmin ? 0.0 : a_full;
    const double c = k == nzmax - 1 ? 0.0 : c_full;
    const double b = -a - c + ld(in.hnode_new + q);
    const Rcp rm = rcp(b - a * cprev);
    cprev = divr(c, rm);
    cps[q * uint32_t(wtg) + uint32_t(w0)] = cprev;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const double rhs = a * (Tc[t] - Tm[t]) + c * (Tc[t] - Tp[t]);
      dprev[t] = divr(rhs - a * dprev[t], rm);
      Tm[t] = Tc[t];
      Tc[t] = Tp[t];
    }
    put(lo, q, w0, wtg, dprev);
  }
  double x[2] = {0.0, 0.0}, Tn[2];
  get(T, base + uint32_t(nzmax - 1), t0, tg, Tn);
#pragma unroll 2
  for (int k = nzmax - 1; k >= nzmin; --k) {
    const uint32_t q = base + uint32_t(k);
    double d[2], Tv[2] = {Tn[0], Tn[1]};
    const double c = cps[q * uint32_t(wtg) + uint32_t(w0)];
    get(lo, q, w0, wtg, d);
    if (k > nzmin) get(T, q - 1, t0, tg, Tn);   // ahead of the store
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      x[t] = d[t] - c * x[t];
      Tv[t] = Tv[t] + x[t];
    }
    put(T, q, t0, tg, Tv);
  }
}

// ---------------------------- adv_tra_vert_impl (tracer_adv.py:487-529): implicit w_i
// advection of LO, the tracers' workspace slots [w0, w0 + nt)
template <int nt, bool IL>
__device__ __forceinline__ void block_vert_impl(const Inst& in, int n0, int columns, int w0,
                                                double* sh) {
  const DevMesh& m = in.m;
  if (!in.w_i || n0 >= m.N) return;   // block-uniform
  const int L = m.L;
  const ColRows s(sh, columns, L);
  const int64_t sN = in.ws.sN;
  const double dt = in.dt;
  double* LO = in.ws.lo;
  for (int i = threadIdx.x; i < columns * L; i += kColThreads) {
    const int col = i / L, k = i - col * L, n = n0 + col;
    if (n >= m.N) break;
    const int nzmin = ld(m.nzmin + n), nzmax = ld(m.nzmax + n);
    if (k < nzmin || k >= nzmax) continue;
    const uint32_t q = lq(n, L, k);
    const double av = ld(m.areasvol + q);
    const double sa = av > 0.0 ? av : 1.0;
    const double v_top = dt * ld(m.area + q) / sa;
    const double v_bot = dt * (k + 1 < L ? ld(m.area + q + 1) : 0.0) / sa;
    const double wu = ld(in.w_i + q), wd = k + 1 < L ? ld(in.w_i + q + 1) : 0.0;
    const bool surf = k == nzmin, bot = k == nzmax - 1;
    const double a = (surf ? 0.0 : fmin(0.0, wu)) * v_top;
    const double b_top = (surf ? wu : fmax(0.0, wu)) * v_top;
    const double b_bot = (bot ? 0.0 : -fmin(0.0, wd)) * v_bot;
    const double c = (bot ? 0.0 : -fmax(0.0, wd)) * v_bot;
    const double b_adv = b_top + b_bot;
    const int j = s.at(col, k);
    s.a[j] = a;
    s.c[j] = c;
    s.b[j] = ld(in.hnode_new + q) + b_adv;
    for (int t = 0; t < nt; ++t) {
      // the neighbours above the surface and below the bottom enter with a zero
      // coefficient; LO is 0 there in the reference, and this step never wrote them
      const double Tm = surf ? 0.0 : LO[tix<IL>(q - 1, w0 + t, sN, in.wtg)];
      const double T0 = LO[tix<IL>(q, w0 + t, sN, in.wtg)];
      const double Tp = bot ? 0.0 : LO[tix<IL>(q + 1, w0 + t, sN, in.wtg)];
      s.rhs(t)[j] = -(a * Tm + b_adv * T0 + c * Tp);
    }
  }
  __syncthreads();
  col_solve_block<nt>(m, s, n0);
  for (int t = 0; t < nt; ++t)
    for (int i = threadIdx.x; i < columns * L; i += kColThreads) {
      const int col = i / L, k = i - col * L, n = n0 + col;
      if (n >= m.N) break;
      if (k < ld(m.nzmin + n) || k >= ld(m.nzmax + n)) continue;
      const int64_t o = tix<IL>(lq(n, L, k), w0 + t, sN, in.wtg);
      LO[o] = LO[o] + s.rhs(t)[s.at(col, k)];
    }
}

}  // namespace
}  // namespace fct
