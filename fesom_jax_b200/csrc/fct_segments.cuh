// Segment kernels of the fused forward step: the product path of fct_forward, the
// batched engine and the serving engine (fesom_jax/tracer_adv.py:532-578).
//
// One level per thread (the default), NTR tracers: the stream kernels, whose threads walk the
// layers or edge levels with adjacent threads on adjacent levels. Two or more levels per
// thread: a thread takes a *segment*, a run of up to LPT consecutive levels of one node (or one
// edge) and NTR tracers. The entity's neighbour slots, level range and static geometry
// are decoded once per segment and every neighbour gather issues LPT x NTR independent
// loads (consecutive levels of one column), instead of one level per thread re-decoding
// the same lists. Every quantity is the reference's expression; the arithmetic (below)
// trades correctly rounded quotients for reciprocal products and fused multiply-adds, so
// the results equal the one-kernel-per-stage path's to rounding (a few ulp per step), and
// every mapping and layout of these kernels gives the same bits.
//
// Stages (kernels over the plan's segment lists, fct_internal.cuh DevMesh):
//   seg_node_lo     node layers: LO (compute_fct_lo with adv_flux_hor/ver, :96-120,
//                   :298-313) and adf_v (adv_flux_ver_ho minus the LO vertical flux,
//                   :241-295, :568) on the tops of the layers; the bottom interface's
//                   adf_v is 0 and not stored (readers take 0 there)
//   seg_edge_adf    edge levels where MFCT takes the up/down cells' gradients
//                   (fill_up_dn_grad :344-368, adv_flux_hor_ho :196-225): adf_h
//   edge_fix        the other edge lanes: the node-average gradients (:329-341) of the
//                   two end nodes computed on the fly; at 1-2 % of the edge lanes of an
//                   open-ocean mesh this is cheaper than storing node gradients everywhere
//   seg_node_limit  zalesak_limit a1-a4, b1, b2 (:371-451): cluster bounds over the edge
//                   neighbours, the k-1/k/k+1 window (across runs through shared memory),
//                   the antidiffusive sums and the limiter factors
//   seg_node_final  b3, flux2dtracer_fct, ale_reconstruct (:453-484, :142-151): T_new
#pragma once

#include <algorithm>

#include "fct_device.cuh"

namespace fct {
namespace {

// Arithmetic of the segment kernels. Quotients multiply by the divisor's correctly rounded
// reciprocal (within 1.5 ulp of the quotient; the one-kernel-per-stage path rounds every
// quotient correctly instead), products that feed a sum fuse into FMAs written out in the
// source (--fmad=false keeps the compiler from contracting anything else, so every
// template instantiation rounds alike), and max/min are plain comparisons (the same values
// as fmax/fmin on the finite numbers the scheme carries).
struct Rcq {
  double r;
};
__device__ __forceinline__ Rcq rcpq(double y) { return Rcq{__drcp_rn(y)}; }
__device__ __forceinline__ double divq(double x, const Rcq& c) { return x * c.r; }
__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }
// AB2 extrapolation ttfAB = -0.6*T_old + 1.6*T (tracer_adv.py:59-66)
__device__ __forceinline__ double ab2f(double T, double To) { return fma(kAbNew, T, kAbOld * To); }

// The node kernels' neighbour loops load each slot record one slot ahead, so the next
// slot's gathers do not wait behind its record (2-4% faster per node kernel on the
// CORE2-size batched step)
#define FCT_SLOT_BEGIN(e0, e1) \
  int4 sl_nx = (e0) < (e1) ? __ldg(m.ns4 + (e0)) : make_int4(0, 0, 0, 0);
#define FCT_SLOT_GET(j, e1) \
  const int4 sl = sl_nx;    \
  if ((j) + 1 < (e1)) sl_nx = __ldg(m.ns4 + (j) + 1);

// a level clamped into [0, L - 1]: loads at clamped levels are in bounds and their values
// are discarded by the predicates that follow
__device__ __forceinline__ int kclamp(int k, int L) { return k < 0 ? 0 : (k >= L ? L - 1 : k); }

// A field of NTR tracers with its base addresses formed once per thread: interleaved, one
// address (tracer t0) indexed by entity-level x interleave stride; tracer-major, one per
// tracer indexed by the entity-level. The slot loops then form one 32-bit offset per slot
// and level and one 64-bit address per load.
template <int NTR, bool IL>
struct Fld {
  const double* p[IL ? 1 : NTR];
  __device__ __forceinline__ Fld(const double* base, int t0, int64_t stride) {
    if constexpr (IL) {
      p[0] = base + t0;
    } else {
#pragma unroll
      for (int i = 0; i < NTR; ++i) p[i] = base + int64_t(t0 + i) * stride;
    }
  }
  // the offset of entity-level q (below 2^32, see tix)
  __device__ __forceinline__ static uint32_t off(uint32_t q, int tg) {
    return IL ? q * uint32_t(tg) : q;
  }
  __device__ __forceinline__ void ld(uint32_t o, double (&v)[NTR]) const {
    if constexpr (IL && (NTR % 2 == 0)) {
      const double2* b = reinterpret_cast<const double2*>(p[0] + o);
#pragma unroll
      for (int i = 0; i < NTR; i += 2) {
        const double2 x = __ldg(b + i / 2);
        v[i] = x.x;
        v[i + 1] = x.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < NTR; ++i) v[i] = __ldg(IL ? p[0] + o + i : p[IL ? 0 : i] + o);
    }
  }
};

// x with its sign bit flipped where ``mask`` is 0x80000000 (0: unchanged)
__device__ __forceinline__ double flip_sign(double x, int mask) {
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

// ----------------------------------------------------------- LO and adf_v, node runs
template <int NTR, int LPT, bool IL>
__device__ __forceinline__ void seg_node_lo(const Inst& in, int64_t si, int t0, int w0) {
  const DevMesh& m = in.m;
  constexpr int V = seg_variant(LPT);
  if (si >= m.n_nseg[V]) return;
  const uint32_t sg = __ldg(m.nseg[V] + si);
  const int n = lane_ent(sg), k0 = lane_lev(sg), L = m.L;
  const int4 rec = __ldg(m.nrec + n);
  const unsigned pk = unsigned(rec.z);
  const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
  const int nk = min(LPT, nzmax - k0);   // layers of this run
  const uint32_t base = lq(n, L, 0);
  const int tg = in.tg;
  const double dt = in.dt;
  using F = Fld<NTR, IL>;
  const F fT(in.T, t0, in.tstride);
  unsigned onb[LPT];   // per layer of the run: bit j, the j-th slot's edge has the layer
  uint32_t kk[LPT];    // the run's layers (beyond the run: its first again, bits 0)
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    onb[l] = l < nk ? unsigned(__ldg(m.nflags + rec.w + (k0 + l - nzmin))) & kSlotBits : 0u;
    kk[l] = uint32_t(k0 + (l < nk ? l : 0));
  }

  // compute_fct_lo: edge->node upwind divergence in ascending edge id. With s the volume
  // flux out of the node, the face flux -0.5*(T1*(vf+|vf|) + T2*(vf-|vf|)) is -T*s of the
  // upwind end: outflows sum their s (times the own T once, after the loop), inflows add
  // |s| times the neighbour's T.
  double div[LPT][NTR], out[LPT];
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    out[l] = 0.0;
#pragma unroll
    for (int t = 0; t < NTR; ++t) div[l][t] = 0.0;
  }
  const int e0 = rec.x, e1 = rec.x + int((pk >> 16) & 255u);
  // U slots at a time: their gathers are all issued before any is used (in the limiter and the
  // final stage, which hold three values per slot and level, the registers cost more than it
  // gives). Slots past the node's last repeat it with their bits 0; a slot off at a layer reads
  // the own value, times 0.
  constexpr int U = 2;
  int4 sl[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    sl[u] = e0 < e1 ? __ldg(m.ns4 + min(e0 + u, e1 - 1)) : make_int4(0, 0, 0, 0);
  for (int j = e0; j < e1; j += U) {
    double vf[U][LPT], To[U][LPT][NTR];
    int sgn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      sgn[u] = sl[u].z;
#pragma unroll
      for (int l = 0; l < LPT; ++l) {
        const bool on = (onb[l] >> u) & 1u;
        vf[u][l] = __ldg(in.ws.vflux + (uint32_t(sl[u].x) + kk[l]));
        fT.ld(F::off((on ? uint32_t(sl[u].y) : base) + kk[l], tg), To[u][l]);
      }
    }
    if (j + U < e1) {
#pragma unroll
      for (int u = 0; u < U; ++u) sl[u] = __ldg(m.ns4 + min(j + U + u, e1 - 1));
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int l = 0; l < LPT; ++l) {
        const double s = flip_sign(vf[u][l], sgn[u]);
        const bool on = (onb[l] >> u) & 1u, leaves = s > 0.0;
        const double cin = (on && !leaves) ? -s : 0.0;
        if (on && leaves) out[l] += s;
#pragma unroll
        for (int t = 0; t < NTR; ++t) div[l][t] = fma(cin, To[u][l][t], div[l][t]);
      }
#pragma unroll
    for (int l = 0; l < LPT; ++l) onb[l] >>= U;
  }

  // T of the column at levels k0-2 .. k0+LPT (Tw[i] <-> level k0-2+i; the level above
  // the surface reads T[0], the reference's edge-replicated top)
  double Tw[LPT + 3][NTR];
#pragma unroll
  for (int i = 0; i < LPT + 3; ++i)
    fT.ld(F::off(base + uint32_t(kclamp(k0 - 2 + i, L)), tg), Tw[i]);

  // upwind vertical flux at the interfaces k0 .. k0+LPT (layer-masked, tracer_adv.py:108-120)
  double fv[LPT + 1][NTR];
#pragma unroll
  for (int i = 0; i <= LPT; ++i) {
    const int k = k0 + i, kc = kclamp(k, L);
    const bool layer = i <= nk && k < nzmax;
    const double w = __ldg(in.w_e + base + kc), ar = __ldg(m.area + base + kc);
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      fv[i][t] = layer ? vflux_up(Tw[i + 2][t], Tw[i + 1][t], w, ar) : 0.0;
  }
  // LO on the run's layers
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    if (l >= nk) break;
    const uint32_t qn = base + uint32_t(k0 + l);
    const double hn = __ldg(in.hnode + qn), hnn = __ldg(in.hnode_new + qn);
    const double iav = __ldg(m.iavol + qn);
    const double fdt = dt * iav;   // dt / areasvol
    const Rcq rhn = rcpq(hnn);
    const bool valid = (hnn > 0.0) && (iav > 0.0);
    double lo[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double dh = fma(-out[l], Tw[l + 2][t], div[l][t]);
      lo[t] = valid ? divq(fma(Tw[l + 2][t], hn, (dh + (fv[l][t] - fv[l + 1][t])) * fdt), rhn)
                    : 0.0;
    }
    stv<NTR, IL>(in.ws.lo, qn, w0, in.ws.sN, in.wtg, lo);
  }

  // adv_flux_ver_ho (QR4C on ttfAB) minus the LO vertical flux at the layer tops
  const F fTo(in.T_old, t0, in.tstride);
  double A[LPT + 3][NTR];   // ttfAB at levels k0-2 .. k0+LPT
#pragma unroll
  for (int i = 0; i < LPT + 3; ++i) {
    double To[NTR];
    fTo.ld(F::off(base + uint32_t(kclamp(k0 - 2 + i, L)), tg), To);
#pragma unroll
    for (int t = 0; t < NTR; ++t) A[i][t] = ab2f(Tw[i][t], To[t]);
  }
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    if (l >= nk) break;
    const int k = k0 + l;
    const uint32_t qn = base + uint32_t(k);
    const double w = __ldg(in.w_e + qn);
    const double Wf = in.w_i ? w + __ldg(in.w_i + qn) : w;
    const double area_k = __ldg(m.area + qn);
    double hi[NTR];
    if (k == nzmin) {
#pragma unroll
      for (int t = 0; t < NTR; ++t) hi[t] = -A[l + 2][t] * Wf * area_k;
    } else if (k == nzmin + 1 || k == nzmax - 1) {
#pragma unroll
      for (int t = 0; t < NTR; ++t) hi[t] = -0.5 * (A[l + 1][t] + A[l + 2][t]) * Wf * area_k;
    } else {   // nzmin + 2 <= k <= nzmax - 2
      // QR4C stencil (tracer_adv.py:228-238, 265-273): reciprocal depth gaps and a third of
      // the depths to the interface, from the plan's table or the moving depths
      double rdc, rdu, rdd, d1, d2;
      if (in.Z3d) {
        const double* Zc = in.Z3d + base;
        const double Znz = __ldg(Zc + k), Zm1 = __ldg(Zc + k - 1), Zm2 = __ldg(Zc + k - 2);
        const double Zp1 = __ldg(Zc + (k + 1 < L ? k + 1 : L - 1)), zb = __ldg(in.zbar3 + qn);
        rdc = __drcp_rn(safe_nz(Zm1 - Znz));
        rdu = __drcp_rn(safe_nz(Znz - Zp1));
        rdd = __drcp_rn(safe_nz(Zm2 - Zm1));
        d1 = (zb - Znz) * (1.0 / 3.0);
        d2 = (zb - Zm1) * (1.0 / 3.0);
      } else {
        const double* q = m.qr4c + k;
        rdc = __ldg(q);
        rdu = __ldg(q + L);
        rdd = __ldg(q + 2 * L);
        d1 = __ldg(q + 3 * L);
        d2 = __ldg(q + 4 * L);
      }
      const double wa = -0.5 * Wf * area_k;
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        const double qc = (A[l + 1][t] - A[l + 2][t]) * rdc;
        const double qu = (A[l + 2][t] - A[l + 3][t]) * rdu;
        const double qd = (A[l][t] - A[l + 1][t]) * rdd;
        const double Tmean1 = fma(fma(2.0, qc, qu), d1, A[l + 2][t]);
        const double Tmean2 = fma(fma(2.0, qc, qd), d2, A[l + 1][t]);
        hi[t] = (Tmean1 + Tmean2) * wa;
      }
    }
    double adf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double lo_v = in.w_i ? vflux_up(Tw[l + 2][t], Tw[l + 1][t], Wf, area_k) : fv[l][t];
      adf[t] = hi[t] - lo_v;
    }
    stv<NTR, IL>(in.ws.adfv, qn, w0, in.ws.sN, in.wtg, adf);
  }
}

// ---------------------------------------------- adf_h on a run of up/down-cell levels
// HO - LO = -0.5*((vf+|vf|)*(Tm1 - T1) + (vf-|vf|)*(Tm2 - T2)) is -vf*(Tm - T) of the
// upwind end alone, with Tm = A_u + (2*(A_d - A_u) + edx*a*gx + edy*R*gy)/6 over that end's
// cell (the up cell at the first node, the down cell at the second; its gradient is one
// weighted vertex sum whose weights carry the sign of the end). So a level gathers the six
// values of the upwind side instead of the eight of both. (A NaN on the downwind cell still
// reaches both ends: it makes LO, hence the limiter factors, of the downwind node NaN. After an
// infinite value one of that node's two factors may be finite, and the upwind end with it.)
template <int NTR, int LPT, bool IL>
__device__ __forceinline__ void seg_edge_adf(const Inst& in, int64_t si, int t0, int w0) {
  const DevMesh& m = in.m;
  constexpr int V = seg_variant(LPT);
  if (si >= m.n_eseg[V]) return;
  const uint32_t sg = __ldg(m.eseg[V] + si);
  const int e = lane_ent(sg), k0 = lane_lev(sg), L = m.L;
  const int4 er = __ldg(m.erec + e);
  const int nk = min(LPT, int((unsigned(er.z) >> 8) & 255u) - k0);
  const int4 ov = __ldg(m.emf4 + e);
  const double2* wp = reinterpret_cast<const double2*>(m.emfw + 8 * int64_t(e));
  const double2 u01 = __ldg(wp), u2x = __ldg(wp + 1), d01 = __ldg(wp + 2), d2x = __ldg(wp + 3);
  const uint32_t q1 = lq(er.x, L, k0), q2 = lq(er.y, L, k0), qe = lq(e, L, k0);
  const uint32_t qua = lq(ov.x, L, k0), qub = lq(ov.y, L, k0);
  const uint32_t qda = lq(ov.z, L, k0), qdb = lq(ov.w, L, k0);
  const int tg = in.tg;
  using F = Fld<NTR, IL>;
  const F fT(in.T, t0, in.tstride), fO(in.T_old, t0, in.tstride);
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    const uint32_t lc = uint32_t(l < nk ? l : 0);   // levels beyond the run repeat its first
    const double vf = __ldg(in.ws.vflux + (qe + lc));
    const bool first = vf > 0.0;   // the first node is upwind
    const uint32_t ou = F::off((first ? q1 : q2) + lc, tg), od = F::off((first ? q2 : q1) + lc, tg);
    const uint32_t oa = F::off((first ? qua : qda) + lc, tg),
                   ob = F::off((first ? qub : qdb) + lc, tg);
    const double c0 = first ? u01.x : d01.x, c1 = first ? u01.y : d01.y,
                 c2 = first ? u2x.x : d2x.x;
    double Tu[NTR], Td[NTR], Ou[NTR], Od[NTR], va[NTR], vb[NTR];
    fT.ld(ou, Tu);
    fT.ld(od, Td);
    fO.ld(ou, Ou);
    fO.ld(od, Od);
    fT.ld(oa, va);
    fT.ld(ob, vb);
    double adf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double Au = ab2f(Tu[t], Ou[t]), Ad = ab2f(Td[t], Od[t]);
      const double g = fma(c1, va[t], fma(c2, vb[t], c0 * Tu[t]));
      const double Tm = fma(Ad - Au, 1.0 / 3.0, Au) + g;
      adf[t] = -vf * (Tm - Tu[t]);
    }
    if (l < nk) stv<NTR, IL>(in.ws.adfh, qe + uint32_t(l), w0, in.ws.sEd, in.wtg, adf);
  }
}

// The same, one level at a time (T and S on the CORE2-size mesh: 139 -> 107 us; 8 tracers of
// two members, 4 per thread: 0.82 -> 0.66 ms), for a thread that walks the segments si, si + stride, ...: the
// next level's records and volume flux are loaded while this level's gathers are under way, so
// a level costs one memory round trip instead of three in a row (segment, records, gathers).
template <int NTR, bool IL>
__device__ __forceinline__ void stream_edge_adf(const Inst& in, int64_t si, int64_t stride, int t0,
                                                int w0) {
  const DevMesh& m = in.m;
  const int64_t count = m.n_eseg[0];
  if (si >= count) return;
  const int L = m.L, tg = in.tg;
  using F = Fld<NTR, IL>;
  const F fT(in.T, t0, in.tstride), fO(in.T_old, t0, in.tstride);
  const uint32_t* __restrict__ list = m.eseg[0];
  const int4* __restrict__ erec = m.erec;
  const int4* __restrict__ emf4 = m.emf4;
  const double* __restrict__ emfw = m.emfw;
  const double* __restrict__ vflux = in.ws.vflux;
  uint32_t sg = __ldg(list + si);
  uint32_t sg1 = si + stride < count ? __ldg(list + si + stride) : sg;
  int4 er = __ldg(erec + lane_ent(sg)), ov = __ldg(emf4 + lane_ent(sg));
  double vf = __ldg(vflux + lq(lane_ent(sg), L, lane_lev(sg)));
  for (; si < count; si += stride) {
    const int e = lane_ent(sg), k = lane_lev(sg);
    const bool first = vf > 0.0;   // the first node is upwind
    const uint32_t ou = F::off(lq(first ? er.x : er.y, L, k), tg);
    const uint32_t od = F::off(lq(first ? er.y : er.x, L, k), tg);
    const uint32_t oa = F::off(lq(first ? ov.x : ov.z, L, k), tg);
    const uint32_t ob = F::off(lq(first ? ov.y : ov.w, L, k), tg);
    const double* wp = emfw + (8 * int64_t(e) + (first ? 0 : 4));
    double Tu[NTR], Td[NTR], Ou[NTR], Od[NTR], va[NTR], vb[NTR];
    fT.ld(ou, Tu);
    fT.ld(od, Td);
    fO.ld(ou, Ou);
    fO.ld(od, Od);
    fT.ld(oa, va);
    fT.ld(ob, vb);
    const double2 c01 = __ldg(reinterpret_cast<const double2*>(wp));
    const double c2 = __ldg(wp + 2), v = vf;
    // the next level's records, and the segment after it
    sg = sg1;
    er = __ldg(erec + lane_ent(sg));
    ov = __ldg(emf4 + lane_ent(sg));
    vf = __ldg(vflux + lq(lane_ent(sg), L, lane_lev(sg)));
    sg1 = si + 2 * stride < count ? __ldg(list + si + 2 * stride) : sg;
    double adf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double Au = ab2f(Tu[t], Ou[t]), Ad = ab2f(Td[t], Od[t]);
      const double g = fma(c01.y, va[t], fma(c2, vb[t], c01.x * Tu[t]));
      const double Tm = fma(Ad - Au, 1.0 / 3.0, Au) + g;
      adf[t] = -v * (Tm - Tu[t]);
    }
    stv<NTR, IL>(in.ws.adfh, lq(e, L, k), w0, in.ws.sEd, in.wtg, adf);
  }
}

// ----------------------------------------------- adf_h on the remaining edge lanes
// kFixThreads adjacent threads take one edge lane, one per end node: each forms its node's
// average gradient (_node_avg_grad, tracer_adv.py:329-341: the mean over the node's cells wet
// at the level, in the node's cell order; a chain of dependent loads, the cells' records one
// ahead), and the first one combines them. (With one thread per lane the kernel held 128
// registers; with eight per lane, one cell in four each, it took twice the time.) Where MFCT
// takes the up/down cells although they do not hold the edge's nodes, each end has one cell.
// ``i`` may lie beyond the list (the whole warp takes part in the shuffle).
constexpr int kFixThreads = 2;
template <int NTR, bool IL>
__device__ __forceinline__ void body_edge_fix(const Inst& in, int64_t i, int g, int t0, int w0) {
  const DevMesh& m = in.m;
  const bool valid = i < m.n_efix;
  const uint32_t lane = __ldg(m.efix + (valid ? i : 0));
  const int e = lane_ent(lane), k = lane_lev(lane), L = m.L;
  const int4 er = __ldg(m.erec + e);
  const bool use_tri = in_range(k, unsigned(__ldg(m.etr + e)));
  const int4 rec = __ldg(m.nrec + (g ? er.y : er.x));
  const int count = use_tri ? 1 : int(unsigned(rec.z) >> 24);
  double nx[NTR], ny[NTR], den = 0.0;
#pragma unroll
  for (int t = 0; t < NTR; ++t) nx[t] = ny[t] = 0.0;
  int4 sl = make_int4(0, 0, 0, 0);
  unsigned r = 0xffu << 8;   // every level
  if (use_tri) {
    sl = __ldg(m.eud4 + 2 * e + g);
  } else if (count > 0) {
    sl = __ldg(m.nel4 + rec.y);
    r = unsigned(__ldg(m.nelr + rec.y));
  }
  for (int j = 0; j < count; ++j) {
    const int4 c = sl;
    const bool on = in_range(k, r);
    if (j + 1 < count) {
      sl = __ldg(m.nel4 + rec.y + j + 1);
      r = unsigned(__ldg(m.nelr + rec.y + j + 1));
    }
    if (!on) continue;
    const double a = use_tri ? 1.0 : __ldg(m.earea + c.x);
    double gx[NTR], gy[NTR];
    cell_grad<NTR, IL>(in, c.x, c.y, c.z, c.w, k, t0, gx, gy);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      nx[t] += gx[t] * a;
      ny[t] += gy[t] * a;
    }
    den += a;
  }
  const Rcp rdd = rcp(den > 0.0 ? den : 1.0);
  const double c1 = __ldg(m.ecoef + 2 * e), c2 = __ldg(m.ecoef + 2 * e + 1);
  double X[NTR], Xo[NTR];   // c1 gx + c2 gy of this thread's end and of the other's
#pragma unroll
  for (int t = 0; t < NTR; ++t) {
    X[t] = c1 * divr(nx[t], rdd) + c2 * divr(ny[t], rdd);
    Xo[t] = __shfl_xor_sync(0xffffffffu, X[t], 1);
  }
  if (!valid || g != 0) return;
  const double vf = __ldg(in.ws.vflux + lq(e, L, k));
  const double avf = fabs(vf);
  const uint32_t q1 = lq(er.x, L, k), q2 = lq(er.y, L, k);
  const int64_t ts = in.tstride;
  const int tg = in.tg;
  double T1[NTR], T2[NTR], O1[NTR], O2[NTR], adf[NTR];
  ldn<NTR, IL>(in.T, q1, t0, ts, tg, T1);
  ldn<NTR, IL>(in.T, q2, t0, ts, tg, T2);
  ldn<NTR, IL>(in.T_old, q1, t0, ts, tg, O1);
  ldn<NTR, IL>(in.T_old, q2, t0, ts, tg, O2);
  const Rcp r6{6.0, 1.0 / 6.0, true};
#pragma unroll
  for (int t = 0; t < NTR; ++t) {
    const double fl = -0.5 * (T1[t] * (vf + avf) + T2[t] * (vf - avf));
    const double A1 = ab2(T1[t], O1[t]), A2 = ab2(T2[t], O2[t]);
    const double diff = A2 - A1;
    const double Tm1 = A1 + divr(2.0 * diff + X[t], r6);
    const double Tm2 = A2 - divr(2.0 * diff + Xo[t], r6);
    const double ho = -0.5 * ((vf + avf) * Tm1 + (vf - avf) * Tm2);
    adf[t] = ho - fl;
  }
  stn<NTR, IL>(in.ws.adfh, lq(e, L, k), w0, in.ws.sEd, in.wtg, adf);
}

// ---------------------------------------- limiter factors on a node's layer run
// The cluster bound of node n at level k is the max (min) of max(LO, T) (min(LO, T)) over
// the nodes of n's cells that are wet at k, padded with -BIG (+BIG) when one of n's cells
// is dry at k (tracer_adv.py:389-405). Every cell of n has two edges at n, so those nodes
// are n itself (when any cell is wet at k) and the edge neighbours with a wet cell at k;
// max/min are exact, so this equals the per-cell evaluation bit for bit. The neighbour comes
// first in each comparison: a non-finite one (a comparison with NaN is false) leaves the bound
// as it is instead of replacing it.
// The a4 window (k-1, k, k+1 of the same column) crosses a run's ends: each thread leaves
// the bounds of its run's first and last level in shared memory, and the neighbouring
// runs of the column (the adjacent segment slots of the block: a column's runs are
// consecutive) read them. A block's first and last slot are halo runs that only publish
// their bounds; ``sh`` holds [4][NTR][256] doubles (first-level max, min, last-level max,
// min) and ``S`` is the distance between adjacent slots in threads.
template <int NTR, int LPT, bool IL>
__device__ __forceinline__ void seg_node_limit(const Inst& in, int64_t si, bool core, int t0,
                                               int w0, int tid, int S, double* sh) {
  const DevMesh& m = in.m;
  constexpr int V = seg_variant(LPT);
  using F = Fld<NTR, IL>;
  const bool valid = si >= 0 && si < m.n_nseg[V];
  const int L = m.L;
  const int64_t sN = in.ws.sN;
  int n = 0, k0 = 0, nzmin = 0, nzmax = 1, nk = 1;
  uint32_t base = 0;
  double mx[LPT][NTR], mn[LPT][NTR], sp[LPT][NTR], sm[LPT][NTR], lo[LPT][NTR];
#pragma unroll
  for (int l = 0; l < LPT; ++l)
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      mx[l][t] = -INFINITY; mn[l][t] = INFINITY; sp[l][t] = 0.0; sm[l][t] = 0.0;
      lo[l][t] = 0.0;
    }
  if (valid) {
    const uint32_t sg = __ldg(m.nseg[V] + si);
    n = lane_ent(sg);
    k0 = lane_lev(sg);
    const int4 rec = __ldg(m.nrec + n);
    const unsigned pk = unsigned(rec.z);
    nzmin = int(pk & 255u);
    nzmax = int((pk >> 8) & 255u);
    nk = min(LPT, nzmax - k0);
    base = lq(n, L, 0);
    const F fT(in.T, t0, in.tstride), fL(in.ws.lo, w0, sN), fA(in.ws.adfh, w0, in.ws.sEd);
    const int tg = in.tg, wtg = in.wtg;
    unsigned onb[LPT], wetb[LPT], cell[LPT];   // the run's node-layer flags (0 beyond the run)
    uint32_t own[LPT];
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      const unsigned long long f =
          l < nk ? __ldg(m.nflags + rec.w + (k0 + l - nzmin)) : 0ull;
      onb[l] = unsigned(f);
      wetb[l] = unsigned(f >> kSlotWet);
      cell[l] = unsigned(f >> kOwnBit);
      own[l] = base + uint32_t(k0 + (l < nk ? l : 0));
    }
    // the node itself
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      double tv[NTR];
      fL.ld(F::off(own[l], wtg), lo[l]);
      fT.ld(F::off(own[l], tg), tv);
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        mx[l][t] = dmax(lo[l][t], tv[t]);
        mn[l][t] = dmin(lo[l][t], tv[t]);
      }
    }
    const int e0 = rec.x, e1 = rec.x + int((pk >> 16) & 255u);
    FCT_SLOT_BEGIN(e0, e1)
    for (int j = e0; j < e1; ++j) {
      FCT_SLOT_GET(j, e1)
#pragma unroll
      for (int l = 0; l < LPT; ++l) {
        // an edge without a wet cell here reads the node's own values again (max and min do
        // not change); one without this level adds no flux
        const uint32_t qo = (wetb[l] & 1u) ? uint32_t(sl.y) + uint32_t(k0 + l) : own[l];
        const bool on = onb[l] & 1u;
        wetb[l] >>= 1;
        onb[l] >>= 1;
        double lv[NTR], tv[NTR], a[NTR];
        fL.ld(F::off(qo, wtg), lv);
        fT.ld(F::off(qo, tg), tv);
#pragma unroll
        for (int t = 0; t < NTR; ++t) a[t] = 0.0;
        if (on) fA.ld(F::off(uint32_t(sl.x) + uint32_t(k0 + l), wtg), a);
#pragma unroll
        for (int t = 0; t < NTR; ++t) {
          mx[l][t] = dmax(dmax(lv[t], tv[t]), mx[l][t]);
          mn[l][t] = dmin(dmin(lv[t], tv[t]), mn[l][t]);
          const double sv = flip_sign(a[t], sl.z);   // adf_h leaves the edge's first node
          if (sv > 0.0) sp[l][t] += sv;
          if (sv < 0.0) sm[l][t] += sv;
        }
      }
    }
    // no wet cell at the level: no bounds; the padding of dry cells
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      const bool ow = cell[l] & 1u, of = cell[l] & 2u;
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        if (!ow) {
          mx[l][t] = -INFINITY;
          mn[l][t] = INFINITY;
        }
        if (of) {
          mx[l][t] = dmax(mx[l][t], -kBig);
          mn[l][t] = dmin(mn[l][t], kBig);
        }
      }
    }
    // publish the first and last level's bounds for the neighbouring runs
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      sh[(0 * NTR + t) * 256 + tid] = mx[0][t];
      sh[(1 * NTR + t) * 256 + tid] = mn[0][t];
    }
#pragma unroll
    for (int l = 0; l < LPT; ++l)
      if (l == nk - 1)
#pragma unroll
        for (int t = 0; t < NTR; ++t) {
          sh[(2 * NTR + t) * 256 + tid] = mx[l][t];
          sh[(3 * NTR + t) * 256 + tid] = mn[l][t];
        }
  }
  __syncthreads();
  if (!valid || !core) return;
  const double dt = in.dt;
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    if (l >= nk) break;
    const int k = k0 + l;
    const uint32_t qn = base + uint32_t(k);
    const bool interior = k != nzmin && k != nzmax - 1;   // a4: window over k-1, k, k+1
    const double av = __ldg(m.areasvol + qn), hnn = __ldg(in.hnode_new + qn);
    const bool valid_n = (av > 0.0) && (hnn > 0.0);
    const double sa = av > 0.0 ? av : 1.0, sh_ = hnn > 0.0 ? hnn : 1.0;
    const double fdt = dt * __drcp_rn(sa * sh_);   // dt / (areasvol * hnode_new)
    double ft[NTR], fb[NTR];
    ldv<NTR, IL>(in.ws.adfv, qn, w0, sN, in.wtg, ft);
    if (k + 1 < nzmax) {
      ldv<NTR, IL>(in.ws.adfv, qn + 1, w0, sN, in.wtg, fb);
    } else {   // the bottom interface carries no flux
#pragma unroll
      for (int t = 0; t < NTR; ++t) fb[t] = 0.0;
    }
    double pf[NTR], mf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      double wmx = mx[l][t], wmn = mn[l][t];
      if (interior) {
        const double ax = l > 0 ? mx[l - 1][t] : sh[(2 * NTR + t) * 256 + tid - S];
        const double an = l > 0 ? mn[l - 1][t] : sh[(3 * NTR + t) * 256 + tid - S];
        const double bx = l + 1 < nk ? mx[l + 1 < LPT ? l + 1 : l][t]
                                     : sh[(0 * NTR + t) * 256 + tid + S];
        const double bn = l + 1 < nk ? mn[l + 1 < LPT ? l + 1 : l][t]
                                     : sh[(1 * NTR + t) * 256 + tid + S];
        wmx = dmax(dmax(ax, wmx), bx);
        wmn = dmin(dmin(an, wmn), bn);
      }
      const double plus = (dmax(ft[t], 0.0) + dmax(-fb[t], 0.0)) + sp[l][t];
      const double minus = (dmin(ft[t], 0.0) + dmin(-fb[t], 0.0)) + sm[l][t];
      pf[t] = 1.0;
      mf[t] = 1.0;
      if (valid_n) {
        const double flux_pos = fma(plus, fdt, kFluxEps);
        const double flux_neg = fma(minus, fdt, -kFluxEps);
        pf[t] = dmin(1.0, (wmx - lo[l][t]) * __drcp_rn(flux_pos));
        mf[t] = dmin(1.0, (wmn - lo[l][t]) * __drcp_rn(flux_neg));
      }
    }
    stv<NTR, IL>(in.ws.pf, qn, w0, sN, in.wtg, pf);
    stv<NTR, IL>(in.ws.mf, qn, w0, sN, in.wtg, mf);
  }
}

// ------------------- zalesak b3 + flux2dtracer_fct + ale_reconstruct on a layer run
template <int NTR, int LPT, bool IL>
__device__ __forceinline__ void seg_node_final(const Inst& in, int64_t si, int t0, int w0) {
  const DevMesh& m = in.m;
  constexpr int V = seg_variant(LPT);
  constexpr int NB = LPT + 2;   // factor levels k0-1 .. k0+LPT
  if (si >= m.n_nseg[V]) return;
  const uint32_t sg = __ldg(m.nseg[V] + si);
  const int n = lane_ent(sg), k0 = lane_lev(sg), L = m.L;
  const int4 rec = __ldg(m.nrec + n);
  const unsigned pk = unsigned(rec.z);
  const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
  const int nk = min(LPT, nzmax - k0);
  const uint32_t base = lq(n, L, 0);
  const int64_t sN = in.ws.sN;
  const int tg = in.tg;
  using F = Fld<NTR, IL>;
  const F fP(in.ws.pf, w0, sN), fM(in.ws.mf, w0, sN), fA(in.ws.adfh, w0, in.ws.sEd);
  const int wtg = in.wtg;
  // limited horizontal fluxes, ascending edge id
  double hsc[LPT][NTR];
#pragma unroll
  for (int l = 0; l < LPT; ++l)
#pragma unroll
    for (int t = 0; t < NTR; ++t) hsc[l][t] = 0.0;
  double pfw[NB][NTR], mfw[NB][NTR];   // own factors at levels k0-1 .. k0+LPT
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const uint32_t o = F::off(base + uint32_t(kclamp(k0 - 1 + b, L)), wtg);
    fP.ld(o, pfw[b]);
    fM.ld(o, mfw[b]);
  }
  unsigned onb[LPT];   // per layer of the run: bit j, the j-th slot's edge has the layer
#pragma unroll
  for (int l = 0; l < LPT; ++l)
    onb[l] = l < nk ? unsigned(__ldg(m.nflags + rec.w + (k0 + l - nzmin))) : 0u;
  const int e0 = rec.x, e1 = rec.x + int((pk >> 16) & 255u);
  FCT_SLOT_BEGIN(e0, e1)
  for (int j = e0; j < e1; ++j) {
    FCT_SLOT_GET(j, e1)
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      const bool on = onb[l] & 1u;
      onb[l] >>= 1;
      double a[NTR], pfo[NTR], mfo[NTR];
#pragma unroll
      for (int t = 0; t < NTR; ++t) a[t] = pfo[t] = mfo[t] = 0.0;
      if (on) {
        const uint32_t qo = F::off(uint32_t(sl.y) + uint32_t(k0 + l), wtg);
        fA.ld(F::off(uint32_t(sl.x) + uint32_t(k0 + l), wtg), a);
        fP.ld(qo, pfo);
        fM.ld(qo, mfo);
      }
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        // b3 (tracer_adv.py:461-465): adf >= 0 ? min(plus(n1), minus(n2)) : min(minus(n1),
        // plus(n2)); min is symmetric, so in the node's own terms the factor is min(own
        // plus, other minus) when the flux leaves the node, else the other pair
        const double s = flip_sign(a[t], sl.z);   // adf_h leaves the edge's first node
        const bool leaves = s >= 0.0;
        const double fo = leaves ? pfw[l + 1][t] : mfw[l + 1][t];
        const double fx = leaves ? mfo[t] : pfo[t];
        hsc[l][t] = fma(dmin(fo, fx), s, hsc[l][t]);
      }
    }
  }
  const double dt = in.dt;
#pragma unroll
  for (int l = 0; l < LPT; ++l) {
    if (l >= nk) break;
    const int k = k0 + l;
    const uint32_t qn = base + uint32_t(k);
    const double iav = __ldg(m.iavol + qn);   // 1 / areasvol (0 where there is no volume)
    const double hn = __ldg(in.hnode + qn), hnn = __ldg(in.hnode_new + qn);
    const double fdt = dt * (iav > 0.0 ? iav : 1.0);
    const Rcq rhn = rcpq(hnn);
    double ft[NTR], vt[NTR], vb[NTR];
    ldv<NTR, IL>(in.ws.adfv, qn, w0, sN, in.wtg, ft);
    // limited vertical flux at the top interface k (tracer_adv.py:453-459)
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double pf0 = pfw[l + 1][t], mf0 = mfw[l + 1][t];
      vt[t] = k == nzmin ? (ft[t] >= 0.0 ? pf0 : mf0) * ft[t]
                         : (ft[t] >= 0.0 ? dmin(mfw[l][t], pf0) : dmin(pfw[l][t], mf0)) * ft[t];
    }
    // limited vertical flux at the bottom interface k+1 (0 at the node's bottom)
    if (k + 1 >= nzmax) {
#pragma unroll
      for (int t = 0; t < NTR; ++t) vb[t] = 0.0;
    } else {
      double fb[NTR];
      ldv<NTR, IL>(in.ws.adfv, qn + 1, w0, sN, in.wtg, fb);
#pragma unroll
      for (int t = 0; t < NTR; ++t)
        vb[t] = (fb[t] >= 0.0 ? dmin(mfw[l + 1][t], pfw[l + 2][t])
                              : dmin(pfw[l + 1][t], mfw[l + 2][t])) * fb[t];
    }
    double Tv[NTR], lo[NTR], out[NTR];
    ldv<NTR, IL>(in.T, qn, t0, in.tstride, tg, Tv);
    ldv<NTR, IL>(in.ws.lo, qn, w0, sN, in.wtg, lo);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double lo_trans = fma(lo[t], hnn, -Tv[t] * hn);
      const double vdiv = iav > 0.0 ? (vt[t] - vb[t]) * fdt : 0.0;
      double d = fma(hsc[l][t], fdt, lo_trans + vdiv);
      d = fma(Tv[t], hn - hnn, d);
      out[t] = Tv[t] + (hnn > 0.0 ? divq(d, rhn) : 0.0);
    }
    stv<NTR, IL>(in.T_new, qn, t0, in.tstride, tg, out);
    count_nonfinite<NTR>(in.nonfinite, out);
  }
}

// ------------------------------------------- node stages, threads that walk the layers
// What bounds these stages is the wait for their gathers (L2 answers in 300 to 650 cycles on
// an idle chip, DRAM in 840), and what a thread waits for first used to be the chain segment ->
// record -> slots. So a thread walks the layers si, si + stride, ... (nseg[0], one layer per segment, in the order
// of the flag words). The next layer's record, flag word and first slots are loaded while this
// layer's gathers are under way, and a batch of U slots issues all its gathers before it uses
// any, so the memory round trips of a layer are those of its gathers alone. Blocks per SM and U
// per stage (fct_seg_*.cu) were swept together, 1 to 6 blocks and U of 1 to 3: fewer blocks
// with more registers and longer batches win except where they start to spill.
template <int U>
struct NodeWalk {
  const uint32_t* __restrict__ list;
  const int4* __restrict__ nrec;
  const int4* __restrict__ ns4;
  const unsigned long long* __restrict__ flags;
  int64_t count;
  uint32_t sg, sg1;
  int4 rec, rec1, sl[U];
  unsigned long long fl, fl1;
  __device__ __forceinline__ NodeWalk(const DevMesh& m, int64_t si, int64_t stride)
      : list(m.nseg[0]), nrec(m.nrec), ns4(m.ns4), flags(m.nflags), count(m.n_nseg[0]) {
    const int64_t i = si < 0 ? 0 : (si < count ? si : count - 1);
    const int64_t j = si + stride < count ? si + stride : i;
    sg = __ldg(list + i);
    sg1 = __ldg(list + j);
    fl = __ldg(flags + i);
    rec = __ldg(nrec + lane_ent(sg));
    first_slots(rec);
  }
  __device__ __forceinline__ int degree() const { return int((unsigned(rec.z) >> 16) & 255u); }
  __device__ __forceinline__ void first_slots(const int4& r) {
    const int e1 = r.x + int((unsigned(r.z) >> 16) & 255u);
#pragma unroll
    for (int u = 0; u < U; ++u) sl[u] = __ldg(ns4 + max(min(r.x + u, e1 - 1), 0));
  }
  // the records of the batch after the one at j (the last batch keeps what it has)
  __device__ __forceinline__ void more_slots(int j) {
    const int e1 = rec.x + degree();
    if (j + U < e1) {
#pragma unroll
      for (int u = 0; u < U; ++u) sl[u] = __ldg(ns4 + min(j + U + u, e1 - 1));
    }
  }
  // the next layer's record and flags, and the segment after it
  __device__ __forceinline__ void ahead(int64_t si, int64_t stride) {
    const int64_t j = si + stride < count ? si + stride : (si < 0 ? 0 : min(si, count - 1));
    rec1 = __ldg(nrec + lane_ent(sg1));
    fl1 = __ldg(flags + j);
  }
  // the first slots of the next layer (its record has arrived)
  __device__ __forceinline__ void ahead_slots() { first_slots(rec1); }
  __device__ __forceinline__ void next(int64_t si, int64_t stride) {
    rec = rec1;
    fl = fl1;
    sg = sg1;
    const int64_t j = si + 2 * stride;
    sg1 = j < count ? __ldg(list + j) : sg1;
  }
};

template <int NTR, bool IL, int U>
__device__ __forceinline__ void stream_node_final(const Inst& in, int64_t si, int64_t stride,
                                                  int t0, int w0) {
  const DevMesh& m = in.m;
  if (si >= m.n_nseg[0]) return;
  using F = Fld<NTR, IL>;
  const int64_t sN = in.ws.sN;
  const F fP(in.ws.pf, w0, sN), fM(in.ws.mf, w0, sN), fA(in.ws.adfh, w0, in.ws.sEd);
  const F fV(in.ws.adfv, w0, sN), fL(in.ws.lo, w0, sN), fT(in.T, t0, in.tstride);
  const int L = m.L, tg = in.tg, wtg = in.wtg;
  const double dt = in.dt;
  NodeWalk<U> nw(m, si, stride);
  for (; si < nw.count; si += stride) {
    const int n = lane_ent(nw.sg), k = lane_lev(nw.sg);
    const unsigned pk = unsigned(nw.rec.z);
    const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
    const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k), on_ = F::off(qn, wtg);
    double pf0[NTR], mf0[NTR], hsc[NTR];
    fP.ld(on_, pf0);
    fM.ld(on_, mf0);
#pragma unroll
    for (int t = 0; t < NTR; ++t) hsc[t] = 0.0;
    unsigned onb = unsigned(nw.fl) & kSlotBits;
    const int e1 = nw.rec.x + nw.degree();
    for (int j = nw.rec.x; j < e1; j += U) {
      double a[U][NTR], pfo[U][NTR], mfo[U][NTR];
      int sgn[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t qo = F::off(uint32_t(nw.sl[u].y) + uint32_t(k), wtg);
        sgn[u] = nw.sl[u].z;
        fA.ld(F::off(uint32_t(nw.sl[u].x) + uint32_t(k), wtg), a[u]);
        fP.ld(qo, pfo[u]);
        fM.ld(qo, mfo[u]);
      }
      if (j == nw.rec.x) nw.ahead(si, stride);
      nw.more_slots(j);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = (onb >> u) & 1u;
#pragma unroll
        for (int t = 0; t < NTR; ++t) {
          const double s = flip_sign(a[u][t], sgn[u]);   // adf_h leaves the edge's first node
          const bool leaves = s >= 0.0;
          const double h = fma(dmin(leaves ? pf0[t] : mf0[t], leaves ? mfo[u][t] : pfo[u][t]), s,
                               hsc[t]);
          hsc[t] = on ? h : hsc[t];
        }
      }
      onb >>= U;
    }
    if (e1 == nw.rec.x) nw.ahead(si, stride);
    nw.ahead_slots();
    const double iav = __ldg(m.iavol + qn);   // 1 / areasvol (0 where there is no volume)
    const double hn = __ldg(in.hnode + qn), hnn = __ldg(in.hnode_new + qn);
    double ft[NTR], fb[NTR], Tv[NTR], lo[NTR], pu[NTR], mu[NTR], pd[NTR], md[NTR];
    const bool below = k + 1 < nzmax, above = k > nzmin;
    const uint32_t oa = F::off(above ? qn - 1 : qn, wtg), ob = F::off(below ? qn + 1 : qn, wtg);
    fV.ld(on_, ft);
    fV.ld(ob, fb);
    fT.ld(F::off(qn, tg), Tv);
    fL.ld(on_, lo);
    fP.ld(oa, pu);
    fM.ld(oa, mu);
    fP.ld(ob, pd);
    fM.ld(ob, md);
    nw.next(si, stride);
    const double fdt = dt * (iav > 0.0 ? iav : 1.0);
    const Rcq rhn = rcpq(hnn);
    double out[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      // limited vertical fluxes at the top (k) and bottom (k + 1) interfaces
      const double vt = above ? (ft[t] >= 0.0 ? dmin(mu[t], pf0[t]) : dmin(pu[t], mf0[t])) * ft[t]
                              : (ft[t] >= 0.0 ? pf0[t] : mf0[t]) * ft[t];
      const double vb =
          below ? (fb[t] >= 0.0 ? dmin(mf0[t], pd[t]) : dmin(pf0[t], md[t])) * fb[t] : 0.0;
      const double lo_trans = fma(lo[t], hnn, -Tv[t] * hn);
      const double vdiv = iav > 0.0 ? (vt - vb) * fdt : 0.0;
      double d = fma(hsc[t], fdt, lo_trans + vdiv);
      d = fma(Tv[t], hn - hnn, d);
      out[t] = Tv[t] + (hnn > 0.0 ? divq(d, rhn) : 0.0);
    }
    stv<NTR, IL>(in.T_new, qn, t0, in.tstride, tg, out);
    count_nonfinite<NTR>(in.nonfinite, out);
  }
}

template <int NTR, bool IL, int U>
__device__ __forceinline__ void stream_node_lo(const Inst& in, int64_t si, int64_t stride, int t0,
                                               int w0) {
  const DevMesh& m = in.m;
  if (si >= m.n_nseg[0]) return;
  using F = Fld<NTR, IL>;
  const F fT(in.T, t0, in.tstride), fTo(in.T_old, t0, in.tstride);
  const int L = m.L, tg = in.tg;
  const double dt = in.dt;
  NodeWalk<U> nw(m, si, stride);
  for (; si < nw.count; si += stride) {
    const int n = lane_ent(nw.sg), k = lane_lev(nw.sg);
    const unsigned pk = unsigned(nw.rec.z);
    const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
    const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k);
    double div[NTR], out = 0.0;
#pragma unroll
    for (int t = 0; t < NTR; ++t) div[t] = 0.0;
    unsigned onb = unsigned(nw.fl) & kSlotBits;
    const int e1 = nw.rec.x + nw.degree();
    for (int j = nw.rec.x; j < e1; j += U) {
      double vf[U], To[U][NTR];
      int sgn[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = (onb >> u) & 1u;
        sgn[u] = nw.sl[u].z;
        vf[u] = __ldg(in.ws.vflux + (uint32_t(nw.sl[u].x) + uint32_t(k)));
        fT.ld(F::off((on ? uint32_t(nw.sl[u].y) : base) + uint32_t(k), tg), To[u]);
      }
      if (j == nw.rec.x) nw.ahead(si, stride);
      nw.more_slots(j);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double s = flip_sign(vf[u], sgn[u]);
        const bool on = (onb >> u) & 1u, leaves = s > 0.0;
        const double cin = (on && !leaves) ? -s : 0.0;
        if (on && leaves) out += s;
#pragma unroll
        for (int t = 0; t < NTR; ++t) div[t] = fma(cin, To[u][t], div[t]);
      }
      onb >>= U;
    }
    if (e1 == nw.rec.x) nw.ahead(si, stride);
    nw.ahead_slots();
    // the column at k-2 .. k+1 (the level above the surface reads the top again), w and areas
    const uint32_t q0 = base + uint32_t(kclamp(k - 2, L)), q1 = base + uint32_t(kclamp(k - 1, L));
    const uint32_t q3 = base + uint32_t(kclamp(k + 1, L));
    double T0[NTR], T1[NTR], T2[NTR], T3[NTR], O0[NTR], O1[NTR], O2[NTR], O3[NTR];
    fT.ld(F::off(q0, tg), T0);
    fT.ld(F::off(q1, tg), T1);
    fT.ld(F::off(qn, tg), T2);
    fT.ld(F::off(q3, tg), T3);
    fTo.ld(F::off(q0, tg), O0);
    fTo.ld(F::off(q1, tg), O1);
    fTo.ld(F::off(qn, tg), O2);
    fTo.ld(F::off(q3, tg), O3);
    const double w = __ldg(in.w_e + qn), area = __ldg(m.area + qn);
    const double wb = __ldg(in.w_e + q3), areab = __ldg(m.area + q3);
    const double hn = __ldg(in.hnode + qn), hnn = __ldg(in.hnode_new + qn);
    const double iav = __ldg(m.iavol + qn);
    nw.next(si, stride);
    const bool below = k + 1 < nzmax;
    const double fdt = dt * iav;   // dt / areasvol
    const Rcq rhn = rcpq(hnn);
    const bool valid = (hnn > 0.0) && (iav > 0.0);
    double lo[NTR], fv[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      fv[t] = vflux_up(T2[t], T1[t], w, area);
      const double fvb = below ? vflux_up(T3[t], T2[t], wb, areab) : 0.0;
      const double dh = fma(-out, T2[t], div[t]);
      lo[t] = valid ? divq(fma(T2[t], hn, (dh + (fv[t] - fvb)) * fdt), rhn) : 0.0;
    }
    stv<NTR, IL>(in.ws.lo, qn, w0, in.ws.sN, in.wtg, lo);
    // adv_flux_ver_ho (QR4C on ttfAB) minus the LO vertical flux at the layer top
    const double Wf = in.w_i ? w + __ldg(in.w_i + qn) : w;
    double hi[NTR];
    if (k == nzmin) {
#pragma unroll
      for (int t = 0; t < NTR; ++t) hi[t] = -ab2f(T2[t], O2[t]) * Wf * area;
    } else if (k == nzmin + 1 || k == nzmax - 1) {
#pragma unroll
      for (int t = 0; t < NTR; ++t)
        hi[t] = -0.5 * (ab2f(T1[t], O1[t]) + ab2f(T2[t], O2[t])) * Wf * area;
    } else {
      double rdc, rdu, rdd, d1, d2;
      if (in.Z3d) {
        const double* Zc = in.Z3d + base;
        const double Znz = __ldg(Zc + k), Zm1 = __ldg(Zc + k - 1), Zm2 = __ldg(Zc + k - 2);
        const double Zp1 = __ldg(Zc + (k + 1 < L ? k + 1 : L - 1)), zb = __ldg(in.zbar3 + qn);
        rdc = __drcp_rn(safe_nz(Zm1 - Znz));
        rdu = __drcp_rn(safe_nz(Znz - Zp1));
        rdd = __drcp_rn(safe_nz(Zm2 - Zm1));
        d1 = (zb - Znz) * (1.0 / 3.0);
        d2 = (zb - Zm1) * (1.0 / 3.0);
      } else {
        const double* q = m.qr4c + k;
        rdc = __ldg(q);
        rdu = __ldg(q + L);
        rdd = __ldg(q + 2 * L);
        d1 = __ldg(q + 3 * L);
        d2 = __ldg(q + 4 * L);
      }
      const double wa = -0.5 * Wf * area;
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        const double A0 = ab2f(T2[t], O2[t]), Am1 = ab2f(T1[t], O1[t]);
        const double Am2 = ab2f(T0[t], O0[t]), Ap1 = ab2f(T3[t], O3[t]);
        const double qc = (Am1 - A0) * rdc, qu = (A0 - Ap1) * rdu, qd = (Am2 - Am1) * rdd;
        const double Tmean1 = fma(fma(2.0, qc, qu), d1, A0);
        const double Tmean2 = fma(fma(2.0, qc, qd), d2, Am1);
        hi[t] = (Tmean1 + Tmean2) * wa;
      }
    }
    double adf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      adf[t] = hi[t] - (in.w_i ? vflux_up(T2[t], T1[t], Wf, area) : fv[t]);
    stv<NTR, IL>(in.ws.adfv, qn, w0, in.ws.sN, in.wtg, adf);
  }
}

// The limiter: a block's segment slots hold consecutive layers, the first and the last one
// halo layers that only publish their bounds; ``sh`` holds two sets (alternate rounds, so one
// barrier a round is enough) of [2][NTR][256] doubles.
template <int NTR, bool IL, int U>
__device__ __forceinline__ void stream_node_limit(const Inst& in, int64_t si, int64_t stride,
                                                  int64_t rounds, bool core, int t0, int w0,
                                                  int tid, int S, double* sh) {
  if (rounds <= 0) return;   // block-uniform
  const DevMesh& m = in.m;
  using F = Fld<NTR, IL>;
  const int64_t sN = in.ws.sN;
  const F fT(in.T, t0, in.tstride), fL(in.ws.lo, w0, sN), fA(in.ws.adfh, w0, in.ws.sEd);
  const F fV(in.ws.adfv, w0, sN);
  const int L = m.L, tg = in.tg, wtg = in.wtg;
  const double dt = in.dt;
  NodeWalk<U> nw(m, si, stride);
  for (int64_t r = 0; r < rounds; ++r, si += stride) {
    const bool valid = si >= 0 && si < nw.count;
    const int n = lane_ent(nw.sg), k = lane_lev(nw.sg);
    const unsigned pk = unsigned(nw.rec.z);
    const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
    const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k);
    double mx[NTR], mn[NTR], sp[NTR], sm[NTR], lo[NTR];
    {
      double tv[NTR];
      fL.ld(F::off(qn, wtg), lo);
      fT.ld(F::off(qn, tg), tv);
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        mx[t] = dmax(lo[t], tv[t]);
        mn[t] = dmin(lo[t], tv[t]);
        sp[t] = sm[t] = 0.0;
      }
    }
    unsigned onb = unsigned(nw.fl) & kSlotBits;
    unsigned wetb = unsigned(nw.fl >> kSlotWet) & kSlotBits;
    const bool ow = (nw.fl >> kOwnBit) & 1ull, of = (nw.fl >> kOffBit) & 1ull;
    const int e1 = nw.rec.x + nw.degree();
    for (int j = nw.rec.x; j < e1; j += U) {
      double lv[U][NTR], tv[U][NTR], a[U][NTR];
      int sgn[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        // an edge without a wet cell here reads the node's own values again
        const uint32_t qo = ((wetb >> u) & 1u) ? uint32_t(nw.sl[u].y) + uint32_t(k) : qn;
        sgn[u] = nw.sl[u].z;
        fL.ld(F::off(qo, wtg), lv[u]);
        fT.ld(F::off(qo, tg), tv[u]);
        fA.ld(F::off(uint32_t(nw.sl[u].x) + uint32_t(k), wtg), a[u]);
      }
      if (j == nw.rec.x) nw.ahead(si, stride);
      nw.more_slots(j);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = (onb >> u) & 1u;
#pragma unroll
        for (int t = 0; t < NTR; ++t) {
          mx[t] = dmax(dmax(lv[u][t], tv[u][t]), mx[t]);
          mn[t] = dmin(dmin(lv[u][t], tv[u][t]), mn[t]);
          const double sv = flip_sign(a[u][t], sgn[u]);   // adf_h leaves the first node
          if (on && sv > 0.0) sp[t] += sv;
          if (on && sv < 0.0) sm[t] += sv;
        }
      }
      onb >>= U;
      wetb >>= U;
    }
    if (e1 == nw.rec.x) nw.ahead(si, stride);
    nw.ahead_slots();
    double* shr = sh + (r & 1) * (2 * NTR * 256);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      if (!ow) {   // no wet cell at the level: no bounds
        mx[t] = -INFINITY;
        mn[t] = INFINITY;
      }
      if (of) {   // the padding of dry cells
        mx[t] = dmax(mx[t], -kBig);
        mn[t] = dmin(mn[t], kBig);
      }
      shr[t * 256 + tid] = mx[t];
      shr[(NTR + t) * 256 + tid] = mn[t];
    }
    const bool below = k + 1 < nzmax;
    double ft[NTR], fb[NTR];
    fV.ld(F::off(qn, wtg), ft);
    fV.ld(F::off(below ? qn + 1 : qn, wtg), fb);
    const double av = __ldg(m.areasvol + qn), hnn = __ldg(in.hnode_new + qn);
    nw.next(si, stride);
    __syncthreads();
    if (!valid || !core) continue;
    const bool interior = k != nzmin && k != nzmax - 1;   // a4: window over k-1, k, k+1
    const bool valid_n = (av > 0.0) && (hnn > 0.0);
    const double sa = av > 0.0 ? av : 1.0, shn = hnn > 0.0 ? hnn : 1.0;
    const double fdt = dt * __drcp_rn(sa * shn);   // dt / (areasvol * hnode_new)
    double pf[NTR], mf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      double wmx = mx[t], wmn = mn[t];
      if (interior) {
        wmx = dmax(dmax(shr[t * 256 + tid - S], wmx), shr[t * 256 + tid + S]);
        wmn = dmin(dmin(shr[(NTR + t) * 256 + tid - S], wmn), shr[(NTR + t) * 256 + tid + S]);
      }
      const double vb = below ? fb[t] : 0.0;   // the bottom interface carries no flux
      const double plus = (dmax(ft[t], 0.0) + dmax(-vb, 0.0)) + sp[t];
      const double minus = (dmin(ft[t], 0.0) + dmin(-vb, 0.0)) + sm[t];
      pf[t] = 1.0;
      mf[t] = 1.0;
      if (valid_n) {
        const double flux_pos = fma(plus, fdt, kFluxEps);
        const double flux_neg = fma(minus, fdt, -kFluxEps);
        pf[t] = dmin(1.0, (wmx - lo[t]) * __drcp_rn(flux_pos));
        mf[t] = dmin(1.0, (wmn - lo[t]) * __drcp_rn(flux_neg));
      }
    }
    stv<NTR, IL>(in.ws.pf, qn, w0, sN, in.wtg, pf);
    stv<NTR, IL>(in.ws.mf, qn, w0, sN, in.wtg, mf);
  }
}

// ------------------------------------------------------------- kernels and launchers
// Kernel wrappers: ``_1`` takes one instance by value (tracer-major layout, the
// single-call path; tracer slice = blockIdx.y), ``_n`` instance blockIdx.y of a device
// table (interleaved layout; the S adjacent threads of a segment take adjacent tracer
// slices, so together they read whole interleaved lines; S is any number up to 8, so an odd
// tracer count is one launch too). A 256-thread block holds 256/S segments.
//
// Resident 256-thread blocks per SM the compiler must fit (runs of two or more levels), by
// stage and by the updates u a thread carries. The kernels wait on their gathers, so resident
// warps pay until the cap makes the compiler spill; the limiter and the LO stage hold more per
// update and take one block less (T and S on the CORE2-size mesh, 2 tracers x 4 levels: limiter
// 384 us against 638; edge 221 against 195 the other way round).
__host__ __device__ constexpr int seg_min_blocks(int stage, int u) {
  return (stage == kStageEdge || stage == kStageFinal)
             ? (u <= 2 ? 5 : u <= 4 ? 4 : u <= 8 ? 3 : 2)
             : (u <= 2 ? 4 : u <= 4 ? 3 : 2);
}

// thread t of a block of 256/S segments: segment t / S, slice t % S (``mul`` = 65536/S + 1
// divides exactly below 256)
__device__ __forceinline__ int slice_div(int t, unsigned mul) { return int((unsigned(t) * mul) >> 16); }

#define FCT_SEG_KERNEL(name, body, stage)                                                \
  template <int NTR, int LPT>                                                            \
  __global__ void __launch_bounds__(256, seg_min_blocks(stage, NTR * LPT))               \
      name##_1(const __grid_constant__ Inst in, int t0, int w0) {                        \
    const int sub = int(blockIdx.y) * NTR;                                               \
    body<NTR, LPT, false>(in, lane_index(), t0 + sub, w0 + sub);                         \
  }                                                                                      \
  template <int NTR, int LPT>                                                            \
  __global__ void __launch_bounds__(256, seg_min_blocks(stage, NTR * LPT))               \
      name##_n(const Inst* __restrict__ tab, int t0, int w0, int S, unsigned mul) {      \
    const int slots = slice_div(256, mul), slot = slice_div(int(threadIdx.x), mul);      \
    if (slot >= slots) return;                                                           \
    const int sub = (int(threadIdx.x) - slot * S) * NTR;                                 \
    body<NTR, LPT, true>(tab[blockIdx.y], int64_t(blockIdx.x) * slots + slot, t0 + sub,  \
                         w0 + sub);                                                      \
  }

// The limiter stage: a block's first and last segment slot are halo runs.
#define FCT_SEG_LIMIT_KERNEL(name)                                                       \
  template <int NTR, int LPT>                                                            \
  __global__ void __launch_bounds__(256, seg_min_blocks(kStageLimit, NTR * LPT))         \
      name##_1(const __grid_constant__ Inst in, int t0, int w0) {                        \
    __shared__ double sh[4 * NTR * 256];                                                 \
    const int tid = threadIdx.x;                                                         \
    const int64_t si = int64_t(blockIdx.x) * 254 + tid - 1;                              \
    const int sub = int(blockIdx.y) * NTR;                                               \
    seg_node_limit<NTR, LPT, false>(in, si, tid >= 1 && tid <= 254, t0 + sub, w0 + sub,  \
                                    tid, 1, sh);                                         \
  }                                                                                      \
  template <int NTR, int LPT>                                                            \
  __global__ void __launch_bounds__(256, seg_min_blocks(kStageLimit, NTR * LPT))         \
      name##_n(const Inst* __restrict__ tab, int t0, int w0, int S, unsigned mul) {      \
    __shared__ double sh[4 * NTR * 256];                                                 \
    const int tid = threadIdx.x;                                                         \
    const int slots = slice_div(256, mul), slot = slice_div(tid, mul);                   \
    const int64_t si =                                                                   \
        slot < slots ? int64_t(blockIdx.x) * (slots - 2) + slot - 1 : int64_t(-1);       \
    const int sub = slot < slots ? (tid - slot * S) * NTR : 0;                           \
    seg_node_limit<NTR, LPT, true>(tab[blockIdx.y], si, slot >= 1 && slot <= slots - 2,  \
                                   t0 + sub, w0 + sub, tid, S, sh);                      \
  }

inline unsigned seg_blocks(int64_t lanes, int per_block) {
  return unsigned(std::max<int64_t>(1, (lanes + per_block - 1) / per_block));
}
// grids: 256/S segments per block; the limiter's blocks hold two halo slots
#define FCT_GRID(lanes, S) seg_blocks(lanes, 256 / (S))
#define FCT_LIMIT_GRID(lanes, S) seg_blocks(lanes, 256 / (S) - 2)

#define FCT_SEG_CASE_N(kern, P, V)                                                       \
  case P * 16 + V:                                                                       \
    kern##_n<P, V><<<g, 256, 0, s>>>(tab, t0, w0, S, mul);                               \
    break;
#define FCT_SEG_CASE_1(kern, P, V)                                                       \
  case P * 16 + V:                                                                       \
    kern##_1<P, V><<<g, 256, 0, s>>>(single, t0, w0);                                    \
    break;

// One segment stage over the tracers [c0, c1) of a workspace chunk (workspace index of
// tracer t is t - c0): launches of P tracers x S slices. ``COUNT(V)`` is the largest
// segment count of the variant over the launch's instances.
#define FCT_SEG_LAUNCHER(fn, kern, COUNT, GRID, STAGE)                                   \
  int fn(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1, \
         cudaStream_t s) {                                                               \
    const int lpt = d.smap_levels[STAGE], per_thread = d.smap_tracers[STAGE];            \
    const int V = seg_variant(lpt);                                                      \
    const int64_t lanes = COUNT(V);                                                      \
    for (int t0 = c0; t0 < c1;) {                                                        \
      const int rem = c1 - t0;                                                           \
      const SegSplit sp = seg_split(rem, per_thread, tab != nullptr, seg_even(d));       \
      const int P = sp.tracers, S = sp.slices, w0 = t0 - c0;                             \
      if (tab) {                                                                         \
        const unsigned mul = 65536u / unsigned(S) + 1u;                                  \
        const dim3 g(GRID(lanes, S), unsigned(n));                                       \
        switch (P * 16 + lpt) {                                                          \
          FCT_SEG_CASE_N(kern, 1, 2) FCT_SEG_CASE_N(kern, 1, 4)                          \
          FCT_SEG_CASE_N(kern, 1, 8) FCT_SEG_CASE_N(kern, 2, 2)                          \
          FCT_SEG_CASE_N(kern, 2, 4) FCT_SEG_CASE_N(kern, 2, 8)                          \
          FCT_SEG_CASE_N(kern, 4, 2) FCT_SEG_CASE_N(kern, 4, 4)                          \
          FCT_SEG_CASE_N(kern, 4, 8)                                                     \
          default:                                                                       \
            return set_error(FCT_ERR_INVALID, "no segment kernel for %d tracers x %d "  \
                             "levels per thread", P, lpt);                              \
        }                                                                                \
      } else {                                                                           \
        const dim3 g(GRID(lanes, 1), unsigned(S));                                       \
        switch (P * 16 + lpt) {                                                          \
          FCT_SEG_CASE_1(kern, 1, 2) FCT_SEG_CASE_1(kern, 1, 4)                          \
          FCT_SEG_CASE_1(kern, 1, 8) FCT_SEG_CASE_1(kern, 2, 2)                          \
          FCT_SEG_CASE_1(kern, 2, 4) FCT_SEG_CASE_1(kern, 2, 8)                          \
          default:                                                                       \
            return set_error(FCT_ERR_INVALID, "no segment kernel for %d tracers x %d "  \
                             "levels per thread", P, lpt);                              \
        }                                                                                \
      }                                                                                  \
      t0 += P * S;                                                                       \
    }                                                                                    \
    const cudaError_t e = cudaGetLastError();                                            \
    return e == cudaSuccess ? FCT_OK : cuda_error(e, #fn);                               \
  }

// Kernels whose threads walk the segments (one level per thread): as many blocks as are
// resident at once (stream_grid). ``BODY(NTR, IL)`` names the body's instantiation.
#define FCT_STREAM_KERNEL(name, BODY, blocks)                                            \
  template <int NTR>                                                                     \
  __global__ void __launch_bounds__(256, blocks(NTR, false))                             \
      name##_1(const __grid_constant__ Inst in, int t0, int w0) {                        \
    const int sub = int(blockIdx.y) * NTR;                                               \
    BODY(NTR, false)(in, lane_index(), int64_t(gridDim.x) * 256, t0 + sub, w0 + sub);    \
  }                                                                                      \
  template <int NTR>                                                                     \
  __global__ void __launch_bounds__(256, blocks(NTR, true))                              \
      name##_n(const Inst* __restrict__ tab, int n, int t0, int w0, int S, unsigned mul) { \
    const int slots = slice_div(256, mul), slot = slice_div(int(threadIdx.x), mul);      \
    if (slot >= slots) return;                                                           \
    const int sub = (int(threadIdx.x) - slot * S) * NTR;                                 \
    for (int i = int(blockIdx.y); i < n; i += int(gridDim.y))                            \
      BODY(NTR, true)(tab[i], int64_t(blockIdx.x) * slots + slot,                        \
                      int64_t(gridDim.x) * slots, t0 + sub, w0 + sub);                   \
  }
#define FCT_STREAM_LIMIT_KERNEL(name, blocks, batch)                                         \
  template <int NTR>                                                                     \
  __global__ void __launch_bounds__(256, blocks(NTR, false))                             \
      name##_1(const __grid_constant__ Inst in, int t0, int w0) {                        \
    __shared__ double sh[4 * NTR * 256];                                                 \
    const int tid = threadIdx.x, sub = int(blockIdx.y) * NTR;                            \
    const int64_t stride = int64_t(gridDim.x) * 254, b0 = int64_t(blockIdx.x) * 254;     \
    const int64_t rounds = (in.m.n_nseg[0] - b0 + stride - 1) / stride;                  \
    stream_node_limit<NTR, false, batch(NTR, false)>(in, b0 + tid - 1, stride, rounds,                   \
                                     tid >= 1 && tid <= 254, t0 + sub, w0 + sub, tid, 1, sh); \
  }                                                                                      \
  template <int NTR>                                                                     \
  __global__ void __launch_bounds__(256, blocks(NTR, true))                              \
      name##_n(const Inst* __restrict__ tab, int n, int t0, int w0, int S, unsigned mul) { \
    __shared__ double sh[4 * NTR * 256];                                                 \
    const int tid = threadIdx.x;                                                         \
    const int slots = slice_div(256, mul), slot = slice_div(tid, mul);                   \
    const int sub = slot < slots ? (tid - slot * S) * NTR : 0;                           \
    const int64_t stride = int64_t(gridDim.x) * (slots - 2);                             \
    const int64_t b0 = int64_t(blockIdx.x) * (slots - 2);                                \
    for (int i = int(blockIdx.y); i < n; i += int(gridDim.y)) {                          \
      const int64_t rounds = (tab[i].m.n_nseg[0] - b0 + stride - 1) / stride;            \
      stream_node_limit<NTR, true, batch(NTR, true)>(tab[i], b0 + slot - 1, stride, rounds,             \
                                      slot >= 1 && slot <= slots - 2, t0 + sub, w0 + sub, \
                                      tid, S, sh);                                       \
      __syncthreads();                                                                   \
    }                                                                                    \
  }
#define FCT_STREAM_LAUNCHER(fn, kern, COUNT, GRID, STAGE, blocks)                        \
  int fn(const Inst& single, const Inst* tab, int n, const LaunchDims& d, int c0, int c1, \
         cudaStream_t s) {                                                               \
    for (int t0 = c0; t0 < c1;) {                                                        \
      const SegSplit sp =                                                                \
          seg_split(c1 - t0, d.smap_tracers[STAGE], tab != nullptr, seg_even(d));        \
      const int P = sp.tracers, S = sp.slices, w0 = t0 - c0;                             \
      const int64_t need = GRID(COUNT(0), tab ? S : 1), full = int64_t(148) * blocks(P, tab != nullptr); \
      if (tab) {                                                                         \
        const unsigned mul = 65536u / unsigned(S) + 1u;                                  \
        const dim3 g = stream_grid(need, full, n);                                       \
        if (P == 4) kern##_n<4><<<g, 256, 0, s>>>(tab, n, t0, w0, S, mul);               \
        else if (P == 2) kern##_n<2><<<g, 256, 0, s>>>(tab, n, t0, w0, S, mul);          \
        else kern##_n<1><<<g, 256, 0, s>>>(tab, n, t0, w0, S, mul);                      \
      } else {                                                                           \
        const int64_t per = std::max<int64_t>(1, full / S);                              \
        const dim3 g(unsigned(std::max<int64_t>(1, std::min(need, per))), unsigned(S));  \
        if (P == 2) kern##_1<2><<<g, 256, 0, s>>>(single, t0, w0);                       \
        else kern##_1<1><<<g, 256, 0, s>>>(single, t0, w0);                              \
      }                                                                                  \
      t0 += P * S;                                                                       \
    }                                                                                    \
    const cudaError_t e = cudaGetLastError();                                            \
    return e == cudaSuccess ? FCT_OK : cuda_error(e, #fn);                               \
  }

}  // namespace
}  // namespace fct
