// FCT forward kernels (sm_100a, FP64): fesom_jax/tracer_adv.py:532-578 split into
// stage kernels over wet-lane lists. Every edge->node or element->node reduction is a
// deterministic gather over a CSR list in ascending edge/element id, so results are
// bit-identical run to run (no atomics).
//
// Stage map (reference function -> kernel):
//   edge_vflux (tracer_adv.py:69-93)                         -> k_vflux      (edge lanes)
//   tracer_gradient_elements (:316-326)                      -> k_elem_grad  (element lanes)
//   adv_flux_hor/adv_flux_ver (:96-120), compute_fct_lo (:298-313),
//   _node_avg_grad (:329-341), adv_flux_ver_ho (:241-295)    -> k_node_lo    (interface lanes)
//   adv_tra_vert_impl (:487-529), w_split only               -> k_vert_impl  (node columns)
//   fill_up_dn_grad (:344-368), adv_flux_hor_ho (:196-225)   -> k_edge_adf   (edge lanes)
//   zalesak_limit a2 (:393-397)                              -> k_elem_bounds(element lanes)
//   zalesak_limit a3 (:399-405)                              -> k_node_cluster (layer lanes)
//   zalesak_limit a4, b1, b2 (:407-451)                      -> k_node_factors (layer lanes)
//   zalesak_limit b3 (:453-465), flux2dtracer_fct (:469-484),
//   ale_reconstruct (:142-151)                               -> k_node_final (layer lanes)
//   invalid lanes keep T (ale_reconstruct)                   -> k_copy_dry   (dry lanes)
//
// Each thread owns one lane and NTR tracers (a compile-time chunk of the instance's
// tracers, which share its velocities): mesh indices, geometry and velocity terms are
// loaded once per lane and every neighbour gather issues NTR independent loads, so the
// gathers overlap.
#include <algorithm>

#include "fct_columns.cuh"

namespace fct {

namespace {

// ---------------------------------------------------------------- edge_vflux
// A thread walks the edge lanes i, i + stride, ...: the next lane's cells are loaded while this
// lane's velocities are under way (82 us on the CORE2-size mesh when each thread took one lane
// and waited for its lane, its cells and its velocities in a row).
__device__ __forceinline__ void body_vflux(const Inst& in, int64_t i, int64_t stride) {
  const DevMesh& m = in.m;
  const int64_t count = m.n_edge;
  if (i >= count) return;
  const int L = m.L;
  const double2* uv = reinterpret_cast<const double2*>(in.uv);
  uint32_t lane = ld(m.edge_lanes + i);
  uint32_t lane1 = i + stride < count ? ld(m.edge_lanes + i + stride) : lane;
  int4 ec = __ldg(m.ecell4 + lane_ent(lane));   // cells and their layer ranges in one load
  for (; i < count; i += stride) {
    const int e = lane_ent(lane), k = lane_lev(lane);
    const unsigned tr = unsigned(ec.z);
    const bool on1 = in_range(k, tr & 0xffffu);
    const bool on2 = ((tr >> 16) & 255u) != kNoCell && in_range(k, tr >> 16);
    const double2* cr = reinterpret_cast<const double2*>(m.cross + 4 * int64_t(e));
    const double2 c1 = __ldg(cr), c2 = __ldg(cr + 1);
    double2 U1 = make_double2(0.0, 0.0), U2 = U1;
    double h1 = 0.0, h2 = 0.0;
    if (on1) {
      const uint32_t q = lq(ec.x, L, k);
      U1 = __ldg(uv + q);
      h1 = ld(in.helem + q);
    }
    if (on2) {
      const uint32_t q = lq(ec.y, L, k);
      U2 = __ldg(uv + q);
      h2 = ld(in.helem + q);
    }
    lane = lane1;
    ec = __ldg(m.ecell4 + lane_ent(lane));
    lane1 = i + 2 * stride < count ? ld(m.edge_lanes + i + 2 * stride) : lane;
    const double t1 = on1 ? (U1.x * c1.y - U1.y * c1.x) * h1 : 0.0;
    const double t2 = on2 ? (U2.y * c2.x - U2.x * c2.y) * h2 : 0.0;
    in.ws.vflux[lq(e, L, k)] = t1 + t2;
  }
}

template <int NTR>
__device__ __forceinline__ void body_elem_grad(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_elem) return;
  const uint32_t lane = ld(m.elem_lanes + i);
  const int e = lane_ent(lane), k = lane_lev(lane), L = m.L;
  double gx[NTR], gy[NTR];
  cell_grad<NTR, false>(in, e, k, t0, gx, gy);
  const uint32_t q = lq(e, L, k);
  stn<NTR, false>(in.ws.gx, q, w0, in.ws.sE, in.wtg, gx);
  stn<NTR, false>(in.ws.gy, q, w0, in.ws.sE, in.wtg, gy);
}

// -------------------------------- LO solution, node-average gradient, adf_v
template <int NTR>
__device__ __forceinline__ void body_node_lo(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_iface) return;
  const int4 rec = __ldg(m.iface4 + i);
  const unsigned pk = unsigned(rec.w);
  const int n = lane_ent(uint32_t(rec.x)), k = lane_lev(uint32_t(rec.x)), L = m.L;
  const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
  const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k);
  const bool layer = k < nzmax;
  const bool layer1 = (k + 1) < nzmax;
  const int km1 = k > 0 ? k - 1 : 0;
  const double w = ld(in.w_e + qn);
  const double Wf = in.w_i ? w + ld(in.w_i + qn) : w;   // w_full for the HO flux
  const double area_k = ld(m.area + qn);
  const int64_t ts = in.tstride;
  const int tg = in.tg;

  double Tc[NTR], Ta[NTR];   // T[k], T[k-1]
  ldn<NTR, false>(in.T, qn, t0, ts, tg, Tc);
  ldn<NTR, false>(in.T, base + km1, t0, ts, tg, Ta);
  double fvk[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) fvk[t] = layer ? vflux_up(Tc[t], Ta[t], w, area_k) : 0.0;

  if (layer) {
    const double hn = ld(in.hnode + qn), hnn = ld(in.hnode_new + qn);
    const double av = ld(m.areasvol + qn);
    const Rcp rav = rcp_known(av, ld(m.iavol + qn)), rhn = rcp(hnn);   // shared by the NTR
                                                                       // quotients below
    const double dt = in.dt;
    double fvk1[NTR];
    if (layer1) {
      const double w1 = ld(in.w_e + qn + 1), area1 = ld(m.area + qn + 1);
      double Tb[NTR];
      ldn<NTR, false>(in.T, qn + 1, t0, ts, tg, Tb);
#pragma unroll
      for (int t = 0; t < NTR; ++t) fvk1[t] = vflux_up(Tb[t], Tc[t], w1, area1);
    } else {
#pragma unroll
      for (int t = 0; t < NTR; ++t) fvk1[t] = 0.0;
    }
    // compute_fct_lo: edge->node upwind divergence in ascending edge id
    double div[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) div[t] = 0.0;
    const int e0 = rec.y, e1 = rec.y + int((pk >> 16) & 255u);
    const unsigned long long flags = __ldg(m.nflags + __ldg(m.nrec + n).w + (k - nzmin));
    unsigned onb = unsigned(flags);   // bit j: the j-th slot's edge has the layer
    for (int j = e0; j < e1; ++j, onb >>= 1) {
      const int4 sl = __ldg(m.ns4 + j);
      if (!(onb & 1u)) continue;   // vflux == 0 there
      const double vf = ld(in.ws.vflux + (uint32_t(sl.x) + uint32_t(k)));
      const double avf = fabs(vf);
      // the face flux with the node's own value first (a + b == b + a exactly)
      const double cown = sl.z ? vf - avf : vf + avf, coth = sl.z ? vf + avf : vf - avf;
      double To[NTR];
      ldn<NTR, false>(in.T, uint32_t(sl.y) + uint32_t(k), t0, ts, tg, To);
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        const double fl = -0.5 * (Tc[t] * cown + To[t] * coth);
        div[t] += sl.z ? -fl : fl;
      }
    }
  
    const bool valid = (hnn > 0.0) && (av > 0.0);
    double lo[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      lo[t] = valid ? divr(Tc[t] * hn + divr((div[t] + (fvk[t] - fvk1[t])) * dt, rav), rhn)
                    : 0.0;
    stn<NTR, false>(in.ws.lo, qn, w0, in.ws.sN, in.wtg, lo);
    // _node_avg_grad: area-weighted mean over the node's active elements, at the levels
    // where an edge of the node takes it (kGradBit; its readers, the edge stage's and the
    // reverse pass's node-gradient lanes, read no other level)
    if ((flags >> kGradBit) & 1ull) {
      double nx[NTR], ny[NTR], den = 0.0;
#pragma unroll
      for (int t = 0; t < NTR; ++t) nx[t] = ny[t] = 0.0;
      const int c0 = rec.z, c1 = rec.z + int(pk >> 24);
      for (int j = c0; j < c1; ++j) {
        const int el = ld(m.nel_idx + j);
        if (k >= ld(m.eul + el) && k < ld(m.enl + el)) {
          const double a = ld(m.earea + el);
          const uint32_t qe = lq(el, L, k);
          double gx[NTR], gy[NTR];
          ldn<NTR, false>(in.ws.gx, qe, w0, in.ws.sE, in.wtg, gx);
          ldn<NTR, false>(in.ws.gy, qe, w0, in.ws.sE, in.wtg, gy);
#pragma unroll
          for (int t = 0; t < NTR; ++t) {
            nx[t] += gx[t] * a;
            ny[t] += gy[t] * a;
          }
          den += a;
        }
      }
      const Rcp rdd = rcp(den > 0.0 ? den : 1.0);
      if (w0 == 0) in.ws.nden[qn] = rdd.y;   // kept for the reverse pass (tracer independent)
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        nx[t] = divr(nx[t], rdd);
        ny[t] = divr(ny[t], rdd);
      }
      stn<NTR, false>(in.ws.gnx, qn, w0, in.ws.sN, in.wtg, nx);
      stn<NTR, false>(in.ws.gny, qn, w0, in.ws.sN, in.wtg, ny);
    }
  }

  // adv_flux_ver_ho (QR4C on ttfAB) minus the LO vertical flux (tracer_adv.py:241-295)
  double hi[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) hi[t] = 0.0;
  if (k == nzmin) {
    double To[NTR];
    ldn<NTR, false>(in.T_old, qn, t0, ts, tg, To);
#pragma unroll
    for (int t = 0; t < NTR; ++t) hi[t] = -ab2(Tc[t], To[t]) * Wf * area_k;
  } else if (k == nzmax) {
    // bottom interface: no flux
  } else if (k == nzmin + 1 || k == nzmax - 1) {
    double To[NTR], Tom[NTR];
    ldn<NTR, false>(in.T_old, qn, t0, ts, tg, To);
    ldn<NTR, false>(in.T_old, qn - 1, t0, ts, tg, Tom);
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      hi[t] = -0.5 * (ab2(Ta[t], Tom[t]) + ab2(Tc[t], To[t])) * Wf * area_k;
  } else if (k >= nzmin + 2 && k <= nzmax - 2) {
    double Znz, Zm1, Zm2, Zp1, zb;   // QR4C stencil depths (tracer_adv.py:228-238, 265-273)
    if (in.Z3d) {
      const double* Zc = in.Z3d + base;
      Znz = ld(Zc + k); Zm1 = ld(Zc + k - 1); Zm2 = ld(Zc + k - 2);
      Zp1 = ld(Zc + (k + 1 < L ? k + 1 : L - 1)); zb = ld(in.zbar3 + qn);
    } else {
      Znz = ld(m.Zp + k); Zm1 = ld(m.Zp + k - 1); Zm2 = ld(m.Zp + k - 2);
      Zp1 = ld(m.Zp + (k + 1 < L ? k + 1 : L - 1)); zb = ld(m.zbar + k);
    }
    Rcp rdc, rdu, rdd;
    if (in.Z3d) {
      rdc = rcp(safe_nz(Zm1 - Znz));
      rdu = rcp(safe_nz(Znz - Zp1));
      rdd = rcp(safe_nz(Zm2 - Zm1));
    } else {   // the static depths' reciprocals come from the plan
      rdc = rcp_known(safe_nz(Zm1 - Znz), ld(m.qr4c + k));
      rdu = rcp_known(safe_nz(Znz - Zp1), ld(m.qr4c + L + k));
      rdd = rcp_known(safe_nz(Zm2 - Zm1), ld(m.qr4c + 2 * L + k));
    }
    const Rcp r3{3.0, 1.0 / 3.0, true};
    double To[NTR], Tom[NTR], Tm2[NTR], Tom2[NTR], Tp[NTR], Top[NTR];
    ldn<NTR, false>(in.T_old, qn, t0, ts, tg, To);
    ldn<NTR, false>(in.T_old, qn - 1, t0, ts, tg, Tom);
    ldn<NTR, false>(in.T, qn - 2, t0, ts, tg, Tm2);
    ldn<NTR, false>(in.T_old, qn - 2, t0, ts, tg, Tom2);
    ldn<NTR, false>(in.T, qn + 1, t0, ts, tg, Tp);
    ldn<NTR, false>(in.T_old, qn + 1, t0, ts, tg, Top);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double A0 = ab2(Tc[t], To[t]), Am1 = ab2(Ta[t], Tom[t]);
      const double Am2 = ab2(Tm2[t], Tom2[t]), Ap1 = ab2(Tp[t], Top[t]);
      const double qc = divr(Am1 - A0, rdc);
      const double qu = divr(A0 - Ap1, rdu);
      const double qd = divr(Am2 - Am1, rdd);
      const double Tmean1 = A0 + divr((2.0 * qc + qu) * (zb - Znz), r3);
      const double Tmean2 = Am1 + divr((2.0 * qc + qd) * (zb - Zm1), r3);
      hi[t] = -0.5 * (Tmean1 + Tmean2) * Wf * area_k;
    }
  }
  double adf[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) {
    const double lo_v = in.w_i ? (layer ? vflux_up(Tc[t], Ta[t], Wf, area_k) : 0.0) : fvk[t];
    adf[t] = hi[t] - lo_v;
  }
  stn<NTR, false>(in.ws.adfv, qn, w0, in.ws.sN, in.wtg, adf);
}

// -------------------------- fill_up_dn_grad + adv_flux_hor_ho - LO flux = adf_h
// -0.5 ((vf + |vf|) Tm1 + (vf - |vf|) Tm2) is exactly -0.5 times the upwind end's term (the
// other one is 0 times a finite value), so only that end's gradient is read, and one component
// of the other's, times 0: a non-finite value on the other cell makes the flux NaN, as it does
// in the formula (a vertex that is not finite makes both components so; the reverse pass takes
// it from adf_h). 10-step chain on the CORE2-size mesh: 24.3 ms without that component,
// 24.6 with it, 24.9 with both gradients in full here and in r_edge. A thread walks the lanes
// i, i + stride, ...: the next lane's record, volume flux and cells are loaded while this lane's
// gathers are under way.
template <int NTR>
__device__ __forceinline__ void body_edge_adf(const Inst& in, int64_t i, int64_t stride, int t0,
                                              int w0) {
  const DevMesh& m = in.m;
  const int64_t count = m.n_edge;
  if (i >= count) return;
  const int L = m.L;
  const int64_t ts = in.tstride;
  const int tg = in.tg;
  const int2* updn = reinterpret_cast<const int2*>(m.eupdn);
  const double2* coef = reinterpret_cast<const double2*>(m.ecoef);
  int4 rec = __ldg(m.edge4 + i);
  int4 rec1 = i + stride < count ? __ldg(m.edge4 + i + stride) : rec;
  double vf1 = ld(in.ws.vflux + lq(lane_ent(uint32_t(rec.x)), L, lane_lev(uint32_t(rec.x))));
  int2 ud1 = __ldg(updn + lane_ent(uint32_t(rec.x)));
  for (; i < count; i += stride) {
    const int e = lane_ent(uint32_t(rec.x)), k = lane_lev(uint32_t(rec.x));
    const bool use_tri = in_range(k, unsigned(rec.w));
    const double vf = vf1, avf = fabs(vf);
    const uint32_t q1 = lq(rec.y, L, k), q2 = lq(rec.z, L, k);
    const bool first = vf > 0.0;
    double T1[NTR], T2[NTR], O1[NTR], O2[NTR], gx[NTR], gy[NTR], gd[NTR];
    ldn<NTR, false>(in.T, q1, t0, ts, tg, T1);
    ldn<NTR, false>(in.T, q2, t0, ts, tg, T2);
    ldn<NTR, false>(in.T_old, q1, t0, ts, tg, O1);
    ldn<NTR, false>(in.T_old, q2, t0, ts, tg, O2);
    if (use_tri) {
      // both cells are wet at k here (k is above every adjacent cell's bottom)
      const uint32_t q = lq(first ? ud1.x : ud1.y, L, k);
      ldn<NTR, false>(in.ws.gx, q, w0, in.ws.sE, in.wtg, gx);
      ldn<NTR, false>(in.ws.gy, q, w0, in.ws.sE, in.wtg, gy);
      ldn<NTR, false>(in.ws.gx, lq(first ? ud1.y : ud1.x, L, k), w0, in.ws.sE, in.wtg, gd);
    } else {
      const uint32_t q = first ? q1 : q2;
      ldn<NTR, false>(in.ws.gnx, q, w0, in.ws.sN, in.wtg, gx);
      ldn<NTR, false>(in.ws.gny, q, w0, in.ws.sN, in.wtg, gy);
      ldn<NTR, false>(in.ws.gnx, first ? q2 : q1, w0, in.ws.sN, in.wtg, gd);
    }
    const double2 c = __ldg(coef + e);
    rec = rec1;
    vf1 = ld(in.ws.vflux + lq(lane_ent(uint32_t(rec.x)), L, lane_lev(uint32_t(rec.x))));
    ud1 = __ldg(updn + lane_ent(uint32_t(rec.x)));
    rec1 = i + 2 * stride < count ? __ldg(m.edge4 + i + 2 * stride) : rec;
    double adf[NTR];
    const Rcp r6{6.0, 1.0 / 6.0, true};
    const double cu = first ? vf + avf : vf - avf;
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double fl = -0.5 * (T1[t] * (vf + avf) + T2[t] * (vf - avf));
      const double A1 = ab2(T1[t], O1[t]), A2 = ab2(T2[t], O2[t]);
      const double diff = A2 - A1;
      const double X = divr(2.0 * diff + c.x * gx[t] + c.y * gy[t], r6);
      const double Tm = first ? A1 + X : A2 - X;
      const double ho = -0.5 * (cu * Tm) + 0.0 * gd[t];
      adf[t] = ho - fl;
    }
    stn<NTR, false>(in.ws.adfh, lq(e, L, k), w0, in.ws.sEd, in.wtg, adf);
  }
}

// ------------------------ zalesak a2: element max/min of the LO/T window
template <int NTR>
__device__ __forceinline__ void body_elem_bounds(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_elem) return;
  const uint32_t lane = ld(m.elem_lanes + i);
  const int e = lane_ent(lane), k = lane_lev(lane), L = m.L;
  const uint32_t q[3] = {lq(ld(m.enodes + 3 * e), L, k),
                        lq(ld(m.enodes + 3 * e + 1), L, k),
                        lq(ld(m.enodes + 3 * e + 2), L, k)};
  double mx[NTR], mn[NTR], hi[3][NTR], lw[3][NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) { mx[t] = -INFINITY; mn[t] = INFINITY; }
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    double a[NTR], b[NTR];
    ldn<NTR, false>(in.ws.lo, q[v], w0, in.ws.sN, in.wtg, a);
    ldn<NTR, false>(in.T, q[v], t0, in.tstride, in.tg, b);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      hi[v][t] = fmax(a[t], b[t]);
      lw[v][t] = fmin(a[t], b[t]);
      mx[t] = fmax(mx[t], hi[v][t]);
      mn[t] = fmin(mn[t], lw[v][t]);
    }
  }
  const uint32_t qe = lq(e, L, k);
  {   // vertices attaining the bounds (the reverse pass splits cotangents evenly over them)
    int cx[NTR], cn[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      cx[t] = (hi[0][t] == mx[t]) + (hi[1][t] == mx[t]) + (hi[2][t] == mx[t]);
      cn[t] = (lw[0][t] == mn[t]) + (lw[1][t] == mn[t]) + (lw[2][t] == mn[t]);
    }
    stc<NTR, false>(in.ws.ecx, qe, w0, in.ws.sE, in.wtg, cx);
    stc<NTR, false>(in.ws.ecn, qe, w0, in.ws.sE, in.wtg, cn);
  }
  stn<NTR, false>(in.ws.amax, qe, w0, in.ws.sE, in.wtg, mx);
  stn<NTR, false>(in.ws.amin, qe, w0, in.ws.sE, in.wtg, mn);
}

// ------------------------ zalesak a3: node cluster max/min over elements
template <int NTR>
__device__ __forceinline__ void body_node_cluster(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_layer) return;
  const int4 rec = __ldg(m.layer4 + i);
  const int n = lane_ent(uint32_t(rec.x)), k = lane_lev(uint32_t(rec.x)), L = m.L;
  const int c0 = rec.z, c1 = rec.z + int(unsigned(rec.w) >> 24);
  double mx[NTR], mn[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) { mx[t] = -INFINITY; mn[t] = INFINITY; }
  for (int j = c0; j < c1; ++j) {
    const int el = ld(m.nel_idx + j);
    if (k >= ld(m.eul + el) && k < ld(m.enl + el)) {
      const uint32_t q = lq(el, L, k);
      double a[NTR], b[NTR];
      ldn<NTR, false>(in.ws.amax, q, w0, in.ws.sE, in.wtg, a);
      ldn<NTR, false>(in.ws.amin, q, w0, in.ws.sE, in.wtg, b);
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        mx[t] = fmax(mx[t], a[t]);
        mn[t] = fmin(mn[t], b[t]);
      }
    } else {   // a cell without this level pads with -+BIG (tracer_adv.py:396-397)
#pragma unroll
      for (int t = 0; t < NTR; ++t) {
        mx[t] = fmax(mx[t], -kBig);
        mn[t] = fmin(mn[t], kBig);
      }
    }
  }
  const uint32_t qn = lq(n, L, k);
  stn<NTR, false>(in.ws.tvmax, qn, w0, in.ws.sN, in.wtg, mx);
  stn<NTR, false>(in.ws.tvmin, qn, w0, in.ws.sN, in.wtg, mn);
  // cells attaining the cluster bounds (padded values included), for the reverse pass
  int cx[NTR], cn[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) cx[t] = cn[t] = 0;
  for (int j = c0; j < c1; ++j) {
    const int el = ld(m.nel_idx + j);
    double a[NTR], b[NTR];
    if (k >= ld(m.eul + el) && k < ld(m.enl + el)) {
      const uint32_t q = lq(el, L, k);
      ldn<NTR, false>(in.ws.amax, q, w0, in.ws.sE, in.wtg, a);
      ldn<NTR, false>(in.ws.amin, q, w0, in.ws.sE, in.wtg, b);
    } else {
#pragma unroll
      for (int t = 0; t < NTR; ++t) { a[t] = -kBig; b[t] = kBig; }
    }
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      cx[t] += a[t] == mx[t];
      cn[t] += b[t] == mn[t];
    }
  }
  stc<NTR, false>(in.ws.ccx, qn, w0, in.ws.sN, in.wtg, cx);
  stc<NTR, false>(in.ws.ccn, qn, w0, in.ws.sN, in.wtg, cn);
}

// ------------------- zalesak a4 + b1 + b2: admissible window, sums, factors
template <int NTR>
__device__ __forceinline__ void body_node_factors(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_layer) return;
  const int4 rec = __ldg(m.layer4 + i);
  const unsigned pk = unsigned(rec.w);
  const int n = lane_ent(uint32_t(rec.x)), k = lane_lev(uint32_t(rec.x)), L = m.L;
  const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
  const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k);
  const bool use_own = (k == nzmin) || (k == nzmax - 1);
  const double av = ld(m.areasvol + qn), hnn = ld(in.hnode_new + qn);
  const bool valid = (av > 0.0) && (hnn > 0.0);
  const double sh = hnn > 0.0 ? hnn : 1.0;
  const Rcp rsa = av > 0.0 ? rcp_known(av, ld(m.iavol + qn)) : Rcp{1.0, 1.0, true};
  const Rcp rsh = rcp(sh);
  const double dt = in.dt;
  const int64_t sN = in.ws.sN;
  double tmax[NTR], tmin[NTR];
  ldn<NTR, false>(in.ws.tvmax, qn, w0, sN, in.wtg, tmax);
  ldn<NTR, false>(in.ws.tvmin, qn, w0, sN, in.wtg, tmin);
  if (!use_own) {   // interior: max/min over k-1, k, k+1 (all layers of this column)
    double am[NTR], an[NTR], bm[NTR], bn[NTR];
    ldn<NTR, false>(in.ws.tvmax, qn - 1, w0, sN, in.wtg, am);
    ldn<NTR, false>(in.ws.tvmin, qn - 1, w0, sN, in.wtg, an);
    ldn<NTR, false>(in.ws.tvmax, qn + 1, w0, sN, in.wtg, bm);
    ldn<NTR, false>(in.ws.tvmin, qn + 1, w0, sN, in.wtg, bn);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      tmax[t] = fmax(fmax(am[t], tmax[t]), bm[t]);
      tmin[t] = fmin(fmin(an[t], tmin[t]), bn[t]);
    }
  }
  double lo[NTR], ft[NTR], fb[NTR];
  ldn<NTR, false>(in.ws.lo, qn, w0, sN, in.wtg, lo);
  ldn<NTR, false>(in.ws.adfv, qn, w0, sN, in.wtg, ft);
  ldn<NTR, false>(in.ws.adfv, qn + 1, w0, sN, in.wtg, fb);   // k+1 <= nzmax < L
  double sp[NTR], sm[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) sp[t] = sm[t] = 0.0;
  const int e0 = rec.y, e1 = rec.y + int((pk >> 16) & 255u);
  unsigned onb = unsigned(__ldg(m.nflags + i));   // (flag words in lane order)
  for (int j = e0; j < e1; ++j, onb >>= 1) {
    const int4 sl = __ldg(m.ns4 + j);
    if (!(onb & 1u)) continue;   // no flux on this level
    double a[NTR];
    ldn<NTR, false>(in.ws.adfh, uint32_t(sl.x) + uint32_t(k), w0, in.ws.sEd, in.wtg, a);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      const double s = sl.z ? -a[t] : a[t];
      sp[t] += fmax(s, 0.0);
      sm[t] += fmin(s, 0.0);
    }
  }
  double pf[NTR], mf[NTR], pl[NTR], mi[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) {
    const double plus = (fmax(ft[t], 0.0) + fmax(-fb[t], 0.0)) + sp[t];
    const double minus = (fmin(ft[t], 0.0) + fmin(-fb[t], 0.0)) + sm[t];
    pl[t] = plus;
    mi[t] = minus;
    pf[t] = 1.0;
    mf[t] = 1.0;
    if (valid) {
      const double flux_pos = divr(divr(plus * dt, rsa), rsh) + kFluxEps;
      const double flux_neg = divr(divr(minus * dt, rsa), rsh) - kFluxEps;
      pf[t] = fmin(1.0, (tmax[t] - lo[t]) / flux_pos);
      mf[t] = fmin(1.0, (tmin[t] - lo[t]) / flux_neg);
    }
  }
  stn<NTR, false>(in.ws.pf, qn, w0, sN, in.wtg, pf);
  stn<NTR, false>(in.ws.mf, qn, w0, sN, in.wtg, mf);
  stn<NTR, false>(in.ws.fplus, qn, w0, sN, in.wtg, pl);    // kept for the reverse pass
  stn<NTR, false>(in.ws.fminus, qn, w0, sN, in.wtg, mi);
}

// ---------- zalesak b3 + flux2dtracer_fct + ale_reconstruct: T_new on layers
template <int NTR>
__device__ __forceinline__ void body_node_final(const Inst& in, int64_t i, int t0, int w0) {
  const DevMesh& m = in.m;
  if (i >= m.n_layer) return;
  const int4 rec = __ldg(m.layer4 + i);
  const unsigned pk = unsigned(rec.w);
  const int n = lane_ent(uint32_t(rec.x)), k = lane_lev(uint32_t(rec.x)), L = m.L;
  const int nzmin = int(pk & 255u), nzmax = int((pk >> 8) & 255u);
  const uint32_t base = lq(n, L, 0), qn = base + uint32_t(k);
  const double av = ld(m.areasvol + qn);
  const double hn = ld(in.hnode + qn), hnn = ld(in.hnode_new + qn);
  const Rcp rsa = av > 0.0 ? rcp_known(av, ld(m.iavol + qn)) : Rcp{1.0, 1.0, true};
  const Rcp rhn = rcp(hnn);
  const double dt = in.dt;
  const int tg = in.tg;
  const int64_t sN = in.ws.sN;
  // own limiter factors at k (and k-1 / k+1 for the vertical fluxes)
  double pf0[NTR], mf0[NTR], ft[NTR];
  ldn<NTR, false>(in.ws.pf, qn, w0, sN, in.wtg, pf0);
  ldn<NTR, false>(in.ws.mf, qn, w0, sN, in.wtg, mf0);
  ldn<NTR, false>(in.ws.adfv, qn, w0, sN, in.wtg, ft);
  // limited vertical flux at the top interface k (tracer_adv.py:453-459)
  double vt[NTR];
  if (k == nzmin) {
#pragma unroll
    for (int t = 0; t < NTR; ++t) vt[t] = (ft[t] >= 0.0 ? pf0[t] : mf0[t]) * ft[t];
  } else {
    double pfa[NTR], mfa[NTR];
    ldn<NTR, false>(in.ws.pf, qn - 1, w0, sN, in.wtg, pfa);
    ldn<NTR, false>(in.ws.mf, qn - 1, w0, sN, in.wtg, mfa);
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      vt[t] = (ft[t] >= 0.0 ? fmin(mfa[t], pf0[t]) : fmin(pfa[t], mf0[t])) * ft[t];
  }
  // limited vertical flux at the bottom interface k+1 (0 at the node's bottom)
  double vb[NTR];
  if (k + 1 >= nzmax) {
#pragma unroll
    for (int t = 0; t < NTR; ++t) vb[t] = 0.0;
  } else {
    double fb[NTR], pfb[NTR], mfb[NTR];
    ldn<NTR, false>(in.ws.adfv, qn + 1, w0, sN, in.wtg, fb);
    ldn<NTR, false>(in.ws.pf, qn + 1, w0, sN, in.wtg, pfb);
    ldn<NTR, false>(in.ws.mf, qn + 1, w0, sN, in.wtg, mfb);
#pragma unroll
    for (int t = 0; t < NTR; ++t)
      vb[t] = (fb[t] >= 0.0 ? fmin(mf0[t], pfb[t]) : fmin(pf0[t], mfb[t])) * fb[t];
  }
  // limited horizontal fluxes, ascending edge id
  double hsc[NTR];
#pragma unroll
  for (int t = 0; t < NTR; ++t) hsc[t] = 0.0;
  const int e0 = rec.y, e1 = rec.y + int((pk >> 16) & 255u);
  unsigned onb = unsigned(__ldg(m.nflags + i));   // (flag words in lane order)
  for (int j = e0; j < e1; ++j, onb >>= 1) {
    const int4 sl = __ldg(m.ns4 + j);
    if (!(onb & 1u)) continue;   // no flux on this level
    const uint32_t qo = uint32_t(sl.y) + uint32_t(k);
    double a[NTR], pfo[NTR], mfo[NTR];
    ldn<NTR, false>(in.ws.adfh, uint32_t(sl.x) + uint32_t(k), w0, in.ws.sEd, in.wtg, a);
    ldn<NTR, false>(in.ws.pf, qo, w0, sN, in.wtg, pfo);
    ldn<NTR, false>(in.ws.mf, qo, w0, sN, in.wtg, mfo);
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
      // ae = a >= 0 ? min(plus(n1), minus(n2)) : min(minus(n1), plus(n2)): the own plus and
      // the other's minus when the flux leaves the node, else the other pair
      const bool leaves = (a[t] >= 0.0) != (sl.z != 0);
      const double ae = fmin(leaves ? pf0[t] : mf0[t], leaves ? mfo[t] : pfo[t]);
      const double lim = ae * a[t];
      hsc[t] += sl.z ? -lim : lim;
    }
  }
  double Tv[NTR], lo[NTR], out[NTR];
  ldn<NTR, false>(in.T, qn, t0, in.tstride, tg, Tv);
  ldn<NTR, false>(in.ws.lo, qn, w0, sN, in.wtg, lo);
#pragma unroll
  for (int t = 0; t < NTR; ++t) {
    const double lo_trans = -Tv[t] * hn + lo[t] * hnn;
    const double vdiv = av > 0.0 ? divr((vt[t] - vb[t]) * dt, rsa) : 0.0;
    double d = divr(hsc[t] * dt, rsa) + (lo_trans + vdiv);
    d = d + Tv[t] * (hn - hnn);
    out[t] = Tv[t] + (hnn > 0.0 ? divr(d, rhn) : 0.0);
  }
  stn<NTR, false>(in.T_new, qn, t0, in.tstride, tg, out);
  count_nonfinite<NTR>(in.nonfinite, out);
}

// Kernel wrappers: ``_1`` takes one instance by value, ``_n`` reads instance blockIdx.y of a
// device table (interleaved layout, the batched path). The stage-by-stage kernels take one
// instance (tracer-major); a launch covers S = 2^lg tracer slices of NTR tracers each, the
// slice is blockIdx.y, so lanes stay contiguous along x within each tracer plane.
// Resident 256-thread blocks per SM the compiler must fit (registers capped
// accordingly): latency hiding pays more than the spills it costs (one tracer, the
// adjoint's taped forward on the CORE2-size mesh: 11.1 ms for 10 steps at 6 blocks,
// 10.6 ms at 7, no gain at 8).
template <int NTR>
constexpr int kMinBlocks = NTR == 1 ? 7 : NTR == 2 ? 5 : NTR == 4 ? 4 : 2;

#define FCT_KERNEL_T(name, body)                                                        \
  template <int NTR>                                                                    \
  __global__ void __launch_bounds__(256, kMinBlocks<NTR>) name##_1(                       \
      const __grid_constant__ Inst in, int t0, int w0) {                                \
    const int sub = int(blockIdx.y) * NTR;                                              \
    body<NTR>(in, lane_index(), t0 + sub, w0 + sub);                                    \
  }

// unfused stages (every intermediate in the workspace; the reverse pass reads them)
FCT_KERNEL_T(k_elem_grad, body_elem_grad)
FCT_KERNEL_T(k_node_lo, body_node_lo)
// (a walk over the edge lanes)
template <int NTR>
constexpr int kWalkBlocks = NTR == 1 ? 5 : NTR == 2 ? 4 : NTR == 4 ? 2 : 1;
template <int NTR>
__global__ void __launch_bounds__(256, kWalkBlocks<NTR>) k_edge_adf_1(
    const __grid_constant__ Inst in, int t0, int w0) {
  const int sub = int(blockIdx.y) * NTR;
  body_edge_adf<NTR>(in, lane_index(), int64_t(gridDim.x) * 256, t0 + sub, w0 + sub);
}
FCT_KERNEL_T(k_elem_bounds, body_elem_bounds)
FCT_KERNEL_T(k_node_cluster, body_node_cluster)
FCT_KERNEL_T(k_node_factors, body_node_factors)
FCT_KERNEL_T(k_node_final, body_node_final)

// column solves (fct_columns.cuh) of NT tracers: blockIdx.y the instance (batched)
#define FCT_KERNEL_COL(name, block_body)                                                 \
  template <int NT>                                                                      \
  __global__ void __launch_bounds__(kColThreads) name##_1(                               \
      const __grid_constant__ Inst in, int columns, int t0) {                            \
    extern __shared__ double col_sh[];                                                   \
    block_body<NT, false>(in, int(blockIdx.x) * columns, columns, t0, col_sh);           \
  }                                                                                      \
  template <int NT>                                                                      \
  __global__ void __launch_bounds__(kColThreads) name##_n(                               \
      const Inst* __restrict__ tab, int columns, int t0) {                               \
    extern __shared__ double col_sh[];                                                   \
    block_body<NT, true>(tab[blockIdx.y], int(blockIdx.x) * columns, columns, t0, col_sh); \
  }
// implicit vertical diffusion (the epilogue of the batched step and fct_vert_diff)
FCT_KERNEL_COL(k_vdiff, block_vdiff)
FCT_KERNEL_COL(k_vert_impl, block_vert_impl)
__global__ void __launch_bounds__(256, kPairBlocks) k_vdiff_pairs_n(
    const Inst* __restrict__ tab, int t0) {
  const int64_t g = lane_index();
  const int sub = int(g % (kPairTracers / 2)) * 2;
  pair_vdiff(tab[blockIdx.y], g / (kPairTracers / 2), t0 + sub, sub);
}

constexpr int kVfluxBlocks = 5;
__global__ void __launch_bounds__(256, kVfluxBlocks) k_vflux_1(const __grid_constant__ Inst in) {
  body_vflux(in, lane_index(), int64_t(gridDim.x) * 256);
}
__global__ void __launch_bounds__(256, kVfluxBlocks) k_vflux_n(const Inst* __restrict__ tab,
                                                               int n) {
  for (int i = int(blockIdx.y); i < n; i += int(gridDim.y))
    body_vflux(tab[i], lane_index(), int64_t(gridDim.x) * 256);
}
__global__ void __launch_bounds__(256) k_copy_dry_1(const __grid_constant__ Inst in) {
  body_copy_dry<false>(in, lane_index());
}
__global__ void __launch_bounds__(256) k_copy_dry_n(const Inst* __restrict__ tab) {
  body_copy_dry<true>(tab[blockIdx.y], lane_index());
}

}  // namespace

const char* const kStageNames[kNumStages] = {
    "vflux", "elem_grad", "node_lo", "vert_impl", "edge_adf", "elem_bounds",
    "node_cluster", "node_factors", "node_final", "copy_dry"};

// One stage-by-stage stage over the tracers [c0, c1) of a workspace chunk: launches of S slices
// x NTR tracers, NTR in {8, 4, 2, 1} (largest first) and S the largest power of two (at most 8)
// with S*NTR tracers left; the workspace index of tracer t is t - c0.
#define FCT_STAGE_AS(name, lanes, P)                                                    \
  name##_1<P><<<dim3(xblocks(lanes), 1u << lg), B, 0, s>>>(single, t0, w0)

#define FCT_SPLIT(AS, name, lanes)                                                      \
  do {                                                                                  \
    for (int t0 = c0; t0 < c1;) {                                                       \
      const int rem = c1 - t0;                                                          \
      const int P = rem >= 8 ? 8 : rem >= 4 ? 4 : rem >= 2 ? 2 : 1;                     \
      int lg = 0;                                                                       \
      while (lg < 3 && (P << (lg + 1)) <= rem) ++lg;                                    \
      const int w0 = t0 - c0;                                                           \
      if (P == 8) AS(name, lanes, 8);                                                   \
      else if (P == 4) AS(name, lanes, 4);                                              \
      else if (P == 2) AS(name, lanes, 2);                                              \
      else AS(name, lanes, 1);                                                          \
      t0 += P << lg;                                                                    \
    }                                                                                   \
  } while (0)
#define FCT_STAGE(name, lanes) FCT_SPLIT(FCT_STAGE_AS, name, lanes)
// a stage whose threads walk its lanes
#define FCT_WALK_AS(name, lanes, P)                                                     \
  name##_1<P><<<dim3(unsigned(std::min<int64_t>(xblocks(lanes), 148 * kWalkBlocks<P>)),  \
                     1u << lg), B, 0, s>>>(single, t0, w0)

// the fused step's edge stage beside its LO stage when the caller provides a fork
constexpr bool kForkEdge = true;

int fork_create(Fork& f) {
  FCT_CUDA(cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking));
  for (auto& e : f.ev) FCT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return FCT_OK;
}

void fork_destroy(Fork& f) {
  if (f.side) {
    cudaStreamSynchronize(f.side);
    cudaStreamDestroy(f.side);
  }
  for (auto& e : f.ev)
    if (e) cudaEventDestroy(e);
  f = Fork{};
}

namespace {

using ColKernel1 = void (*)(Inst, int, int);
using ColKernelN = void (*)(const Inst*, int, int);
struct ColKernels {
  ColKernel1 one[kColMaxTracers];
  ColKernelN many[kColMaxTracers];
};
#define FCT_COL_TABLE(name)                                                              \
  ColKernels{{name##_1<1>, name##_1<2>, name##_1<3>, name##_1<4>, name##_1<5>, name##_1<6>, \
              name##_1<7>, name##_1<8>},                                                 \
             {name##_n<1>, name##_n<2>, name##_n<3>, name##_n<4>, name##_n<5>, name##_n<6>, \
              name##_n<7>, name##_n<8>}}

// One column solve over the tracers [t0, t0 + nt): launches of up to kColMaxTracers tracers,
// which share a block's matrix rows.
int launch_columns(const ColKernels& K, const Inst& single, const Inst* tab, int n, int64_t nodes,
                   int L, int t0, int nt, cudaStream_t s, const char* what) {
  for (int t = t0; t < t0 + nt;) {
    const int g = std::min(t0 + nt - t, kColMaxTracers);
    const int columns = col_columns(L, g);
    const size_t sh = col_smem(columns, L, g);
    cudaError_t e = cudaSuccess;
    // the opt-in limit is the same value every time, so concurrent callers do not disturb it
    if (sh > size_t(48) << 10)
      e = tab ? cudaFuncSetAttribute(K.many[g - 1], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kColMaxSmem)
              : cudaFuncSetAttribute(K.one[g - 1], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kColMaxSmem);
    if (e != cudaSuccess) return cuda_error(e, what);
    const dim3 grid(unsigned(std::max<int64_t>(1, (nodes + columns - 1) / columns)),
                    tab ? unsigned(n) : 1u);
    if (tab) K.many[g - 1]<<<grid, kColThreads, sh, s>>>(tab, columns, t);
    else K.one[g - 1]<<<grid, kColThreads, sh, s>>>(single, columns, t);
    t += g;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, what);
}

}  // namespace

int launch_forward_events(const Inst& single, const Inst* tab, int n, const LaunchDims& d,
                          cudaStream_t s, cudaEvent_t* after, bool stop_before_final,
                          int chunk_sel) {
  constexpr int B = 256;
  auto xblocks = [&](int64_t lanes) {
    return unsigned(std::max<int64_t>(1, (lanes + B - 1) / B));
  };
  auto grid = [&](int64_t lanes) { return dim3(xblocks(lanes), unsigned(n), 1); };
  if (tab && !d.fused)   // (their kernels read ``single``)
    return set_error(FCT_ERR_INVALID, "the stage-by-stage kernels take one instance");
  const int chunk = d.chunk > 0 ? d.chunk : d.ntr;
  const int nchunks = (d.ntr + chunk - 1) / chunk;
  // the dry-level copy on the side stream, beside the stages (190 of 9,200 us of a step of
  // 300,000 nodes x 70 levels x 4 tracers when it ran after them)
  const bool dry_early = d.fused && !after && d.copy_dry && !stop_before_final &&
                         !d.any_vdiff && chunk_sel < 0;
  const bool dry_first = dry_early && !tab && seg_first_fits(d, 0, std::min(chunk, d.ntr));
  const bool dry_aside = dry_early && !dry_first && kForkEdge && d.fork;
  for (int ci = 0; ci < nchunks; ++ci) {
    if (chunk_sel >= 0 && ci != chunk_sel) continue;
    const int c0 = ci * chunk, c1 = std::min(d.ntr, c0 + chunk);
    int stage = 0;
    auto mark = [&]() {
      if (after) cudaEventRecord(after[stage], s);
      ++stage;
    };
    if (ci == 0) {   // the volume flux is shared by all tracers
      if (tab && d.any_derive_w && !d.skip_vflux) {   // producer: w_e from continuity, in the same graph
        const int st = launch_compute_w_tab(tab, n, d.max_nodes, s);
        if (st) return st;
      }
      if (!d.skip_vflux) {
        const dim3 g = stream_grid(xblocks(d.max_edge), int64_t(148) * kVfluxBlocks, n);
        if (tab) k_vflux_n<<<g, B, 0, s>>>(tab, n);
        else k_vflux_1<<<g, B, 0, s>>>(single);
      }
    }
    mark();
    if (d.fused) {
      // segment kernels (fct_seg_*.cu), 5 launches per chunk; the stages folded into
      // others record empty intervals (elem_grad: the node gradients are evaluated only
      // where MFCT needs them, in the edge stage; elem_bounds and node_cluster: the factors
      // stage). With a fork (and no stage timing) the edge stage runs on the side stream
      // beside the LO stage and the limiter waits for both.
      // A small single instance takes all of these in one launch (launch_seg_first).
      const bool first = !tab && !after && seg_first_fits(d, c0, c1);
      const Fork* fk = (kForkEdge && d.fork && !after && !first) ? d.fork : nullptr;
      mark();
      int st;
      if (first) {
        if ((st = launch_seg_first(single, d, c0, c1, dry_first && ci == 0, s))) return st;
      }
      if (fk) {
        FCT_CUDA(cudaEventRecord(fk->ev[0], s));
        FCT_CUDA(cudaStreamWaitEvent(fk->side, fk->ev[0], 0));
        if ((st = launch_seg_edge(single, tab, n, d, c0, c1, fk->side))) return st;
        if ((st = launch_edge_fix(single, tab, n, d, c0, c1, fk->side))) return st;
        FCT_CUDA(cudaEventRecord(fk->ev[1], fk->side));
        if (dry_aside && ci == 0) {   // reads T's, writes T_new's dry levels: no stage does
          if (tab) k_copy_dry_n<<<grid(d.max_dry), B, 0, fk->side>>>(tab);
          else k_copy_dry_1<<<grid(d.max_dry), B, 0, fk->side>>>(single);
          FCT_CUDA(cudaEventRecord(fk->ev[2], fk->side));
        }
      }
      if (!first && (st = launch_seg_lo(single, tab, n, d, c0, c1, s))) return st;
      mark();
      if (d.any_wi && (st = launch_columns(FCT_COL_TABLE(k_vert_impl), single, tab, n,
                                           d.max_nodes, d.max_levels, 0, c1 - c0, s,
                                           "split vertical velocity launch")))
        return st;
      mark();
      if (fk) {
        FCT_CUDA(cudaStreamWaitEvent(s, fk->ev[1], 0));
      } else if (!first) {
        if ((st = launch_seg_edge(single, tab, n, d, c0, c1, s))) return st;
        if ((st = launch_edge_fix(single, tab, n, d, c0, c1, s))) return st;
      }
      mark();
      mark();
      mark();
      if ((st = launch_seg_limit(single, tab, n, d, c0, c1, s))) return st;
      mark();
      if (stop_before_final) continue;
      if ((st = launch_seg_final(single, tab, n, d, c0, c1, s))) return st;
      if (d.any_vdiff) {   // epilogue: implicit vertical diffusion of this chunk, in place
        if (d.copy_dry) {  // the dry levels of T_new must hold T before it runs
          if (tab) k_copy_dry_n<<<grid(d.max_dry), B, 0, s>>>(tab);
          else k_copy_dry_1<<<grid(d.max_dry), B, 0, s>>>(single);
        }
        // eight aligned tracers of many columns walk them from memory (pair_vdiff)
        if (tab && seg_even(d) && c1 - c0 == kPairTracers && n * d.max_nodes >= kPairColumns)
          k_vdiff_pairs_n<<<grid(d.max_nodes * (kPairTracers / 2)), B, 0, s>>>(tab, c0);
        else if ((st = launch_columns(FCT_COL_TABLE(k_vdiff), single, tab, n, d.max_nodes,
                                      d.max_levels, c0, c1 - c0, s, "vertical diffusion launch")))
          return st;
      }
      mark();
      continue;
    }
    FCT_STAGE(k_elem_grad, d.max_elem);
    mark();
    FCT_STAGE(k_node_lo, d.max_iface);
    mark();
    if (d.any_wi) {
      const int st = launch_columns(FCT_COL_TABLE(k_vert_impl), single, tab, n, d.max_nodes,
                                    d.max_levels, 0, c1 - c0, s,
                                    "split vertical velocity launch");
      if (st) return st;
    }
    mark();
    FCT_SPLIT(FCT_WALK_AS, k_edge_adf, d.max_edge);
    mark();
    FCT_STAGE(k_elem_bounds, d.max_elem);
    mark();
    FCT_STAGE(k_node_cluster, d.max_layer);
    mark();
    FCT_STAGE(k_node_factors, d.max_layer);
    mark();
    if (stop_before_final) continue;
    FCT_STAGE(k_node_final, d.max_layer);
    mark();
  }
  if (dry_aside) {
    FCT_CUDA(cudaStreamWaitEvent(s, d.fork->ev[2], 0));
  } else if (!dry_first && d.copy_dry && !stop_before_final && (chunk_sel < 0 || chunk_sel == nchunks - 1)) {
    if (tab) k_copy_dry_n<<<grid(d.max_dry), B, 0, s>>>(tab);
    else k_copy_dry_1<<<grid(d.max_dry), B, 0, s>>>(single);
  }
  if (after) cudaEventRecord(after[kNumStages - 1], s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "forward kernel launch");
  return FCT_OK;
}

int launch_forward(const Inst& single, const Inst* tab, int n, const LaunchDims& d,
                   cudaStream_t s) {
  return launch_forward_events(single, tab, n, d, s, nullptr, false, -1);
}

int launch_forward_stages(const Inst& single, const LaunchDims& d, cudaStream_t s,
                          bool through_factors) {
  return launch_forward_events(single, nullptr, 1, d, s, nullptr, through_factors, -1);
}

int launch_vdiff(const Inst& single, const LaunchDims& d, cudaStream_t s) {
  return launch_columns(FCT_COL_TABLE(k_vdiff), single, nullptr, 1, d.max_nodes, d.max_levels, 0,
                        d.ntr, s, "vertical diffusion launch");
}

int launch_copy_dry(const Inst* tab, int n, int64_t max_dry, cudaStream_t s) {
  const dim3 g(unsigned(std::max<int64_t>(1, (max_dry + 255) / 256)), unsigned(n), 1);
  k_copy_dry_n<<<g, 256, 0, s>>>(tab);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCT_OK : cuda_error(e, "copy_dry launch");
}

}  // namespace fct
