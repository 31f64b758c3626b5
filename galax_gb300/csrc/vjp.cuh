// Reverse-mode pieces shared by the adjoint kernels: the Hessian-vector
// product and parameter derivatives of one component (the transposed Jacobian
// of the Hamiltonian field, f = (p, -grad Phi(q)) so J^T (u, v) = (-H(q) v, u)),
// and a plain constant-step Runge-Kutta step.
#pragma once

#include "integrate.cuh"

namespace gal {

constexpr int kAdjMaxComps = 8;

// H(x) v and d(grad Phi(x) . v)/d(m, l1, l2) of one component, accumulated.
__device__ __forceinline__ void comp_vjp(const DevComp& c, const double* x, const double* v, double* Hv,
                                         double* dp) {
  const double d0 = x[0] - c.ox, d1 = x[1] - c.oy, d2 = x[2] - c.oz;
  if (c.kind == MIYAMOTO_NAGAI) {
    const double zb2 = fma(d2, d2, c.l2sq);
    const double izb = rsqrt(zb2);
    const double zb = zb2 * izb;
    const double s = zb + c.l1;
    const double iD = rsqrt(fma(d0, d0, fma(d1, d1, s * s)));
    const double iD2 = iD * iD;
    const double u = c.Gm * iD2 * iD;
    const double w = 3.0 * u * iD2;
    const double vz = d2 * s * izb;
    const double vv = fma(d0, v[0], fma(d1, v[1], vz * v[2]));
    const double izb3 = izb * izb * izb;
    Hv[0] += fma(u, v[0], -w * vv * d0);
    Hv[1] += fma(u, v[1], -w * vv * d1);
    Hv[2] += fma(u * fma(c.l1 * c.l2sq, izb3, 1.0), v[2], -w * vv * vz);
    dp[0] += u * vv * c.inv_m;
    dp[1] += fma(-w * s, vv, u * d2 * izb * v[2]);
    dp[2] += fma(-w * s * c.l2 * izb, vv, -u * c.l1 * c.l2 * d2 * izb3 * v[2]);
    return;
  }
  const double r2 = fma(d0, d0, fma(d1, d1, fma(d2, d2, TINY)));
  const double ir = rsqrt(r2);
  const double ir2 = ir * ir;
  const double r = r2 * ir;
  const double xv = fma(d0, v[0], fma(d1, v[1], d2 * v[2]));
  double g, gpr, dl1 = 0.0, dl2 = 0.0;
  switch (c.kind) {
    case KEPLER:
      g = c.Gm * ir2 * ir;
      gpr = -3.0 * g * ir2;
      break;
    case HERNQUIST: {
      const double dd = r + c.l1, idd = 1.0 / dd;
      g = c.Gm * ir * idd * idd;
      gpr = -c.Gm * (3.0 * r + c.l1) * ir2 * ir * idd * idd * idd;
      dl1 = -2.0 * g * idd * xv;
      break;
    }
    case NFW: {
      const double L = log1p_pos(r * c.inv_l1), q = c.l1 + r, iq = 1.0 / q;
      g = c.Gm * ir2 * fma(L, ir, -iq);
      gpr = c.Gm * ir2 * ir * (3.0 * ir * iq - 3.0 * L * ir2 + iq * iq);
      dl1 = -c.Gm * ir * c.inv_l1 * iq * iq * xv;
      break;
    }
    case ISOCHRONE: {  // g = G m / ((b + s)^2 s); dg/db = -g (2 (1 + b/s) / (b + s) + b / s^2)
      const double s2 = r2 + c.l2sq, is = rsqrt(s2), s = s2 * is, d = c.l1 + s, id = 1.0 / d;
      g = c.Gm * is * id * id;
      gpr = -g * (2.0 * id * is + is * is);
      dl1 = -g * fma(2.0 * id, fma(c.l1, is, 1.0), c.l1 * is * is) * xv;
      break;
    }
    case LOGARITHMIC: {  // g = v^2 / (r_s^2 + r^2); dg/dr_s = -2 r_s g / q
      const double iq = 1.0 / (r2 + c.l2sq);
      g = c.Gm * iq;
      gpr = -2.0 * g * iq;
      dl1 = -2.0 * c.l1 * g * iq * xv;
      break;
    }
    case POWERLAW_CUTOFF: {
      const PlcG t = plc_g(c, r2, ir, true, true);
      g = t.g;
      gpr = t.gpr;
      dl1 = t.dg_drc * xv;
      dl2 = t.dg_dalpha * xv;
      break;
    }
    default: {  // PLUMMER
      const double is = rsqrt(r2 + c.l2sq), is2 = is * is;
      g = c.Gm * is2 * is;
      gpr = -3.0 * g * is2;
      dl1 = -3.0 * g * is2 * c.l1 * xv;
      break;
    }
  }
  Hv[0] += fma(g, v[0], gpr * xv * d0);
  Hv[1] += fma(g, v[1], gpr * xv * d1);
  Hv[2] += fma(g, v[2], gpr * xv * d2);
  dp[0] += g * xv * c.inv_m;
  dp[1] += dl1;
  dp[2] += dl2;
}

// ---- the Milky Way's four components together
// Gradient at X; q: ir, L, 1/(r + r_s) of halo, bulge, nucleus, 1/sqrt(z^2 + b^2), 1/D.
__device__ __forceinline__ void mw_stage(const MWParams& p, const double* X, double* q, double* g) {
  double r;
  const double ir = mw_ir(X[0], X[1], X[2], r);
  const double dh = p.rs_h + r, db = r + p.rs_b, dn = r + p.rs_n;
  const double bn = db * dn;
  const double iP = 1.0 / (dh * bn);
  const double ih = iP * dh;
  const double idh = iP * bn, idb = ih * dn, idn = ih * db;
  const double L = mw_halo_log(p, r);
  const double zb2 = fma(X[2], X[2], p.b2_d);
  const double izb = rsqrt(zb2);
  const double s = fma(zb2, izb, p.a_d);
  const double iD = rsqrt(fma(s, s, fma(X[0], X[0], X[1] * X[1])));
  const double u = p.Gm_d * (iD * iD) * iD;
  const double f = p.Gm_h * (ir * ir) * fma(L, ir, -idh) + ir * fma(p.Gm_b, idb * idb, p.Gm_n * (idn * idn));
  g[0] = (u + f) * X[0];
  g[1] = (u + f) * X[1];
  g[2] = fma(u * s, izb, f) * X[2];
  q[0] = ir;
  q[1] = L;
  q[2] = idh;
  q[3] = idb;
  q[4] = idn;
  q[5] = izb;
  q[6] = iD;
}

// H(X) w, and the parameter sums of g . w up to constant factors (mw_param_grads):
// disk m, a, b; halo m, r_s; bulge m, r_s; nucleus m, r_s.
__device__ __forceinline__ void mw_stage_vjp(const MWParams& p, const double* X, const double* q, const double* w,
                                             double* Hw, double* gp) {
  const double ir = q[0], L = q[1], idh = q[2], idb = q[3], idn = q[4], izb = q[5], iD = q[6];
  const double xw = fma(X[0], w[0], fma(X[1], w[1], X[2] * w[2]));
  const double ir2 = ir * ir;
  const double idh2 = idh * idh;
  const double gh = p.Gm_h * ir2 * fma(L, ir, -idh);
  const double gb = p.Gm_b * ir * (idb * idb), gn = p.Gm_n * ir * (idn * idn);
  const double gpr = ir2 * fma(p.Gm_h * ir, idh2, -3.0 * gh) -
                     fma(gb, fma(2.0 * ir, idb, ir2), gn * fma(2.0 * ir, idn, ir2));
  gp[3] = fma(gh, xw, gp[3]);
  gp[4] = fma(ir * idh2, xw, gp[4]);
  const double bw = gb * xw, nw = gn * xw;
  gp[5] += bw;
  gp[6] = fma(bw, idb, gp[6]);
  gp[7] += nw;
  gp[8] = fma(nw, idn, gp[8]);
  const double iD2 = iD * iD;
  const double u = p.Gm_d * iD2 * iD;
  const double w5 = 3.0 * u * iD2;
  const double s = fma(fma(X[2], X[2], p.b2_d), izb, p.a_d);
  const double zi = X[2] * izb;
  const double vz = zi * s;
  const double vw = fma(X[0], w[0], fma(X[1], w[1], vz * w[2]));
  const double izb2 = izb * izb;
  const double t = w5 * vw, ts = t * s;
  const double uz = u * w[2], uzi = uz * zi;
  gp[0] = fma(u, vw, gp[0]);
  gp[1] += uzi - ts;
  gp[2] -= fma(ts, izb, p.a_d * uzi * izb2);
  const double d = u + (gh + (gb + gn));
  const double k = fma(gpr, xw, -t);
  Hw[0] = fma(d, w[0], k * X[0]);
  Hw[1] = fma(d, w[1], k * X[1]);
  Hw[2] = fma(d, w[2], fma(gpr * xw, X[2], fma(-t, vz, p.a_d * p.b2_d * (izb2 * izb) * uz)));
}

// d/d(m, l1, l2) of the four components from the sums of mw_stage_vjp.
__device__ __forceinline__ void mw_param_grads(const MWParams& p, const DevComp* comps, const double* gp, double* out) {
  out[0] = gp[0] * comps[0].inv_m;
  out[1] = gp[1];
  out[2] = comps[0].l2 * gp[2];
  out[3] = gp[3] * comps[1].inv_m;
  out[4] = -p.Gm_h * p.irs_h * gp[4];
  out[6] = gp[5] * comps[2].inv_m;
  out[7] = -2.0 * gp[6];
  out[9] = gp[7] * comps[3].inv_m;
  out[10] = -2.0 * gp[8];
  out[5] = out[8] = out[11] = 0.0;
}

// One constant step of signed length hs from time t (static models ignore t).
template <class TB, class Pot>
__device__ __forceinline__ void rk_step_plain(const Pot& pot, double* y, double hs, double t = 0.0) {
  double F[TB::S][6], y1[6];
  field(pot, y, F[0], t);
  rk_stages<TB>(pot, y, hs, F, t);
  rk_combine<TB>(y, hs, F, y1, nullptr);
#pragma unroll
  for (int j = 0; j < 6; ++j) y[j] = y1[j];
}

}  // namespace gal
