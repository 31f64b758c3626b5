// The stream's serial chains with two Runge-Kutta stages per round. The force
// depends on the position alone, so stage i + 1's position does not depend on
// stage i's gradient (integrate_team.cuh), nor, in the reverse sweep, stage i's
// cotangent on stage i + 1's (in Nystrom form, nystrom.cuh, abar has no entries
// next to its diagonal): one part of the lanes holds one stage of a pair and
// another the next, and a step takes seven rounds of evaluations instead of
// thirteen (Dopri8) or four instead of seven (Dopri5).
// Included by stream.cu, after its argument struct.
#pragma once

#include "integrate_team.cuh"
#include "nystrom.cuh"

namespace gal {

// ------------------------------------------------------------------ forward
// The Milky Way on a four-warp team (TeamMW's division of the gradient).
struct StreamTeamMW {
  struct Shared {
    TeamShared t;
    TeamMW::Shared m;
  };
  const MWParams& p;
  Shared& sh;

  // Gradient component of warp w < 3 at its position component x.
  __device__ __forceinline__ double grad(int warp, int lane, double x, int) const {
    if (warp < 3) sh.t.pos[warp][lane] = x;
    __syncthreads();  // positions written
    const double X = sh.t.pos[0][lane], Y = sh.t.pos[1][lane], Z = sh.t.pos[2][lane];
    if (warp == 3) {
      const MWDisk d = mw_disk(p, X, Y, Z);
      sh.m.u[lane] = d.u;
      sh.m.us[lane] = d.us;
      sh.m.izb[lane] = d.izb;
    } else if (warp == 0) {
      double r;
      const double ir = mw_ir(X, Y, Z, r);
      const MWRecip c = mw_recip(p, r);
      sh.m.B[lane] = fma(p.Gm_b, c.inv_db2, p.Gm_n * c.inv_dn2);
      sh.m.inv_dh[lane] = c.inv_dh;
      sh.m.ir[lane] = ir;
    } else if (warp == 1) {
      double r;
      mw_ir(X, Y, Z, r);
      sh.m.L[lane] = mw_halo_log(p, r);
    } else {
      double r;
      const double ir = mw_ir(X, Y, Z, r);
      sh.m.A[lane] = p.Gm_h * (ir * ir);
    }
    __syncthreads();  // pieces written
    if (warp > 2) return 0.0;
    const double ir = sh.m.ir[lane];
    const double f = fma(ir, sh.m.B[lane], sh.m.A[lane] * fma(sh.m.L[lane], ir, -sh.m.inv_dh[lane]));
    return warp < 2 ? (sh.m.u[lane] + f) * x : fma(sh.m.us[lane], sh.m.izb[lane], f) * x;
  }
};

// Host components and the progenitor's Plummer sphere at its stage positions Q
// ([S][3]), summed as pfield does: component c on warp c % 4, the sphere on warp 3,
// the four partial sums in warp order.
struct StreamTeamTable {
  struct Shared {
    double pos[3][32], g[4][3][32];
  };
  const DevComp* comps;
  int ncomp;
  double GMp, b2;
  Shared& sh;
  const double* Q;

  __device__ __forceinline__ double grad(int warp, int lane, double x, int stage) const {
    if (warp < 3) sh.pos[warp][lane] = x;
    double q[3] = {0.0, 0.0, 0.0};
    if (warp == 3) {
#pragma unroll
      for (int j = 0; j < 3; ++j) q[j] = Q[3 * stage + j];
    }
    __syncthreads();  // positions written
    const double x0 = sh.pos[0][lane], x1 = sh.pos[1][lane], x2 = sh.pos[2][lane];
    double gx = 0.0, gy = 0.0, gz = 0.0;
    for (int c = warp; c < ncomp; c += 4) comp_grad(comps[c], x0, x1, x2, gx, gy, gz);
    if (warp == 3) {
      const double d0 = x0 - q[0], d1 = x1 - q[1], d2 = x2 - q[2];
      const double r2 = fma(d0, d0, fma(d1, d1, fma(d2, d2, TINY)));
      const double is = rsqrt(r2 + b2);
      const double f = GMp * (is * is) * is;
      gx = fma(f, d0, gx);
      gy = fma(f, d1, gy);
      gz = fma(f, d2, gz);
    }
    sh.g[warp][0][lane] = gx;
    sh.g[warp][1][lane] = gy;
    sh.g[warp][2][lane] = gz;
    __syncthreads();  // partial gradients written
    if (warp > 2) return 0.0;
    return ((sh.g[0][warp][lane] + sh.g[1][warp][lane]) + sh.g[2][warp][lane]) + sh.g[3][warp][lane];
  }
};

// One constant step of signed length h for the warp's component (x, v) of the
// orbit in this lane's slot, in the usual Runge-Kutta form (the operations of the
// one-thread step, in its order: a progenitor's first particles follow it so
// closely that a change of rounding in these grows a millionfold).
// record(i, X) gets every stage position component (owners, one half each).
template <class TB, class Team, class Record>
__device__ __forceinline__ void stream_pair_step(const Team& team, int warp, int lane, double h, double& x, double& v,
                                                 Record&& record) {
  constexpr int S = TB::S;
  const bool hi = lane >= 16, own = warp < 3;
  double Fp[S], Fv[S];
  if (own && !hi) record(0, x);
  Fp[0] = v;
  Fv[0] = -team.grad(warp, lane, x, 0);
  static_for<0, (S - 1) / 2>([&](auto r) {
    constexpr int I = 2 * decltype(r)::value + 1;  // stages I (lanes 0-15) and I + 1 (lanes 16-31)
    double X = 0.0;
    if (own) {
      if constexpr (I == 1) {
        Fp[1] = pair_row<TB, 1, 1>(hi, v, h, Fv);
      } else {
        const double V = pair_row<TB, I - 1, I>(hi, v, h, Fv);
        const double W = __shfl_xor_sync(0xffffffffu, V, 16);
        Fp[I - 1] = hi ? W : V;
        Fp[I] = hi ? V : W;
      }
      X = pair_row<TB, I, I + 1>(hi, x, h, Fp);
      record(hi ? I + 1 : I, X);
    }
    const double f = -team.grad(warp, lane, X, hi ? I + 1 : I);
    const double o = __shfl_xor_sync(0xffffffffu, f, 16);
    Fv[I] = hi ? o : f;
    Fv[I + 1] = hi ? f : o;
  });
  if (own) {
    Fp[S - 1] = pair_row<TB, S - 1, S - 1>(hi, v, h, Fv);
    x = weighted_comp<TB, W_SOLUTION, true>(x, h, Fp);
    v = weighted_comp<TB, W_SOLUTION, true>(v, h, Fv);
  }
}

// The progenitor in a Milky Way host: one orbit, the same in every slot. 14 us
// instead of 26 per Dopri8 step.
template <class TB>
__global__ void __launch_bounds__(128) k_stream_progenitor_mw(StreamDev a, MWParams p) {
  constexpr int S = TB::S;
  __shared__ StreamTeamMW::Shared sh;
  const StreamTeamMW team{p, sh};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = warp < 3 ? warp : 0;
  const bool writes = warp < 3 && (lane & 15) == 0;
  double x = a.w_now[j], v = a.w_now[3 + j];
  auto track = [&](double h, double* Q, double* out) {
    if (writes && lane == 0) {
      out[j] = x;
      out[3 + j] = v;
    }
    for (int64_t k = 0; k < a.n_rel; ++k) {
      stream_pair_step<TB>(team, warp, lane, h, x, v, [&](int i, double X) {
        if (Q && writes) Q[(k * S + i) * 3 + j] = X;
      });
      if (writes && lane == 0) {
        out[(k + 1) * 6 + j] = x;
        out[(k + 1) * 6 + 3 + j] = v;
      }
    }
  };
  track(-a.dt, a.Qb, a.B);
  track(a.dt, a.Q, a.P);
}

// Particles, 16 per team. A lane joins when the global step reaches its release
// step. Writes the final states and either the checkpoints or the stored stage
// positions.
template <class TB>
__global__ void __launch_bounds__(128) k_stream_particles_team(StreamDev a, const DevComp* comps) {
  constexpr int S = TB::S;
  __shared__ DevComp s_comps[kAdjMaxComps];
  __shared__ StreamTeamTable::Shared sh;
  stage_comps(comps, a.ncomp, s_comps);
  StreamTeamTable team{s_comps, a.ncomp, a.GMp, a.b2, sh, nullptr};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t first = (int64_t)blockIdx.x * 16, q = first + (lane & 15), n = a.np;
  const bool valid = q < n, own = warp < 3, lo = lane < 16;
  const int j = own ? warp : 0;
  const int64_t rp = valid ? (q >> 1) : LLONG_MAX;
  const int K = a.k_ckpt;
  // lanes past the last particle follow a circular-ish orbit at 8 kpc
  double x = valid ? a.ics[j * n + q] : (j == 0 ? 8.0 : 0.0);
  double v = valid ? a.ics[(3 + j) * n + q] : (j == 1 ? 0.2 : 0.0);
  for (int64_t k = first >> 1; k < a.n_rel; ++k) {
    const bool act = valid && k >= rp;
    if (own && lo && act && a.ckpt && (k == rp || k % K == 0)) {
      const int64_t c = k / K;
      a.ckpt[(c * 6 + j) * n + q] = x;
      a.ckpt[(c * 6 + 3 + j) * n + q] = v;
    }
    double x1 = x, v1 = v;
    team.Q = a.Q + k * S * 3;
    stream_pair_step<TB>(team, warp, lane, a.dt, x1, v1, [&](int i, double X) {
      if (a.Ys && act) a.Ys[stage_idx(k, i, j, q, S, 3)] = X;
    });
    if (act) {
      x = x1;
      v = v1;
    }
  }
  if (own && lo && valid) {
    a.fin[j * n + q] = x;
    a.fin[(3 + j) * n + q] = v;
  }
}

// ------------------------------------------------------------------ reverse
// With L = h lx, and v_i = h G_i the cotangent that stage i's gradient gets,
//   G_i = bbar_i L + b_i lv + sum_{l>i} abar_li E_l,   E_i = h (mu_i - H_i v_i),
//   L += sum_i E_i,   lv += L + sum_i c_i E_i   (the old L),
// mu_i a cotangent that the stage position has from elsewhere. Six lanes per
// orbit: lane 3 s + j holds component j of the pair's stages S-1-2r (s = 0) and
// S-2-2r (s = 1); the last round has stage 0 alone.
template <class TB>
struct PairSweep {
  static constexpr int S = TB::S, R = (S + 1) / 2;
  double H[R][3];  // entries (j, j), (j, j+1), (j, j+2) of the lane's stage's Hessian, indices mod 3
  double mu[R];

  // This lane's stage in round r.
  static __device__ __forceinline__ int stage(int r, bool hi) { return r == R - 1 ? 0 : S - 1 - 2 * r - (hi ? 1 : 0); }

  template <class PutV>
  __device__ __forceinline__ void step(int base, int j, bool hi, double h, double& L, double& lv, PutV&& put_v) const {
    const int row = base + (hi ? 3 : 0);
    const int s1 = row + (j + 1) % 3, s2 = row + (j + 2) % 3, so = base + (hi ? 0 : 3) + j;
    double E[S];
    static_for<0, R>([&](auto r) {
      constexpr int sa = S - 1 - 2 * decltype(r)::value, sb = sa > 0 ? sa - 1 : 0;
      constexpr double xa = kNystrom<TB>.b[sa], xb = kNystrom<TB>.b[sb], va = TB::B[sa], vb = TB::B[sb];
      double G = 0.0;
      if constexpr (va != 0.0 || vb != 0.0) G = (hi ? vb : va) * lv;
      if constexpr (xa != 0.0 || xb != 0.0) G = fma(hi ? xb : xa, L, G);
      static_for<sb + 1, S>([&](auto l) {
        constexpr int Q = decltype(l)::value;
        constexpr double ca = Q > sa ? kNystrom<TB>.a[Q][sa] : 0.0;
        constexpr double cb = Q > sa ? kNystrom<TB>.a[Q][sb] : 0.0;  // abar[sa][sb] = 0: the pair is independent
        if constexpr (ca != 0.0 || cb != 0.0) G = fma(hi ? cb : ca, E[Q], G);
      });
      const double v = h * G;
      put_v(decltype(r)::value, v);
      const double v1 = __shfl_sync(0xffffffffu, v, s1), v2 = __shfl_sync(0xffffffffu, v, s2);
      const int q = decltype(r)::value;
      const double e = h * (mu[q] - fma(H[q][0], v, fma(H[q][1], v1, H[q][2] * v2)));
      const double o = __shfl_sync(0xffffffffu, e, so);
      E[sa] = hi ? o : e;
      if constexpr (sa > 0) E[sb] = hi ? e : o;
      else E[0] = e;
    });
    double sum = 0.0, csum = L;
    static_for<0, S>([&](auto i) {
      constexpr int I = decltype(i)::value;
      constexpr double c = TB::C[I];
      if constexpr (kNystrom<TB>.used[I]) {
        sum += E[I];
        if constexpr (c != 0.0) csum = fma(c, E[I], csum);
      }
    });
    L += sum;
    lv += csum;
  }
};

// Index of the symmetric entry (a, b) in xx xy xz yy yz zz.
__device__ __forceinline__ int sym_index(int a, int b) {
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  return lo == 0 ? hi : lo + hi + 1;
}

constexpr int kSweepParticles = 5;  // particles per warp

// Reverse sweep with the stored Hessians, five particles per warp; the next
// step's Hessian rows are loaded a step ahead. 5 us instead of 41 per Dopri8 step.
template <class TB>
__global__ void __launch_bounds__(32) k_stream_particles_sweep(StreamDev a) {
  constexpr int S = TB::S, R = PairSweep<TB>::R;
  const int lane = threadIdx.x;
  const int slot = lane < 30 ? lane / 6 : 4, part = lane < 30 ? lane % 6 : lane - 24 - 6 * ((lane - 24) / 6);
  const int base = 6 * slot, j = part % 3;
  const bool hi = part >= 3;
  const int64_t first = (int64_t)blockIdx.x * kSweepParticles, n = a.np;
  const int64_t p = first + slot;
  const bool valid = lane < 30 && p < n;
  const int64_t rp = valid ? (p >> 1) : LLONG_MAX;
  const int64_t rmin = first >> 1;
  const double h = a.dt;
  const int e0 = sym_index(j, j), e1 = sym_index(j, (j + 1) % 3), e2 = sym_index(j, (j + 2) % 3);
  double L = 0.0, lv = 0.0;
  if (valid) {
    L = h * (2.0 * (a.fin[j * n + p] - a.target[j * n + p]));
    lv = 2.0 * (a.fin[(3 + j) * n + p] - a.target[(3 + j) * n + p]);
  }
  PairSweep<TB> cur, next;
  auto load = [&](int64_t k, PairSweep<TB>& w) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = PairSweep<TB>::stage(r, hi);
      const bool act = valid && k >= rp;
      w.H[r][0] = act ? a.Hs[stage_idx(k, i, e0, p, S, 6)] : 0.0;
      w.H[r][1] = act ? a.Hs[stage_idx(k, i, e1, p, S, 6)] : 0.0;
      w.H[r][2] = act ? a.Hs[stage_idx(k, i, e2, p, S, 6)] : 0.0;
      w.mu[r] = 0.0;
    }
  };
  load(a.n_rel - 1, next);
  for (int64_t k = a.n_rel - 1; k >= rmin; --k) {
    const bool act = valid && k >= rp;
    cur = next;
    if (k > rmin) load(k - 1, next);
    double L1 = L, lv1 = lv;
    cur.step(base, j, hi, h, L1, lv1, [&](int r, double v) {
      if (act && (!hi || r < R - 1)) a.vs[stage_idx(k, PairSweep<TB>::stage(r, hi), j, p, S, 3)] = v;
    });
    if (act) {
      L = L1;
      lv = lv1;
    }
    if (k == rp && !hi) {
      a.lam_rel[j * n + p] = L / h;
      a.lam_rel[(3 + j) * n + p] = lv;
    }
  }
  if (valid && part == 0) {
    double loss = 0.0;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const double d = a.fin[c * n + p] - a.target[c * n + p];
      loss = fma(d, d, loss);
    }
    for (int c = 0; c < 3 * a.ncomp; ++c) a.gp_all[(int64_t)c * a.ncol + p] = 0.0;
    a.gp_all[(int64_t)(3 * a.ncomp) * a.ncol + p] = loss;
  }
}

// Cotangent on the progenitor's stage positions, sum over particles of H_prog v:
// one warp per stage point, particles in a fixed order. Off the serial sweep,
// which summed these over each warp's lanes at every stage.
__global__ void __launch_bounds__(128) k_stream_mu(StreamDev a, int S) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (w >= a.n_rel * S) return;
  const int64_t k = w / S;
  const int i = (int)(w % S);
  const double* Qi = a.Q + 3 * w;
  const double q[3] = {Qi[0], Qi[1], Qi[2]};
  double m[3] = {0.0, 0.0, 0.0};
  for (int64_t p = lane; p < 2 * (k + 1); p += 32) {
    double d[3], v[3], Hv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      d[c] = a.Ys[stage_idx(k, i, c, p, S, 3)] - q[c];
      v[c] = a.vs[stage_idx(k, i, c, p, S, 3)];
    }
    plummer_hv(a.GMp, a.b2, d, v, Hv);
#pragma unroll
    for (int c = 0; c < 3; ++c) m[c] += Hv[c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double t = warp_sum(m[c]);
    if (lane == 0) a.mu[3 * w + c] = t;
  }
}

// The progenitor's reverse recurrence, forwards track (particles' cotangents mu
// on the stage positions, release-map cotangents nu on the grid states), then
// backwards track.
template <class TB>
__global__ void __launch_bounds__(32) k_stream_prog_sweep(StreamDev a) {
  constexpr int S = TB::S, R = PairSweep<TB>::R;
  const int lane = threadIdx.x, part = lane % 6, j = part % 3;
  const bool hi = part >= 3, writes = lane < 6;
  const int e0 = sym_index(j, j), e1 = sym_index(j, (j + 1) % 3), e2 = sym_index(j, (j + 2) % 3);
  double L = 0.0, lv = 0.0;
  for (int track = 0; track < 2; ++track) {
    const double h = track == 0 ? a.dt : -a.dt;
    if (track == 1) L = -L;  // L = h lx
    const int64_t off = (int64_t)track * a.n_rel * S;
    PairSweep<TB> cur, next;
    double nux = 0.0, nuv = 0.0, nux1 = 0.0, nuv1 = 0.0;
    auto load = [&](int64_t k, PairSweep<TB>& w, double& x, double& v) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int64_t i = k * S + PairSweep<TB>::stage(r, hi);
        const double* Hp = a.Hst + 6 * (off + i);
        w.H[r][0] = Hp[e0];
        w.H[r][1] = Hp[e1];
        w.H[r][2] = Hp[e2];
        w.mu[r] = track == 0 ? a.mu[3 * i + j] : 0.0;
      }
      x = track == 0 ? a.nu[6 * k + j] : 0.0;
      v = track == 0 ? a.nu[6 * k + 3 + j] : 0.0;
    };
    load(a.n_rel - 1, next, nux1, nuv1);
    for (int64_t k = a.n_rel - 1; k >= 0; --k) {
      cur = next;
      nux = nux1;
      nuv = nuv1;
      if (k > 0) load(k - 1, next, nux1, nuv1);
      cur.step(lane - part, j, hi, h, L, lv, [&](int r, double v) {
        if (writes && (!hi || r < R - 1)) a.vst[3 * (off + k * S + PairSweep<TB>::stage(r, hi)) + j] = v;
      });
      L = fma(h, nux, L);
      lv += nuv;
    }
  }
  if (a.grad_w_now && writes && !hi) {
    a.grad_w_now[j] = L / -a.dt;
    a.grad_w_now[3 + j] = lv;
  }
}

}  // namespace gal
