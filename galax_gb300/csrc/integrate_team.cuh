// Four-warp teams with paired stages: the latency-optimal arrangement for few
// or long orbits.
//
// A lone orbit is bound by its chain of FP64 instructions: a GB300 FP64 warp
// instruction holds its sub-partition's FP64 pipe for 64 cycles (76 with all
// four pipes busy) however few lanes are active. A team block (4 warps, one per
// sub-partition) integrates 16 orbits and shortens the chain twice.
//
// Two stages per round. The force depends on the position alone, so with
// F_i = (V_i, -g(X_i)), V_i = v + hs sum_{l<i} a_il (-g_l) and
// X_i = x + hs sum_{l<i} a_il V_l, the position X_{i+1} needs the velocity V_i
// and with it only the gradients up to g_{i-1}: gradients i and i + 1 do not
// depend on one another. The stages are taken in pairs (1,2), (3,4), ...: lanes
// 0-15 hold stage i of the block's 16 orbits and lanes 16-31 stage i + 1, and
// one pass of the gradient code serves both. Dopri5 takes 3 rounds a step
// instead of 6, Dopri8 6 (and one for the next step's first slope) instead of 13.
//
// Four warps per gradient. In the Milky Way model (a table's components are
// shared out likewise):
//   warp 0: the spheres' radius, the shared reciprocal, the bulge and nucleus;
//   warp 1: the radius and the NFW halo's log(1 + r / r_s) (mw_halo_log);
//   warp 2: the radius and the halo's factor;
//   warp 3: the Miyamoto-Nagai disk (mw_disk);
// warps 0-2 own state components (w, w + 3), form their stage states and
// combine the pieces into their gradient component. Dopri5's step control is
// computed redundantly by all four warps from the same shared-memory values;
// Dopri8's by warp 2, while the others evaluate the slope at the step's end. Every
// operation matches the one-thread-per-orbit kernel (k_integrate_mw with
// MWPot::grad, integrate_loop), so results are bitwise identical.
//
// Measured (constant step, one block per SM): a Dopri8 step 17.3 us, where the
// one-thread kernel takes 58 us and a team of 32 orbits with one stage per round
// took about 36; a Dopri5 step 9.2 us instead of 26.
//
// Dopri5 is FSAL: a step's last stage is the next step's first slope, and its
// state is the solution. Dopri8 is not: after an accepted step the slope at the
// new state is one more round, and without a save scratch (a.defer) the saves
// inside an accepted step are written by sub-steps of the partial length (the
// orbit stays "pending" until its last save of the step), each one RK
// evaluation of its own.
#pragma once

#include <type_traits>

#include "integrate.cuh"

namespace gal {

struct TeamShared {
  // field-evaluation exchange: lane = 16 * (stage of the pair) + orbit
  double pos[3][32];
  // controller exchange
  double y1[6][kTeamLanes], err[6][kTeamLanes];
  double next_t1[kTeamLanes], prev_inv[kTeamLanes], prev_prev_inv[kTeamLanes];
  int flags[kTeamLanes];
  long long slot[kTeamLanes];
};

// A callable for a model's side job.
template <class Fn>
struct SideJob {
  static constexpr bool any = true;
  Fn fn;
  __device__ __forceinline__ void operator()() const { fn(); }
};
template <class Fn>
__device__ __forceinline__ SideJob<Fn> side_job(Fn fn) {
  return SideJob<Fn>{fn};
}

// Y_j = y_j + hs sum_{l<I} A[I][l] F_l,j for one component (stage_state's
// arithmetic): row IA on lanes 0-15, row IB on lanes 16-31. Zero coefficients
// add nothing, as in stage_state, where their terms do not exist.
template <class TB, int IA, int IB>
__device__ __forceinline__ double pair_row(bool hi, double yj, double hs, const double (&Fj)[TB::S]) {
  static_assert(TB::A[IA][0] != 0.0 && TB::A[IB][0] != 0.0, "rows start with their first slope");
  constexpr double a0 = TB::A[IA][0], b0 = TB::A[IB][0];
  double acc = (hi ? b0 : a0) * Fj[0];
  static_for<1, (IA > IB ? IA : IB)>([&](auto l) {
    constexpr int L = decltype(l)::value;
    constexpr double ca = L < IA ? TB::A[IA][L] : 0.0, cb = L < IB ? TB::A[IB][L] : 0.0;
    if constexpr (ca != 0.0 || cb != 0.0) {
      constexpr double sa = ca != 0.0 ? ca : cb, sb = cb != 0.0 ? cb : ca;
      const double t = fma(hi ? sb : sa, Fj[L], acc);
      if constexpr (ca == 0.0) acc = hi ? t : acc;
      else if constexpr (cb == 0.0) acc = hi ? acc : t;
      else acc = t;
    }
  });
  return fma(hs, acc, yj);
}

// weighted<TB, WHICH> for one component: y_j + hs sum_l w_l F_l,j, or
// hs sum_l w_l F_l,j without y.
template <class TB, int WHICH, bool WITH_Y>
__device__ __forceinline__ double weighted_comp(double yj, double hs, const double (&Fj)[TB::S]) {
  double acc = 0.0;
  bool first = true;
  static_for<0, TB::S>([&](auto l) {
    constexpr int L = decltype(l)::value;
    constexpr double c = weight<TB, WHICH, L>();
    if constexpr (c != 0.0) {
      acc = first ? c * Fj[L] : fma(c, Fj[L], acc);
      first = false;
    }
  });
  if constexpr (WITH_Y) return fma(hs, acc, yj);
  return hs * acc;
}

// dopri5_dense for one component.
__device__ __forceinline__ double dense_comp(double y0j, double hs, const double (&Fj)[Dopri5::S], double th) {
  const double t2 = th * th;
  const double u = 1.0 - th;
  const double H1 = t2 * fma(th, fma(-8.0, th, 14.0), -5.0);
  const double Hm = 16.0 * t2 * (u * u);
  const double Hf0 = th * (u * u) * fma(-2.0, th, 1.0);
  const double Hf1 = t2 * (-u) * fma(2.0, th, -1.0);
  double W[Dopri5::S];
  static_for<0, Dopri5::S>([&](auto i) {
    constexpr int I = decltype(i)::value;
    constexpr double b = Dopri5::B[I], c = Dopri5::CMID[I];
    double w = (b != 0.0) ? H1 * b : 0.0;
    if constexpr (c != 0.0) w = fma(Hm, c, w);
    if constexpr (I == 0) w += Hf0;
    if constexpr (I == Dopri5::S - 1) w += Hf1;
    W[I] = w;
  });
  double acc = W[0] * Fj[0];
  static_for<1, Dopri5::S>([&](auto i) {
    constexpr int I = decltype(i)::value;
    if constexpr (I != 1) acc = fma(W[I], Fj[I], acc);
  });
  return fma(hs, acc, y0j);
}

// Models: grad() is one round of field evaluations, a point per lane, at time t.
// The owners (warps 0-2) hold their position component q; warp w < 3 gets its
// gradient component. With a side job, warp 2 does that between the two barriers
// and the others take over its share where that is small.
struct NoSide {
  static constexpr bool any = false;
  __device__ __forceinline__ void operator()() const {}
};
//
// The Milky Way.
struct TeamMW {
  static constexpr bool TIMED = false;
  struct Shared {
    double u[32], us[32], izb[32];
    double A[32], B[32], inv_dh[32], ir[32], L[32];
  };
  const MWParams& p;
  Shared& m;

  template <class Side = NoSide>
  __device__ __forceinline__ double grad(TeamShared& sh, int warp, int lane, double q, double,
                                         Side&& side = Side{}) const {
    constexpr bool busy = std::decay_t<Side>::any;  // warp 2 has a side job: warp 3 takes its factor
    if (warp < 3) sh.pos[warp][lane] = q;
    __syncthreads();  // positions written
    const double x = sh.pos[0][lane], y = sh.pos[1][lane], z = sh.pos[2][lane];
    if (busy && warp == 2) {
      side();
    } else if (warp == 3) {
      const MWDisk d = mw_disk(p, x, y, z);
      m.u[lane] = d.u;
      m.us[lane] = d.us;
      m.izb[lane] = d.izb;
      if constexpr (busy) {
        double r;
        const double ir = mw_ir(x, y, z, r);
        m.A[lane] = p.Gm_h * (ir * ir);
        m.ir[lane] = ir;
      }
    } else {  // mw_f's products where their factors are
      double r;
      const double ir = mw_ir(x, y, z, r);
      if (warp == 0) {
        const MWRecip c = mw_recip(p, r);
        m.B[lane] = ir * fma(p.Gm_b, c.inv_db2, p.Gm_n * c.inv_dn2);
        m.inv_dh[lane] = c.inv_dh;
      } else if (warp == 1) {
        m.L[lane] = mw_halo_log(p, r);
      } else {
        m.A[lane] = p.Gm_h * (ir * ir);
        m.ir[lane] = ir;
      }
    }
    __syncthreads();  // pieces written
    if (warp > 2) return 0.0;
    const double f = m.A[lane] * fma(m.L[lane], m.ir[lane], -m.inv_dh[lane]) + m.B[lane];
    if (warp < 2) return (m.u[lane] + f) * q;
    return fma(m.us[lane], m.izb[lane], f) * q;
  }
};

// A table of up to kTeamMaxComps components: each warp evaluates the factors of
// its share (spread by their FP64 instruction counts), and the owners sum them in
// the table's order, as TablePot does. 3,001 orbits in MilkyWayPotential2022
// (default integrator, 1.5 Gyr, 77 saves): 79 ms on single threads, 26 on teams.
template <bool TIMED_>
struct TeamTable {
  static constexpr bool TIMED = TIMED_;
  struct Shared {
    double fxy[kTeamMaxComps][32], fz[kTeamMaxComps][32];
    DevComp c[kTeamMaxComps];
    int warp[kTeamMaxComps];
  };
  int n;
  const DevLinear* lin;
  Shared& m;

  // Components into shared memory, the costliest first to the warp with least.
  __device__ __forceinline__ void stage(const DevComp* comps) const {
    for (int i = threadIdx.x; i < n; i += blockDim.x) m.c[i] = comps[i];
    __syncthreads();
    if (threadIdx.x == 0) {
      int load[4] = {0, 0, 0, 0};
      for (int i = 0; i < n; ++i) m.warp[i] = -1;
      for (int k = 0; k < n; ++k) {
        int best = -1, cost = -1;
        for (int i = 0; i < n; ++i)
          if (m.warp[i] < 0 && team_cost(m.c[i].kind) > cost) cost = team_cost(m.c[best = i].kind);
        int w = 3;
        for (int v = 2; v >= 0; --v)
          if (load[v] < load[w]) w = v;
        m.warp[best] = w;
        load[w] += cost;
      }
    }
    __syncthreads();
  }

  static __device__ __forceinline__ int team_cost(int kind) {  // FP64 instructions of one gradient
    switch (kind) {
      case NFW: return 42;
      case POWERLAW_CUTOFF: return 400;
      case MIYAMOTO_NAGAI: return 22;
      case HERNQUIST: return 22;
      case ISOCHRONE: return 28;
      default: return 16;
    }
  }

  template <class Side = NoSide>
  __device__ __forceinline__ double grad(TeamShared& sh, int warp, int lane, double q, double t,
                                         Side&& side = Side{}) const {
    if (warp < 3) sh.pos[warp][lane] = q;
    __syncthreads();  // positions written
    const double x = sh.pos[0][lane], y = sh.pos[1][lane], z = sh.pos[2][lane];
    if (std::decay_t<Side>::any && warp == 2) side();
    for (int i = 0; i < n; ++i) {
      if (m.warp[i] != warp) continue;
      const DevComp& c = m.c[i];
      const double dx = x - c.ox, dy = y - c.oy, dz = z - c.oz;
      CompFactors f;
      if constexpr (TIMED_) f = comp_factors(comp_at_time(c, lin[i], t), dx, dy, dz);
      else f = comp_factors(c, dx, dy, dz);
      m.fxy[i][lane] = f.fxy;
      m.fz[i][lane] = f.fz;
    }
    __syncthreads();  // factors written
    if (warp > 2) return 0.0;
    double g = 0.0;
    for (int i = 0; i < n; ++i) {
      const double o = warp == 0 ? m.c[i].ox : warp == 1 ? m.c[i].oy : m.c[i].oz;
      g = fma(warp < 2 ? m.fxy[i][lane] : m.fz[i][lane], q - o, g);
    }
    return g;
  }
};

__device__ __forceinline__ void team_write_save(const IntegrateArgs& a, const OrbitState& s, int64_t k, int j,
                                                double v) {
  a.out[j * a.out_stride + save_index(a, s, k)] = v;
}

// Takes queue positions [0, 16 g.count) in stripes, then base + atomicAdd(queue)
// (base: all positions that this launch hands out in stripes).
template <class TB, class Model>
__device__ void team_loop(const IntegrateArgs& a, const Model& pot, const Blocks& g, long long base) {
  constexpr int S = TB::S;
  constexpr double kIdle = 8.0;  // position of lanes without an orbit
  __shared__ TeamShared sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slot = lane & (kTeamLanes - 1);
  const bool hi = lane >= kTeamLanes;  // second stage of the pair
  const bool owner = warp < 3;
  const int j0 = owner ? warp : 0, j1 = j0 + 3;  // owned components (warps 0-2)
  const int jw = hi ? j1 : j0;                   // the one this lane writes out
  const long long qlen = a.queue_len ? (long long)*a.queue_len : (long long)a.n;
  OrbitState s{};
  s.orbit = -1;
  bool need_orbit = true, queue_open = true, first = true;
  double yp = 0.0, yv = 0.0;  // owned position and velocity component (s.y holds all six for the controller)
  double np = 0.0, nv = 0.0;  // Dopri8: the same of the accepted end state while saves are pending
  double F0v = 0.0;           // owned velocity component of the slope at (tau, y); its position component is yv
  bool need_f0 = false;       // Dopri8: the slope at a state committed after its saves is still to be evaluated
  while (true) {
    // ---- orbits for free lanes (warp 0 dequeues)
    if (warp == 0 && !hi && need_orbit && queue_open) {
      const long long k = first ? (long long)slot * g.count + g.index : base + (long long)atomicAdd(a.queue, 1ULL);
      sh.slot[slot] = k < qlen ? (a.order ? (long long)a.order[k] : k) : -1;
    }
    first = false;
    __syncthreads();
    bool fresh = false;
    if (need_orbit && queue_open) {
      const long long o = sh.slot[slot];
      if (o < 0) {
        queue_open = false;
      } else {
        s.orbit = o;
        const double t0 = a.t0[o], t1 = a.t1[o];
        begin_orbit(a, s, t0, t1);
        if (a.phase == 1) {
          resume_orbit(a, s);
          fresh = true;
        } else {
          const int32_t st = !isfinite(t0) || !isfinite(t1) ? ORBIT_NONFINITE : ORBIT_OK;
          if (t0 == t1 || st != ORBIT_OK) {  // as start_orbit: nothing to integrate, or no end
            if (warp == 0 && !hi) {
              if (t0 == t1)
                for (; s.save_i < s.save_end; ++s.save_i) write_save(a, s, s.save_i, s.y);
              finish_orbit(a, s, t0 == t1 ? ORBIT_OK : st);
            }
            s.orbit = -1;
          } else {
            fresh = true;
          }
        }
        if (fresh) {
          yp = j0 == 0 ? s.y[0] : j0 == 1 ? s.y[1] : s.y[2];  // no dynamic index: s.y stays in registers
          yv = j0 == 0 ? s.y[3] : j0 == 1 ? s.y[4] : s.y[5];
          need_orbit = false;
        }
      }
    }
    const bool active = s.orbit >= 0;
    if (!__syncthreads_or(active)) {
      if (!__syncthreads_or(need_orbit && queue_open)) break;
      continue;
    }
    // ---- slope at new states (and, for Dopri8, newly committed ones): one
    // round, only when a lane needs it
    const bool want_f0 = fresh || (need_f0 && active);
    if (__syncthreads_or(want_f0)) {
      const double gr = pot.grad(sh, warp, lane, want_f0 ? yp : kIdle, Model::TIMED ? with_sign(s.dir, s.tau) : 0.0);
      if (want_f0) F0v = -gr;
    }
    need_f0 = false;
    // ---- first step of orbits that start here (start_orbit, initial_step)
    const bool start = fresh && a.phase == 0;
    const bool probe = start && a.adaptive && !gt_zero(a.dt0);
    double h_init = a.dt0;
    if (__syncthreads_or(probe)) {
      if (owner && !hi) {
        sh.y1[j0][slot] = yv;
        sh.y1[j1][slot] = F0v;
      }
      __syncthreads();
      InitialStep is{};
      double F0[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) F0[j] = sh.y1[j][slot];
      if (probe) is = initial_probe(a, s.y, F0);
      const double gr = pot.grad(sh, warp, lane, probe ? fma(is.h0 * s.dir, yv, yp) : kIdle,
                                 Model::TIMED ? fma(is.h0, s.dir, with_sign(s.dir, s.tau)) : 0.0);
      if (owner && !hi) {
        sh.err[j0][slot] = fma(is.h0 * s.dir, F0v, yv);
        sh.err[j1][slot] = -gr;
      }
      __syncthreads();
      if (probe) {
        double F1[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) F1[j] = sh.err[j][slot];
        h_init = initial_finish<TB>(is, F0, F1);
      }
    }
    if (start) first_step(a, s, h_init);
    // ---- one RK evaluation (integrate_loop): a step from (tau, y), or for
    // Dopri8 with saves pending the sub-step from (tau, y) to the next save
    const bool sub = !TB::FSAL && s.pending && active;
    const double hs = with_sign(s.dir, (sub ? save_tau(a, s, s.save_i) : s.tnext) - s.tau);
    double Fp[S], Fv[S];  // owned components of the stage slopes: position, velocity
    Fp[0] = yv;
    Fv[0] = F0v;
    double y1p = 0.0, y1v = 0.0;
    static_for<0, (S - 1) / 2>([&](auto r) {
      constexpr int I = 2 * decltype(r)::value + 1;  // stages I (lanes 0-15) and I + 1 (lanes 16-31)
      double q = 0.0;
      if (owner) {
        if constexpr (I == 1) {
          Fp[1] = pair_row<TB, 1, 1>(hi, yv, hs, Fv);
        } else {
          const double V = pair_row<TB, I - 1, I>(hi, yv, hs, Fv);
          const double W = __shfl_xor_sync(0xffffffffu, V, kTeamLanes);
          Fp[I - 1] = hi ? W : V;
          Fp[I] = hi ? V : W;
        }
        q = pair_row<TB, I, I + 1>(hi, yp, hs, Fp);
      }
      constexpr double ca = TB::C[I], cb = TB::C[I + 1];
      const double f = -pot.grad(sh, warp, lane, active ? q : kIdle,
                                 Model::TIMED ? fma(hi ? cb : ca, hs, with_sign(s.dir, s.tau)) : 0.0);
      const double o = __shfl_xor_sync(0xffffffffu, f, kTeamLanes);
      Fv[I] = hi ? o : f;
      Fv[I + 1] = hi ? f : o;
      if constexpr (TB::FSAL && I + 2 == S) y1p = q;  // the last row is the solution's (lanes 16-31)
    });
    // solution and error for the owned components, then the shared controller
    if (owner) {
      const bool want_err = a.adaptive && !sub;
      Fp[S - 1] = pair_row<TB, S - 1, S - 1>(hi, yv, hs, Fv);
      double Fw[S];  // lanes 0-15 take the position's sums, lanes 16-31 the velocity's
#pragma unroll
      for (int l = 0; l < S; ++l) Fw[l] = hi ? Fv[l] : Fp[l];
      double y1w;
      if constexpr (TB::FSAL) {
        y1w = hi ? Fp[S - 1] : y1p;
        const double last = __shfl_xor_sync(0xffffffffu, y1p, kTeamLanes);
        if (!hi) y1w = last;
      } else {
        y1w = weighted_comp<TB, W_SOLUTION, true>(hi ? yv : yp, hs, Fw);
      }
      const double other = __shfl_xor_sync(0xffffffffu, y1w, kTeamLanes);
      y1p = hi ? other : y1w;
      y1v = hi ? y1w : other;
      sh.y1[jw][slot] = y1w;
      if (want_err) sh.err[jw][slot] = weighted_comp<TB, W_ERROR, false>(0.0, hs, Fw);
    }
    // ---- step control (pid_adapt), and for Dopri8 the slope at the new state
    // beside it: should the step be rejected, that round was in vain. With nothing
    // to run beside, all warps do the control from the same values.
    const bool control = a.adaptive && !sub && active;
    double y1[6], next_t0 = 0.0, next_t1 = 0.0, F1v = 0.0;
    bool keep = true;
    auto read_y1 = [&]() {
#pragma unroll
      for (int j = 0; j < 6; ++j) y1[j] = sh.y1[j][slot];
    };
    auto adapt = [&]() {
      double err[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) err[j] = sh.err[j][slot];
      keep = pid_adapt<TB::ORDER>(a, s, y1, err, s.tnext - s.tau, next_t0, next_t1);
    };
    if constexpr (TB::FSAL) {
      __syncthreads();
      read_y1();
      if (control) adapt();
    } else {
      F1v = -pot.grad(sh, warp, lane, active ? y1p : kIdle, Model::TIMED ? with_sign(s.dir, s.tnext) : 0.0,
                      side_job([&]() {
                        if (!control) return;
                        read_y1();
                        adapt();
                        if (hi) return;
                        sh.next_t1[slot] = next_t1;
                        sh.prev_inv[slot] = s.prev_inv;
                        sh.prev_prev_inv[slot] = s.prev_prev_inv;
                        sh.flags[slot] = (keep ? 1 : 0) | (s.at_dtmin ? 2 : 0) | (s.status << 2);
                      }));
      read_y1();
      if (control) {
        const int flags = sh.flags[slot];
        keep = (flags & 1) != 0;
        s.at_dtmin = (flags >> 1) & 1;
        s.status = flags >> 2;
        s.prev_inv = sh.prev_inv[slot];
        s.prev_prev_inv = sh.prev_prev_inv[slot];
        next_t0 = keep ? s.tnext : s.tau;
        next_t1 = sh.next_t1[slot];
      }
    }
    if (!active) continue;
    bool done = false;
    int32_t st = ORBIT_OK;
    if (sub) {  // the partial step's end is a save of the accepted step
      if (owner) team_write_save(a, s, s.save_i, jw, hi ? y1v : y1p);
      ++s.save_i;
      if (s.save_i < s.save_end && le_bits(save_tau(a, s, s.save_i), s.tau_new)) continue;
      // all saves of the accepted step written: commit it
      s.pending = 0;
#pragma unroll
      for (int j = 0; j < 6; ++j) s.y[j] = s.ynew[j];
      yp = np;
      yv = nv;
      s.tau = clip_start(s.tau_new, s.tau1);
      need_f0 = true;
      s.tnext = s.tnext_new;
    } else {
      ++s.nsteps;
      if (!a.adaptive) {
        next_t0 = s.tnext;
        next_t1 = s.tnext + a.dt0;
      }
      bool finite = true;
#pragma unroll
      for (int j = 0; j < 6; ++j) finite = finite && bits_finite(y1[j]);
      if (!finite) {
        done = true;
        st = ORBIT_NONFINITE;
      } else {
        const double tprev_new = clip_start(next_t0, s.tau1);
        const double tnext_new = clip_to_end(tprev_new, next_t1, s.tau1, keep);
        if (keep) {
          ++s.naccepted;
          if (s.save_i < s.save_end && le_bits(save_tau(a, s, s.save_i), next_t0)) {
            if constexpr (TB::FSAL) {
              const double ih = 1.0 / (s.tnext - s.tau);
              double Fw[S];
#pragma unroll
              for (int l = 0; l < S; ++l) Fw[l] = hi ? Fv[l] : Fp[l];
              do {
                const double th = (save_tau(a, s, s.save_i) - s.tau) * ih;
                if (owner) team_write_save(a, s, s.save_i, jw, dense_comp(hi ? yv : yp, hs, Fw, th));
                ++s.save_i;
              } while (s.save_i < s.save_end && le_bits(save_tau(a, s, s.save_i), next_t0));
            } else if (a.defer != nullptr) {
              do {
                const bool at_end = dbits(save_tau(a, s, s.save_i)) == dbits(s.tnext);  // as put_deferred_save
                if (owner) team_write_save(a, s, s.save_i, jw, at_end ? (hi ? y1v : y1p) : (hi ? yv : yp));
                if (warp == 3 && !hi && !at_end) a.defer[save_index(a, s, s.save_i)] = with_sign(s.dir, s.tau);
                ++s.save_i;
              } while (s.save_i < s.save_end && le_bits(save_tau(a, s, s.save_i), next_t0));
            } else {  // saves inside this step: keep (tau, y) for the sub-steps
              s.pending = 1;
#pragma unroll
              for (int j = 0; j < 6; ++j) s.ynew[j] = y1[j];
              np = y1p;
              nv = y1v;
              s.tau_new = next_t0;
              s.tnext_new = tnext_new;
              continue;
            }
          }
#pragma unroll
          for (int j = 0; j < 6; ++j) s.y[j] = y1[j];
          yp = y1p;
          yv = y1v;
          F0v = TB::FSAL ? Fv[S - 1] : F1v;
        }
        s.tau = tprev_new;
        s.tnext = tnext_new;
      }
    }
    if (!done) {
      if (s.status != ORBIT_OK) {
        done = true;
        st = s.status;
      } else if (le_bits(s.tau1, s.tau)) {
        done = true;
      } else if (s.nsteps >= a.max_steps) {
        done = true;
        st = ORBIT_MAX_STEPS;
      }
    }
    if (done) {
      if (warp == 0 && !hi) finish_orbit(a, s, st);
      s.orbit = -1;
      need_orbit = true;
      need_f0 = false;
    }
  }
}

// A whole batch on teams, two blocks per SM.
template <class TB>
__global__ void __launch_bounds__(128, 2) k_integrate_mw_team(IntegrateArgs a, MWParams p) {
  __shared__ TeamMW::Shared m;
  team_loop<TB>(a, TeamMW{p, m}, all_blocks(), (long long)kTeamLanes * gridDim.x);
}

template <class TB, bool TIMED>
__global__ void __launch_bounds__(128, 2) k_integrate_table_team(IntegrateArgs a, const DevComp* comps, int ncomp) {
  __shared__ typename TeamTable<TIMED>::Shared m;
  const TeamTable<TIMED> pot{ncomp, a.lin, m};
  pot.stage(comps);
  team_loop<TB>(a, pot, all_blocks(), (long long)kTeamLanes * gridDim.x);
}

// Second pass of the two-pass schedule, one block of 128 threads per SM: the
// first *teams blocks are teams and take the longest orbits, the others run one
// thread per orbit; when their first orbits are done, all draw on one queue.
template <class TB>
__global__ void __launch_bounds__(128, 1) k_integrate_mw_mixed(IntegrateArgs a, MWParams p, const unsigned* teams) {
  __shared__ TeamMW::Shared m;
  const unsigned t = min(*teams, gridDim.x - 1);
  const long long first = (long long)kTeamLanes * t;  // queue position of the longest orbit without a team
  if (blockIdx.x < t) {
    team_loop<TB>(a, TeamMW{p, m}, Blocks{t, blockIdx.x, 0}, first + 128LL * (gridDim.x - t));
  } else {
    integrate_loop<TB>(a, MWPot{p}, Blocks{gridDim.x - t, blockIdx.x - t, first});
  }
}

}  // namespace gal
