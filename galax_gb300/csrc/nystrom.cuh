// Runge-Kutta steps of a static potential in Nystrom form.
//
// With a force that depends on the position alone, y' = (v, -g(x)), the stage
// velocities can be eliminated from a Runge-Kutta step (Hairer, Norsett & Wanner,
// Solving Ordinary Differential Equations I, II.14): for row sums c_i = sum_l a_il
// and sum b_i = 1,
//   X_i = x + h (c_i v - h sum_l abar_il g(X_l)),   abar = A A,
//   x1  = x + h (v - h sum_l bbar_l g(X_l)),        bbar = b A,
//   v1  = v - h sum_l b_l g(X_l):
// three sums per stage instead of six, over smaller coefficients (Dopri8: 57
// entries of at most 3.0 instead of 59 of at most 16.7). The results are those of
// the step in its usual form up to rounding.
#pragma once

#include "tableaux.cuh"

namespace gal {

//
// The coefficients are rounded once, from products summed in twice the precision:
// the terms of abar and bbar are up to a thousand times the entries they leave, and
// summed in FP64 the table itself would be wrong by up to 1e-14. The weights b of
// the velocity are FP64 numbers whose sum is exactly 1: rounded each to its nearest,
// Dopri8's sum to 1 - 7.6e-17, a force too weak by as much in every step, which
// drifts along the orbit and adds up over a batch (500 steps of 0.5 Myr against
// extended precision: the mean time by which orbits lag, 4.7e-14 Myr in the usual
// form, 5.4e-14 with plain products and weights, 2.7e-14 so).
template <class TB>
struct NystromTable {
  double a[TB::S][TB::S];
  double b[TB::S];
  double v[TB::S];   // the method's b, its sum 1
  bool used[TB::S];  // the stage's gradient enters a later stage or the result
};

// Sums and products in twice the precision (T. J. Dekker, "A floating-point technique
// for extending the available precision", Numer. Math. 18, 1971).
struct Sum2 {
  double hi, lo;
};
constexpr Sum2 add2(Sum2 s, double v) {
  const double h = s.hi + v, z = h - s.hi;
  return Sum2{h, s.lo + ((s.hi - (h - z)) + (v - z))};
}
constexpr Sum2 fma2(Sum2 s, double x, double y) {
  constexpr double c = 134217729.0;  // 2^27 + 1
  const double xh = c * x - (c * x - x), yh = c * y - (c * y - y), xl = x - xh, yl = y - yh;
  const double t = x * y;
  return add2(add2(s, t), ((xh * yh - t) + xh * yl + xl * yh) + xl * yl);
}
// What the roundings of a method's own coefficients leave of an entry that is zero
// is below 2e-16; the smallest other one is 4e-3.
constexpr double nystrom_entry(Sum2 s) {
  const double v = s.hi + s.lo;
  return v < 1e-15 && v > -1e-15 ? 0.0 : v;
}

template <class TB>
constexpr NystromTable<TB> make_nystrom() {
  NystromTable<TB> t{};
  for (int l = 0; l < TB::S; ++l) {
    Sum2 sb{0.0, 0.0};
    for (int k = 0; k < TB::S; ++k) sb = fma2(sb, TB::B[k], TB::A[k][l]);
    t.b[l] = nystrom_entry(sb);
    t.v[l] = TB::B[l];
    for (int i = 0; i < TB::S; ++i) {
      Sum2 sa{0.0, 0.0};
      for (int k = 0; k < TB::S; ++k) sa = fma2(sa, TB::A[i][k], TB::A[k][l]);
      t.a[i][l] = nystrom_entry(sa);
    }
  }
  // the weights' sum to 1 by steps of one unit in the last place of single weights
  for (bool moved = true; moved;) {
    Sum2 s{-1.0, 0.0};
    for (int l = 0; l < TB::S; ++l) s = add2(s, t.v[l]);
    const double off = s.hi + s.lo;
    double best = off < 0.0 ? -off : off, to = 0.0;
    int at = -1;
    for (int l = 0; l < TB::S; ++l)
      for (int sign = -1; sign <= 1; sign += 2) {
        const double w = t.v[l] + sign * (t.v[l] * 0x1p-53 * 1.25), left = off + (w - t.v[l]);
        if (t.v[l] != 0.0 && (left < 0.0 ? -left : left) < best) {
          best = left < 0.0 ? -left : left;
          at = l;
          to = w;
        }
      }
    moved = at >= 0;
    if (moved) t.v[at] = to;
  }
  for (int l = TB::S - 1; l >= 0; --l) {
    t.used[l] = TB::B[l] != 0.0 || t.b[l] != 0.0;
    for (int i = l + 1; i < TB::S; ++i) t.used[l] = t.used[l] || (t.used[i] && t.a[i][l] != 0.0);
  }
  return t;
}

template <class TB>
inline constexpr NystromTable<TB> kNystrom = make_nystrom<TB>();

// X_i from the state (x, v) and the gradients g[0..i).
template <class TB, int I>
__device__ __forceinline__ void nystrom_stage(const double* x, const double* v, double h,
                                              const double (&g)[TB::S][3], double* X) {
  constexpr double ci = TB::C[I];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double acc = 0.0;
    static_for<0, I>([&](auto l) {
      constexpr int L = decltype(l)::value;
      constexpr double c = kNystrom<TB>.a[I][L];
      if constexpr (c != 0.0) acc = fma(c, g[L][j], acc);
    });
    X[j] = fma(h, fma(-h, acc, ci * v[j]), x[j]);
  }
}

// The step's end state from all gradients.
template <class TB>
__device__ __forceinline__ void nystrom_end(double* x, double* v, double h, const double (&g)[TB::S][3]) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double ax = 0.0, av = 0.0;
    static_for<0, TB::S>([&](auto l) {
      constexpr int L = decltype(l)::value;
      constexpr double cx = kNystrom<TB>.b[L], cv = kNystrom<TB>.v[L];
      if constexpr (cx != 0.0) ax = fma(cx, g[L][j], ax);
      if constexpr (cv != 0.0) av = fma(cv, g[L][j], av);
    });
    x[j] = fma(h, fma(-h, ax, v[j]), x[j]);
    v[j] = fma(-h, av, v[j]);
  }
}

}  // namespace gal
