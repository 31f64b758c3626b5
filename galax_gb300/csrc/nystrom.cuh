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

template <class TB>
struct NystromTable {
  double a[TB::S][TB::S];
  double b[TB::S];
  bool used[TB::S];  // the stage's gradient enters a later stage or the result
};

template <class TB>
constexpr NystromTable<TB> make_nystrom() {
  NystromTable<TB> t{};
  for (int i = 0; i < TB::S; ++i)
    for (int l = 0; l < TB::S; ++l)
      for (int k = 0; k < TB::S; ++k) t.a[i][l] += TB::A[i][k] * TB::A[k][l];
  for (int l = 0; l < TB::S; ++l)
    for (int k = 0; k < TB::S; ++k) t.b[l] += TB::B[k] * TB::A[k][l];
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
      constexpr double cx = kNystrom<TB>.b[L], cv = TB::B[L];
      if constexpr (cx != 0.0) ax = fma(cx, g[L][j], ax);
      if constexpr (cv != 0.0) av = fma(cv, g[L][j], av);
    });
    x[j] = fma(h, fma(-h, ax, v[j]), x[j]);
    v[j] = fma(-h, av, v[j]);
  }
}

}  // namespace gal
