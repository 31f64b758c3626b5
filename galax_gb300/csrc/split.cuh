// Device side of the short-range Plummer sum (see split.cu): cell lookup and
// the tapered potential and gradient, shared by the evaluation kernel and the
// surrogate integrator's stage kernels.
#pragma once

#include <cstdint>

#include "potentials.cuh"

namespace gal {

struct SplitDev {
  const int64_t* start;  // [nx^3 + 1] CSR offsets per cell
  const float4* items;   // [items]: centre relative to its cell's low corner (x, y, z), G m
  const float* b2;       // [items]: b^2
  int nx;
  double lo, h, inv_h;   // cell (ix, iy, iz) covers lo + h [ix, ix+1) x ...
  double rc2, inv_rc2;   // r_cut^2 and its inverse
};

// A point in its cell: place relative to the cell's low corner, list range.
struct SplitCell {
  float x, y, z;
  int64_t b0, b1;  // b0 == b1: nothing near
};

__device__ __forceinline__ SplitCell split_cell(const SplitDev& s, double x, double y, double z) {
  SplitCell c{0.f, 0.f, 0.f, 0, 0};
  const double fx = (x - s.lo) * s.inv_h, fy = (y - s.lo) * s.inv_h, fz = (z - s.lo) * s.inv_h;
  if (!(fx >= 0.0 && fy >= 0.0 && fz >= 0.0)) return c;
  const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
  if (ix >= s.nx || iy >= s.nx || iz >= s.nx) return c;
  const int64_t cell = ((int64_t)iz * s.nx + iy) * s.nx + ix;
  c.b0 = s.start[cell];
  c.b1 = s.start[cell + 1];
  if (c.b0 == c.b1) return c;
  c.x = (float)fma(-(double)ix, s.h, x - s.lo);
  c.y = (float)fma(-(double)iy, s.h, y - s.lo);
  c.z = (float)fma(-(double)iz, s.h, z - s.lo);
  return c;
}

// One list entry's term, accumulated. Without a branch: an entry beyond r_cut adds
// exact zeros, and the loads of the entries that follow do not wait for it (with
// four entries at a time, 20 surrogate steps of 131,072 orbits: 23.7 -> 22.8 ms;
// eight lanes to a point would make 20.5, in another order of the sum).
__device__ __forceinline__ void split_term(const SplitDev& s, int64_t k, float x, float y, float z, float rc2,
                                           float inv_rc2, float& ax, float& ay, float& az, float& ap) {
  const float4 it = s.items[k];
  const float b2 = s.b2[k];
  const float dx = x - it.x, dy = y - it.y, dz = z - it.z;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const bool in = d2 < rc2;
  const float t = fmaf(-d2, inv_rc2, 1.0f);
  const float S = t * t * t;
  const float is = rsqrtf(d2 + b2);
  const float Gmis = in ? it.w * is : 0.0f;
  const float f = Gmis * fmaf(S, is * is, 6.0f * t * t * inv_rc2);
  ax = fmaf(f, dx, ax);
  ay = fmaf(f, dy, ay);
  az = fmaf(f, dz, az);
  ap = fmaf(-Gmis, S, ap);
}

// Accumulates grad of sum_i Phi_i S(d_i / r_c) into g (and the potential into *phi).
// S(q) = (1 - q^2)^3: grad(Phi S) = d G m is (S is^2 + 6 t^2 / r_c^2), t = 1 - q^2,
// is = 1 / sqrt(d^2 + b^2). The point is placed relative to its cell's low
// corner once in FP64; the centres are stored relative to the same corner in
// FP32, so every term is FP32 work only (the FP32 pipe is 64x the FP64 one
// on this chip) and carries ~1e-7 relative error, far below the MLP's share of
// the surrogate's error; the sum is added in FP64.
__device__ __forceinline__ void split_short(const SplitDev& s, double x, double y, double z, double& gx, double& gy,
                                            double& gz, double* phi) {
  const SplitCell c = split_cell(s, x, y, z);
  if (c.b0 == c.b1) return;
  const float rc2 = (float)s.rc2, inv_rc2 = (float)s.inv_rc2;
  float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
#pragma unroll 4
  for (int64_t k = c.b0; k < c.b1; ++k) split_term(s, k, c.x, c.y, c.z, rc2, inv_rc2, ax, ay, az, ap);
  gx += (double)ax;
  gy += (double)ay;
  gz += (double)az;
  if (phi) *phi += (double)ap;
}

}  // namespace gal

struct gal_split;
// Device view of a split (host pointer to a host-side struct; NULL for NULL).
extern "C" const gal::SplitDev* gal_split_device(const gal_split* sp);

namespace gal {

// A potential plus the short-range Plummer sum.
template <class Base>
struct WithShort {
  Base base;
  SplitDev sp;
  __device__ __forceinline__ void grad(double x, double y, double z, double& gx, double& gy, double& gz) const {
    base.grad(x, y, z, gx, gy, gz);
    split_short(sp, x, y, z, gx, gy, gz, nullptr);
  }
};

}  // namespace gal
