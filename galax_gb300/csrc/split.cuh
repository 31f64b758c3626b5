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

// One list entry's term, accumulated.
__device__ __forceinline__ void split_term(const SplitDev& s, int64_t k, float x, float y, float z, float rc2,
                                           float inv_rc2, float& ax, float& ay, float& az, float& ap) {
  const float4 it = s.items[k];
  const float dx = x - it.x, dy = y - it.y, dz = z - it.z;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  if (d2 >= rc2) return;
  const float t = fmaf(-d2, inv_rc2, 1.0f);
  const float S = t * t * t;
  const float is = rsqrtf(d2 + s.b2[k]);
  const float Gmis = it.w * is;
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
  for (int64_t k = c.b0; k < c.b1; ++k) split_term(s, k, c.x, c.y, c.z, rc2, inv_rc2, ax, ay, az, ap);
  gx += (double)ax;
  gy += (double)ay;
  gz += (double)az;
  if (phi) *phi += (double)ap;
}

// The same sums for a warp's 32 points, eight lanes to a point and four points at
// a time: the lanes of a group read neighbouring list entries, where a lane per
// point makes every load a gather of 32 lines. All lanes of the warp take part.
// With the stage state of 131,072 orbits, 512 spheres, r_cut 12 kpc: 85 us with a
// lane per point, 45 us like this.
__device__ __forceinline__ void split_short_warp(const SplitDev& s, double x, double y, double z, float* g) {
  const int lane = threadIdx.x & 31, sub = lane & 7;
  const SplitCell c = split_cell(s, x, y, z);
  const int n = (int)(c.b1 - c.b0);
  const float rc2 = (float)s.rc2, inv_rc2 = (float)s.inv_rc2;
  g[0] = g[1] = g[2] = 0.f;
  for (int q = 0; q < 8; ++q) {
    const int src = 4 * q + (lane >> 3);  // the point of this lane's group
    const float px = __shfl_sync(0xffffffffu, c.x, src), py = __shfl_sync(0xffffffffu, c.y, src),
                pz = __shfl_sync(0xffffffffu, c.z, src);
    const int64_t b0 = __shfl_sync(0xffffffffu, c.b0, src);
    const int m = __shfl_sync(0xffffffffu, n, src);
    float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll 4
    for (int k = sub; k < m; k += 8) {  // split_term without its branch, so that loads run ahead
      const float4 it = s.items[b0 + k];
      const float b2 = s.b2[b0 + k];
      const float dx = px - it.x, dy = py - it.y, dz = pz - it.z;
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float t = fmaf(-d2, inv_rc2, 1.0f);
      const float is = rsqrtf(d2 + b2);
      const float f = it.w * is * fmaf(t * t * t, is * is, 6.0f * t * t * inv_rc2);
      const float g = d2 < rc2 ? f : 0.0f;
      ax = fmaf(g, dx, ax);
      ay = fmaf(g, dy, ay);
      az = fmaf(g, dz, az);
    }
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, w);
      ay += __shfl_xor_sync(0xffffffffu, ay, w);
      az += __shfl_xor_sync(0xffffffffu, az, w);
    }
    // back to the points' own lanes 4 q .. 4 q + 3
    const float rx = __shfl_sync(0xffffffffu, ax, 8 * (lane & 3)), ry = __shfl_sync(0xffffffffu, ay, 8 * (lane & 3)),
                rz = __shfl_sync(0xffffffffu, az, 8 * (lane & 3));
    if ((lane >> 2) == q) {
      g[0] = rx;
      g[1] = ry;
      g[2] = rz;
    }
  }
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

// A potential's gradient in two parts: the short-range sum (all lanes of the warp
// take part), and the rest. False / true: without or with a short-range sum.
template <class Base>
__device__ __forceinline__ bool near_grad(const Base&, double, double, double, float*) {
  return false;
}
template <class Base>
__device__ __forceinline__ bool near_grad(const WithShort<Base>& p, double x, double y, double z, float* g) {
  split_short_warp(p.sp, x, y, z, g);
  return true;
}
template <class Base>
__device__ __forceinline__ bool far_grad(const Base& p, double x, double y, double z, double* g) {
  p.grad(x, y, z, g[0], g[1], g[2]);
  return false;
}
template <class Base>
__device__ __forceinline__ bool far_grad(const WithShort<Base>& p, double x, double y, double z, double* g) {
  p.base.grad(x, y, z, g[0], g[1], g[2]);
  return true;
}

}  // namespace gal
