// Plummer spheres with the inverse power in 64-bit fixed point.
//
// A sphere's gradient is about twenty FP64 instructions, and GB300's FP64 pipe
// takes 64 cycles for each of a warp's; its integer and FP32 pipes take one or
// two. Here the offsets d = x - c are FP64 differences, as in comp_grad, but
// (d^2 + b^2)^(-3/2) comes from 64-bit integers: an FP32 reciprocal square root
// corrected by its exact residual. Six FP64 instructions are left, three for the
// offsets and three that add f d to the sum.
//
// The fixed point floats with each sphere and point: with E the exponent of the
// largest of |d_j| and b, v = 2^(60 - E) d has 2^60 <= max(|v_j|, 2^(60 - E) b) < 2^61,
// and what is shifted out of the smaller components is below 2^-60 of the largest,
// whatever the scales of the table. Then
//   W = 2^-60 (|v|^2 + (2^(60 - E) b)^2)   in [2^60, 2^64),
//   Y = 2^40 / sqrt(W / 2^32)               from FP32, 26 bits,
//   e = 1 - W Y^2 / 2^112                   (|e| < 2^-20), in units of 2^-80,
//   W^(-3/2) = 2^-168 Y^3 (1 - e)^(-3/2) = 2^-168 Y^3 (1 + 3/2 e + 15/8 e^2),
// the next term being below 2^-59: f is right to 56 bits before its rounding to
// FP64, and a term's error is that of the roundings of d, f and their product.
//
// Scales outside 2^-256 .. 2^256 (an offset of zero from a point mass among them),
// infinities and NaN take comp_grad.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>

namespace gal {

struct FixedPlummer {  // 64 bytes
  double c[3];    // centre
  uint64_t b2;    // 2^-60 (2^(60 - exponent of b) b)^2, 0 for b = 0
  uint64_t gm;    // |G m| = gm 2^gexp, gm in [2^63, 2^64), or 0
  uint32_t bhi;   // high word of b; all ones: the sphere takes comp_grad
  int32_t e0;     // exponent of f in units of R's: gexp - 178 + 3 (60 + 1023) (- 3 E, biased)
  uint32_t sign;  // 0x80000000 for m < 0
  uint32_t pad[3];
};
static_assert(sizeof(FixedPlummer) == 64, "FixedPlummer layout");

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ uint32_t fx_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ int fx_clz(uint32_t v) { return __clz((int)v); }
__device__ __forceinline__ float fx_rsqrt(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ uint32_t fx_f2u(float v) { return __float2uint_rn(v); }
__device__ __forceinline__ uint32_t fx_hi(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t fx_lo(double v) { return (uint32_t)__double2loint(v); }
__device__ __forceinline__ double fx_double(uint64_t b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ uint64_t fx_shr(uint64_t v, int n) {  // 0 from 64 bits on
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
  return r;
}
#else
inline uint64_t fx_bits(double v) {
  uint64_t b;
  std::memcpy(&b, &v, sizeof(b));
  return b;
}
inline uint32_t fx_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int fx_clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline float fx_rsqrt(float v) { return 1.0f / __builtin_sqrtf(v); }
inline uint32_t fx_f2u(float v) { return (uint32_t)__builtin_rintf(v); }
inline uint32_t fx_hi(double v) { return (uint32_t)(fx_bits(v) >> 32); }
inline uint32_t fx_lo(double v) { return (uint32_t)fx_bits(v); }
inline double fx_double(uint64_t b) {
  double v;
  std::memcpy(&v, &b, sizeof(v));
  return v;
}
inline uint64_t fx_shr(uint64_t v, int n) { return n < 64 ? v >> n : 0; }
#endif

// m 2^e as the bits of a double, rounded to nearest: m's leading one at bit
// 63 - lz, the result normal.
__host__ __device__ __forceinline__ uint64_t fx_pack(uint64_t m, int lz, int e) {
  const uint64_t n = m << lz;
  // the implicit bit adds one to the exponent field, a carry from rounding another
  return ((uint64_t)(uint32_t)(1023 + 62 - lz + e) << 52) + (n >> 11) + ((n >> 10) & 1u);
}

// The record of a sphere with centre c, scale b >= 0 and G m.
inline FixedPlummer fixed_record(const double* c, double b, double Gm) {
  FixedPlummer f{};
  for (int j = 0; j < 3; ++j) f.c[j] = c[j];
  int e = 0;
  const double m = std::frexp(std::fabs(Gm), &e);
  if (Gm != 0.0 && !(std::isfinite(Gm) && std::abs(e) <= 200)) {  // f's exponent may not stay normal
    f.bhi = 0xffffffffu;
    return f;
  }
  f.gm = (uint64_t)std::ldexp(m, 64);
  f.sign = Gm < 0.0 ? 0x80000000u : 0u;
  f.e0 = (e - 64) - 178 + 3 * (60 + 1023);
  if (b > 0.0) {
    uint64_t bits;
    std::memcpy(&bits, &b, sizeof(bits));
    f.bhi = (uint32_t)(bits >> 32);
    int eb = 0;
    const uint64_t n = (uint64_t)std::ldexp(std::frexp(b, &eb), 53);  // exact; b2 = (n 2^8)^2 / 2^60 = n^2 / 2^44
    const uint64_t hi = n >> 32, lo = n & 0xffffffffu;
    f.b2 = (hi * hi << 20) + ((hi * lo) >> 11) + ((lo * lo) >> 44);
  }
  return f;
}

// Factor f and offset d of one sphere at x: grad = f d. False, and f = 0, where
// the range does not do.
__host__ __device__ __forceinline__ bool fixed_plummer(const FixedPlummer& p, const double* x, double* f, double* d) {
  uint32_t a[3], M = p.bhi;
  for (int j = 0; j < 3; ++j) {
    d[j] = x[j] - p.c[j];
    a[j] = fx_hi(d[j]) & 0x7fffffffu;
    M = a[j] > M ? a[j] : M;
  }
  const int E = (int)(M >> 20);
  const bool fits = (uint32_t)(E - (1023 - 256)) < 512u;
  uint64_t S = 0;
  int64_t T = 0;
  for (int j = 0; j < 3; ++j) {
    const int drop = E - (int)(a[j] >> 20);
    const uint64_t m = (uint64_t)((a[j] & 0xfffffu) | 0x100000u) << 32 | fx_lo(d[j]);
    const uint64_t v = fx_shr(m << 8, drop);  // zero has the lowest exponent: nothing is left of its implicit bit
    const int32_t lo = (int32_t)v;
    const int32_t hi = (int32_t)((uint32_t)(v >> 32) + ((uint32_t)lo >> 31));  // v = 2^32 hi + lo, lo signed
    S += (uint64_t)((int64_t)hi * hi);
    T += (int64_t)hi * lo;
  }
  const int sh = 2 * (E - (int)((p.bhi >> 20) & 0x7ffu));  // >= 0: b is among the candidates for the largest
  uint64_t W = (S << 4) + (uint64_t)(T >> 27) + 4u;  // + the mean of 2^-60 sum lo^2
  W += fx_shr(p.b2, sh);
  const uint32_t Wh = (uint32_t)(W >> 32), Wl = (uint32_t)W;
  const uint32_t Y = fx_f2u(fx_rsqrt((float)Wh) * 1099511627776.0f);
  const uint64_t Y2 = (uint64_t)Y * Y;
  const uint32_t Yh = (uint32_t)(Y2 >> 32), Yl = (uint32_t)Y2;
  uint64_t P = (uint64_t)Wh * Yl + fx_mulhi(Wl, Yl);  // W Y^2 / 2^32 modulo 2^64; its leading 2^80 drops out
  P += (uint64_t)Wl * Yh;
  P += (uint64_t)(Wh * Yh) << 32;
  const int64_t Q = -(int64_t)P;  // e 2^80
  const float ef = (float)(int32_t)(Q >> 32);
  const int64_t q = Q >> 16;
  const int64_t c = q + (q >> 1) + (int64_t)(int32_t)fx_f2u(ef * ef * (1.875f / 4294967296.0f));  // (3/2 e + 15/8 e^2) 2^64
  const uint64_t N = Y2 << 11;
  const int32_t ch = (int32_t)(c >> 32);
  const uint32_t cl = (uint32_t)c, Nh = (uint32_t)(N >> 32), Nl = (uint32_t)N;
  const uint64_t U = N + (uint64_t)((int64_t)(int32_t)Nh * ch) + fx_mulhi(Nh, cl) +
                     (uint64_t)(((int64_t)(int32_t)(Nl >> 1) * ch) >> 31);
  const uint32_t Y5 = Y << 5;
  const uint64_t V = (uint64_t)(uint32_t)(U >> 32) * Y5 + fx_mulhi((uint32_t)U, Y5);
  const uint32_t Vh = (uint32_t)(V >> 32), Vl = (uint32_t)V, Gh = (uint32_t)(p.gm >> 32), Gl = (uint32_t)p.gm;
  const uint64_t R = (uint64_t)Vh * Gh + fx_mulhi(Vh, Gl) + fx_mulhi(Vl, Gh);
  const uint64_t bits = fx_pack(R, fx_clz((uint32_t)(R >> 32)) & 31, p.e0 - 3 * E);
  *f = fx_double(p.gm != 0 && fits ? bits | ((uint64_t)p.sign << 32) : 0);
  return fits;
}

#if defined(__CUDACC__)
}  // namespace gal

#include "potentials.cuh"

namespace gal {

// What the other components are, with the spheres' records in device memory: a
// graph captured with the table sees the values of the last gal_potential_update,
// as it does through the component table. Counts and kinds never change.
struct FixedOthers {
  MWParams mw;
  int32_t is_mw;  // a Milky Way's four
};

struct FixedTable {
  const FixedPlummer* f;  // spheres, in the order of the table's Plummer entries
  const FixedOthers* others;
  const int32_t* at;      // the spheres' table indices, then those of the other components
  int n, nother;
};

// A table with its spheres in fixed point, for `lanes` lanes per orbit (a power of
// two): each lane sums its share of the spheres and of the other components, a
// butterfly of shuffles gives every lane the same total (as WarpTablePot), and the
// four components of a Milky Way, if those are the others, are added by its own code.
struct FixedTablePot {
  const FixedPlummer* f;   // shared memory
  const DevComp* others;   // shared memory
  const FixedOthers* o;    // shared memory
  const DevComp* comps;    // the whole table, for spheres out of range
  FixedTable t;
  int lanes;

  __device__ __forceinline__ void grad(double x, double y, double z, double& gx, double& gy, double& gz) const {
    const int sub = threadIdx.x & (lanes - 1);
    double ax = 0.0, ay = 0.0, az = 0.0;
    const double X[3] = {x, y, z};
    bool all = true;
#pragma unroll 1
    for (int i = sub; i < t.n; i += lanes) {
      double w, d[3];
      const bool ok = fixed_plummer(f[i], X, &w, d);
      all &= ok;
      if (ok) {
        ax = fma(w, d[0], ax);
        ay = fma(w, d[1], ay);
        az = fma(w, d[2], az);
      }
    }
    if (!all) {  // the spheres left out above
      for (int i = sub; i < t.n; i += lanes) {
        double w, d[3];
        if (!fixed_plummer(f[i], X, &w, d)) comp_grad(comps[t.at[i]], x, y, z, ax, ay, az);
      }
    }
    const bool mw = o->is_mw != 0;
    if (!mw)
      for (int i = sub; i < t.nother; i += lanes) comp_grad(others[i], x, y, z, ax, ay, az);
    const unsigned mask = lanes >= 32 ? 0xffffffffu : ((1u << lanes) - 1u) << ((threadIdx.x & 31) & ~(unsigned)(lanes - 1));
    for (int m = lanes >> 1; m >= 1; m >>= 1) {
      ax += __shfl_xor_sync(mask, ax, m);
      ay += __shfl_xor_sync(mask, ay, m);
      az += __shfl_xor_sync(mask, az, m);
    }
    if (mw) {
      double hx, hy, hz;
      MWPot{o->mw}.grad(x, y, z, hx, hy, hz);
      ax += hx;
      ay += hy;
      az += hz;
    }
    gx = ax;
    gy = ay;
    gz = az;
  }
};

#endif  // __CUDACC__

}  // namespace gal
