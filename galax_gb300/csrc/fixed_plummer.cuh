// The Plummer spheres of a table in 64-bit fixed point.
//
// A sphere's gradient is about twenty FP64 instructions, and GB300's FP64 pipe
// takes 64 cycles for each of a warp's; its integer and FP32 pipes take one or
// two. Here positions, centres and squared distances are 64-bit integers, and
// (d^2 + b^2)^(-3/2) comes from an FP32 reciprocal square root corrected by its
// exact residual in integers: about 250 instructions, of which only the three
// that add f d to the sum are FP64's. Every intermediate keeps at least 56
// significant bits, so a term's relative error is that of its two roundings to
// FP64 (of f and d), 2^-53 each; the FP64 evaluation rounds about ten times.
//
// With v = 2^(s + k) d, k chosen for each sphere and point so that the largest of
// |v_j| and 2^(s + k) b is in [2^60, 2^61):
//   W = 2^-60 (|v|^2 + (2^(s+k) b)^2)   in [2^60, 2^64),
//   Y = 2^40 / sqrt(W / 2^32)           from FP32, 26 bits,
//   e = 1 - W Y^2 / 2^112               (|e| < 2^-20), in units of 2^-80,
//   W^(-3/2) = 2^-168 Y^3 (1 - e)^(-3/2) = 2^-168 Y^3 (1 + 3/2 e + 15/8 e^2),
// the next term being below 2^-59.
//
// s is set for a table so that its centres and four times their distances fit
// (fixed_table); a point beyond, or one within 2^(32 - s) of a sphere's centre
// whose b is smaller, takes comp_grad.
#pragma once

#include <cstdint>

#include "potentials.cuh"

namespace gal {

struct FixedPlummer {  // 64 bytes
  int64_t c[3];        // centre, 2^s
  uint64_t b2;         // 2^-60 (2^(s + kb) b)^2, 0 for b = 0
  uint64_t gm;         // |G m| = gm 2^gexp, gm in [2^63, 2^64), or 0
  uint32_t bhi;        // high word of 2^s b
  int32_t kb;          // k that b alone would take
  int32_t e0;          // exponent of f 2^-(s + k) in units of R's: gexp - 178 + 2 s (+ 2 k)
  uint32_t sign;       // 0x80000000 for m < 0
  uint64_t pad;
};
static_assert(sizeof(FixedPlummer) == 64, "FixedPlummer layout");

struct FixedTable {
  const FixedPlummer* f;  // spheres, in the order of the table's Plummer entries
  const int32_t* at;      // their table indices, then those of the other components
  int n, nother;
  int s;
  double scale, xmax;     // 2^s; positions up to xmax fit
};

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ uint32_t fx_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ int fx_clz(uint32_t v) { return __clz((int)v); }
__device__ __forceinline__ int fx_clzll(uint64_t v) { return __clzll((long long)v); }
__device__ __forceinline__ float fx_rsqrt(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ uint32_t fx_f2u(float v) { return __float2uint_rn(v); }
#else
inline uint32_t fx_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int fx_clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline int fx_clzll(uint64_t v) { return v ? __builtin_clzll(v) : 64; }
inline float fx_rsqrt(float v) { return 1.0f / __builtin_sqrtf(v); }
inline uint32_t fx_f2u(float v) { return (uint32_t)__builtin_rintf(v); }
#endif

// m 2^e as the bits of a double, rounded to nearest: m's leading one at bit
// 63 - lz, the result normal.
__host__ __device__ __forceinline__ uint64_t fx_pack(uint64_t m, int lz, int e) {
  const uint64_t n = m << lz;
  // the implicit bit adds one to the exponent field, a carry from rounding another
  return ((uint64_t)(uint32_t)(1023 + 62 - lz + e) << 52) + (n >> 11) + ((n >> 10) & 1u);
}

// 2^(s+k) d as a double, rounded to nearest, in 32-bit words (|v| < 2^61).
__host__ __device__ __forceinline__ uint64_t fx_offset(int64_t v) {
  const uint32_t sgn = (uint32_t)((int32_t)(v >> 32) >> 31);
  const uint64_t a = ((uint64_t)v ^ ((uint64_t)sgn << 32 | sgn)) + (sgn & 1u);
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  const bool low = ah == 0;
  const uint32_t th = low ? al : ah, tl = low ? 0u : al;  // leading one in th
  const int lz = fx_clz(th) & 31;
  const uint64_t n = (((uint64_t)th << 32) | tl) << lz;
  const uint32_t nh = (uint32_t)(n >> 32), nl = (uint32_t)n;
  const uint32_t e = (uint32_t)((low ? 1023 + 30 : 1023 + 62) - lz);
  const uint64_t bits = ((uint64_t)((e << 20) + (nh >> 11)) << 32 | ((nh << 21) | (nl >> 11))) + ((nl >> 10) & 1u);
  return th != 0 ? bits | ((uint64_t)(sgn & 0x80000000u) << 32) : 0;
}

// Factor f 2^-(s+k) and offsets 2^(s+k) d of one sphere at the fixed-point
// position x: grad = f d. False, and f = 0, where the range does not do.
__host__ __device__ __forceinline__ bool fixed_plummer(const FixedPlummer& p, const int64_t* x, uint64_t* f,
                                                       uint64_t* d) {
  int64_t v[3];
  uint32_t M = p.bhi;
  for (int j = 0; j < 3; ++j) {
    v[j] = x[j] - p.c[j];
    const int32_t h = (int32_t)(v[j] >> 32);
    M |= (uint32_t)(h ^ (h >> 31));
  }
  const bool fits = M != 0;
  const int k = fx_clz(M | 1u) - 3;  // >= 0 by the choice of s
  uint64_t S = 0;
  int64_t T = 0;
  for (int j = 0; j < 3; ++j) {
    v[j] = (int64_t)((uint64_t)v[j] << k);
    const int32_t lo = (int32_t)v[j];
    const int32_t hi = (int32_t)((uint32_t)(v[j] >> 32) + ((uint32_t)lo >> 31));  // v = 2^32 hi + lo, lo signed
    S += (uint64_t)((int64_t)hi * hi);
    T += (int64_t)hi * lo;
  }
  const int sh = 2 * (p.kb - k);  // >= 0: b is among the candidates for the largest
  uint64_t W = (S << 4) + (uint64_t)(T >> 27) + 4u;  // + the mean of 2^-60 sum lo^2
  W += sh < 64 ? p.b2 >> (sh & 63) : 0;
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
  const uint64_t bits = fx_pack(R, fx_clz((uint32_t)(R >> 32)) & 31, p.e0 + 2 * k);
  *f = p.gm != 0 && fits ? bits | ((uint64_t)p.sign << 32) : 0;
  for (int j = 0; j < 3; ++j) d[j] = fx_offset(v[j]);
  return fits;
}

// A table with its spheres in fixed point, for `lanes` lanes per orbit (a power of
// two): each lane sums its share of the spheres and of the other components, a
// butterfly of shuffles gives every lane the same total (as WarpTablePot), and the
// four components of a Milky Way, if those are the others, are added by its own code.
struct FixedTablePot {
  const FixedPlummer* f;   // shared memory
  const DevComp* others;   // shared memory
  const DevComp* comps;    // the whole table, for points out of range
  FixedTable t;
  int lanes;
  bool mw;
  MWPot milky_way;

  __device__ __forceinline__ void grad(double x, double y, double z, double& gx, double& gy, double& gz) const {
    const int sub = threadIdx.x & (lanes - 1);
    double ax = 0.0, ay = 0.0, az = 0.0;
    if (fabs(x) <= t.xmax && fabs(y) <= t.xmax && fabs(z) <= t.xmax) {
      const int64_t X[3] = {__double2ll_rn(x * t.scale), __double2ll_rn(y * t.scale), __double2ll_rn(z * t.scale)};
      bool all = true;
#pragma unroll 1
      for (int i = sub; i < t.n; i += lanes) {
        uint64_t fb, d[3];
        all &= fixed_plummer(f[i], X, &fb, d);
        const double w = __longlong_as_double((long long)fb);
        ax = fma(w, __longlong_as_double((long long)d[0]), ax);
        ay = fma(w, __longlong_as_double((long long)d[1]), ay);
        az = fma(w, __longlong_as_double((long long)d[2]), az);
      }
      if (!all) {  // the spheres left out above, on whose centres x lies
        for (int i = sub; i < t.n; i += lanes) {
          uint64_t fb, d[3];
          if (!fixed_plummer(f[i], X, &fb, d)) comp_grad(comps[t.at[i]], x, y, z, ax, ay, az);
        }
      }
    } else {
      for (int i = sub; i < t.n; i += lanes) comp_grad(comps[t.at[i]], x, y, z, ax, ay, az);
    }
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
      milky_way.grad(x, y, z, hx, hy, hz);
      ax += hx;
      ay += hy;
      az += hz;
    }
    gx = ax;
    gy = ay;
    gz = az;
  }
};

}  // namespace gal
