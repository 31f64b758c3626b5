// C ABI of the galax_gb300 library (declared in include/galax_gb300.h):
// potential handles, batched potential / gradient / Hessian evaluation, the
// orbit-integration entry point and small utilities.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/galax_gb300.h"
#include "handle.h"
#include "launch.h"

namespace gal {

thread_local std::string g_last_error;
// SMs given to four-warp teams for the longest orbits (gal_set_team), or -1: as
// many as the first pass's step counts suggest; atomic because calls on other
// threads may read it while it is set
static std::atomic<int> g_team_blocks{-1};
// Fraction of every span the first pass of the two-pass schedule covers
// (gal_set_split_fraction), in millionths
static std::atomic<int> g_split_ppm{100000};

// Launch shape per [method == 8][adaptive], set by gal_set_launch. Dopri5 fits
// 3 blocks of 128 per SM without spills (variant 0); Dopri8 needs the uncapped
// variant 2 to avoid spilling. Adaptive batches default to one warp per SM
// sub-partition (128 threads, one block per SM): their longest orbits then run
// at their own latency instead of sharing an FP64 pipe. Read and written under
// g_shape_mu so that a shape is never seen half-set.
static LaunchShape g_shape[2][2] = {{{0, 0, 0, 0}, {128, 1, 2, 0}}, {{0, 0, 2, 0}, {128, 1, 2, 0}}};
static std::mutex g_shape_mu;

// Component tables: 0 = choose one thread or one warp per orbit automatically,
// 1 / 32 = always that (gal_set_table_lanes).
static std::atomic<int> g_table_lanes{0};

static LaunchShape launch_shape(int method, int adaptive) {
  std::lock_guard<std::mutex> lock(g_shape_mu);
  LaunchShape s = g_shape[method == 8][adaptive ? 1 : 0];
  s.table_lanes = g_table_lanes.load(std::memory_order_relaxed);
  return s;
}

gal_status fail(gal_status st, const std::string& msg) {
  g_last_error = msg;
  return st;
}

gal_status cuda_fail(cudaError_t e, const char* where) {
  return fail(GAL_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

// SM count of the current device, looked up once per device (so that launches
// made while a stream is being captured query nothing)
int device_sm_count() {
  static std::atomic<int> cache[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int sms = cache[dev].load(std::memory_order_relaxed);
  if (sms <= 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    cache[dev].store(sms, std::memory_order_relaxed);
  }
  return sms;
}

static DevComp fold(const gal_component& c, double G) {
  return fold_comp(c.kind, c.m, c.l1, c.l2, c.origin[0], c.origin[1], c.origin[2], G);
}

static bool milky_way_shape(const gal_component* c, int n) {
  if (n != 4) return false;
  const int32_t want[4] = {MIYAMOTO_NAGAI, NFW, HERNQUIST, HERNQUIST};
  for (int i = 0; i < 4; ++i) {
    if (c[i].kind != want[i]) return false;
    if (c[i].origin[0] != 0.0 || c[i].origin[1] != 0.0 || c[i].origin[2] != 0.0) return false;
  }
  return true;
}

static MWParams mw_params(const gal_component* c, double G) {
  MWParams p{};
  p.Gm_d = G * c[0].m;
  p.a_d = c[0].l1;
  p.b2_d = c[0].l2 * c[0].l2;
  p.Gm_h = G * c[1].m;
  p.rs_h = c[1].l1;
  p.irs_h = 1.0 / c[1].l1;
  p.Gm_b = G * c[2].m;
  p.rs_b = c[2].l1;
  p.Gm_n = G * c[3].m;
  p.rs_n = c[3].l1;
  return p;
}

// The table's Plummer spheres in fixed point (fixed_plummer.cuh), if they are
// many; p->fixed.n = 0 otherwise. Allocates on the first call for a handle (the
// number and kinds of components never change).
static cudaError_t build_fixed(gal_potential* p) {
  p->fixed = FixedTable{};
  std::vector<int32_t> at, other;
  for (int i = 0; i < p->n; ++i) (p->comps[i].kind == GAL_PLUMMER ? at : other).push_back(i);
  if ((int)at.size() < kWarpMinComponents) return cudaSuccess;
  std::vector<FixedPlummer> h(at.size());
  for (size_t i = 0; i < at.size(); ++i) {
    const gal_component& c = p->comps[at[i]];
    h[i] = fixed_record(c.origin, c.l1, p->G * c.m);
  }
  FixedOthers o{};
  if (other.size() == 4) {
    gal_component four[4];
    for (int i = 0; i < 4; ++i) four[i] = p->comps[other[i]];
    o.is_mw = milky_way_shape(four, 4) ? 1 : 0;
    if (o.is_mw) o.mw = mw_params(four, p->G);
  }
  at.insert(at.end(), other.begin(), other.end());
  // records, the others' values, indices: one copy, so that a launch finds them all as they were or as they are
  const size_t records = sizeof(FixedPlummer) * h.size(), values = 128;
  static_assert(sizeof(FixedOthers) <= 128, "FixedOthers");
  std::vector<char> image(records + values + sizeof(int32_t) * at.size());
  std::memcpy(image.data(), h.data(), records);
  std::memcpy(image.data() + records, &o, sizeof(o));
  std::memcpy(image.data() + records + values, at.data(), sizeof(int32_t) * at.size());
  cudaError_t e = cudaSuccess;
  if (!p->d_fixed) e = cudaMalloc(&p->d_fixed, image.size());
  if (e != cudaSuccess) {
    p->d_fixed = nullptr;
    return e;
  }
  e = cudaMemcpy(p->d_fixed, image.data(), image.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return e;
  char* base = static_cast<char*>(p->d_fixed);
  p->fixed.f = reinterpret_cast<const FixedPlummer*>(base);
  p->fixed.others = reinterpret_cast<const FixedOthers*>(base + records);
  p->fixed.at = reinterpret_cast<const int32_t*>(base + records + values);
  p->fixed.n = (int)h.size();
  p->fixed.nother = (int)other.size();
  return cudaSuccess;
}

static gal_status validate_components(const gal_component* comps, int32_t n) {
  if (!comps || n < 1) return fail(GAL_ERR_INVALID_ARGUMENT, "need at least one component");
  if (n > GAL_MAX_COMPONENTS) return fail(GAL_ERR_TOO_LARGE, "too many components (max GAL_MAX_COMPONENTS)");
  for (int i = 0; i < n; ++i) {
    const gal_component& c = comps[i];
    if (c.kind < GAL_KEPLER || c.kind > GAL_POWERLAW_CUTOFF)
      return fail(GAL_ERR_UNSUPPORTED, "unsupported component kind");
    if (c.flags != 0) return fail(GAL_ERR_INVALID_ARGUMENT, "component flags must be 0");
    const double v[6] = {c.m, c.l1, c.l2, c.origin[0], c.origin[1], c.origin[2]};
    for (double x : v)
      if (!std::isfinite(x)) return fail(GAL_ERR_INVALID_ARGUMENT, "non-finite component parameter");
    if ((c.kind == GAL_HERNQUIST || c.kind == GAL_NFW) && !(c.l1 > 0.0))
      return fail(GAL_ERR_INVALID_ARGUMENT, "r_s must be > 0");
    // a < 0 occurs in the three-disk (MN3) fits; a > -b keeps sqrt(z^2 + b^2) + a > 0
    if (c.kind == GAL_MIYAMOTO_NAGAI && !(c.l2 > 0.0 && c.l1 > -c.l2))
      return fail(GAL_ERR_INVALID_ARGUMENT, "Miyamoto-Nagai needs b > 0 and a > -b");
    if (c.kind == GAL_PLUMMER && c.l1 < 0.0) return fail(GAL_ERR_INVALID_ARGUMENT, "Plummer r_s must be >= 0");
    if ((c.kind == GAL_ISOCHRONE || c.kind == GAL_LOGARITHMIC) && !(c.l1 > 0.0))
      return fail(GAL_ERR_INVALID_ARGUMENT, "isochrone b / logarithmic r_s must be > 0");
    if (c.kind == GAL_POWERLAW_CUTOFF && (!(c.l1 > 0.0) || !(c.l2 >= 0.0 && c.l2 < 2.0)))
      return fail(GAL_ERR_INVALID_ARGUMENT, "power law with cutoff needs r_c > 0 and 0 <= alpha < 2");
  }
  return GAL_OK;
}

// ----------------------------------------------------------------- eval kernels
// Positions with any strides: component j of point i at x[i sp + j sa].
struct Points {
  const double* x;
  int64_t sp, sa;
  __device__ __forceinline__ double operator()(int64_t i, int j) const { return __ldg(x + i * sp + j * sa); }
};

template <class Pot>
__device__ __forceinline__ void eval_gradient(const Pot& pot, const Points& x, int64_t n, double* __restrict__ out,
                                              double sign) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double gx, gy, gz;
    pot.grad(x(i, 0), x(i, 1), x(i, 2), gx, gy, gz);
    out[i] = sign * gx;
    out[n + i] = sign * gy;
    out[2 * n + i] = sign * gz;
  }
}

__global__ void k_eval_gradient_mw(MWPot pot, Points x, int64_t n, double* __restrict__ out, double sign) {
  eval_gradient(pot, x, n, out, sign);
}

// Components staged into shared memory, refolded at time t when time-dependent.
__device__ __forceinline__ void stage_at_time(const DevComp* comps, const DevLinear* lin, int ncomp, double t,
                                              DevComp* s) {
  for (int i = threadIdx.x; i < ncomp; i += blockDim.x) s[i] = lin ? comp_at_time(comps[i], lin[i], t) : comps[i];
}

__global__ void k_eval_gradient_table(const DevComp* comps, const DevLinear* lin, double t, int ncomp, Points x,
                                      int64_t n, double* __restrict__ out, double sign) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s = reinterpret_cast<DevComp*>(smem_raw);
  stage_at_time(comps, lin, ncomp, t, s);
  __syncthreads();
  eval_gradient(TablePot{s, ncomp}, x, n, out, sign);
}

__global__ void k_eval_phi(const DevComp* comps, const DevLinear* lin, double t, int ncomp, Points x, int64_t n,
                           double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s = reinterpret_cast<DevComp*>(smem_raw);
  stage_at_time(comps, lin, ncomp, t, s);
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double phi = 0.0;
    for (int c = 0; c < ncomp; ++c) phi += comp_phi(s[c], x(i, 0), x(i, 1), x(i, 2));
    out[i] = phi;
  }
}

__device__ __forceinline__ void eval_hessian(const DevComp* s, int ncomp, const Points& x, int64_t n,
                                             double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double H[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = 0; c < ncomp; ++c) comp_hessian(s[c], x(i, 0), x(i, 1), x(i, 2), H);
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k * n + i] = H[k];
  }
}

__global__ void k_eval_hessian(const DevComp* comps, const DevLinear* lin, double t, int ncomp, Points x, int64_t n,
                               double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s = reinterpret_cast<DevComp*>(smem_raw);
  stage_at_time(comps, lin, ncomp, t, s);
  __syncthreads();
  eval_hessian(s, ncomp, x, n, out);
}

// The Milky Way's Hessian, FP64-bound: one radius, one logarithm and one
// reciprocal for the three spheres, reciprocal square roots instead of roots and
// quotients, and the six distinct entries, where the component table's general
// code takes a root per component, about a dozen quotients and nine entries.
// Positions are read where they are instead of from a transposed copy. 4,194,304
// points: 2.23 -> 0.80 ms. Against extended precision, of |H| at 200,000 points:
// rms error 3.4e-16 (3.5e-16 by the general code), largest 3.7e-15 (5.7e-15).
// The parameters come from the component table in device memory, so that a
// captured call sees gal_potential_update; one that moved a component off the centre
// leaves the general code.
__global__ void __launch_bounds__(128) k_eval_hessian_mw(const DevComp* comps, Points x, int64_t n,
                                                         double* __restrict__ out) {
  if (!(comps[0].centered && comps[1].centered && comps[2].centered && comps[3].centered)) {
    eval_hessian(comps, 4, x, n, out);
    return;
  }
  const MWParams p = mw_of_table(comps);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double H[6];
    mw_hessian(p, x(i, 0), x(i, 1), x(i, 2), H);
    out[i] = H[0];
    out[n + i] = H[1];
    out[2 * n + i] = H[2];
    out[3 * n + i] = H[1];
    out[4 * n + i] = H[3];
    out[5 * n + i] = H[4];
    out[6 * n + i] = H[2];
    out[7 * n + i] = H[4];
    out[8 * n + i] = H[5];
  }
}

__global__ void k_fp64_probe(int64_t iters, double seed, double* sink) {
  double a0 = seed + threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6,
         a7 = a0 + 7;
  const double m = 0.999999999, c = 1e-9;
  for (int64_t i = 0; i < iters; ++i) {
    a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
    a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
  }
  const double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.678) sink[threadIdx.x] = s;  // keep the chain alive
}

gal_status validate_cfg(const gal_solver_config* c) {
  if (!c) return fail(GAL_ERR_INVALID_ARGUMENT, "config is NULL");
  if (c->method != 5 && c->method != 8) return fail(GAL_ERR_UNSUPPORTED, "method must be 5 (Dopri5) or 8 (Dopri8)");
  if (c->schedule != 0 && c->schedule != 1) return fail(GAL_ERR_INVALID_ARGUMENT, "schedule must be 0 or 1");
  if (c->max_steps < 1) return fail(GAL_ERR_INVALID_ARGUMENT, "max_steps must be >= 1");
  if (!c->adaptive && !(c->dt0 > 0.0)) return fail(GAL_ERR_INVALID_ARGUMENT, "constant step needs dt0 > 0");
  if (c->adaptive) {
    if (!(c->rtol >= 0.0) || !(c->atol >= 0.0) || (c->rtol == 0.0 && c->atol == 0.0))
      return fail(GAL_ERR_INVALID_ARGUMENT, "rtol/atol must be >= 0 and not both 0");
    if (!(c->safety > 0.0) || !(c->factormin > 0.0) || !(c->factormax >= 1.0))
      return fail(GAL_ERR_INVALID_ARGUMENT, "bad safety/factormin/factormax");
  }
  return GAL_OK;
}

// ---- two-phase schedule: order parked orbits by estimated remaining work
constexpr int kBuckets = 120;  // sixths of an octave of remaining step attempts
// The first pass ends an orbit's part after this many step attempts at the
// latest: the longest orbits' rates are known by then, and a tenth of their spans
// would be thousands of steps, in which most lanes have nothing left to do
// (uneven orbits, s. Dopri5, 65,536 of them: 0.59 at 512, 0.59-0.70 at 256, 0.60 at
// 1024, 0.65 without this bound. Dopri8 at 256 / 512 / 1024 / without: 16,384 of
// them 0.41 / 0.42 / 0.44 / 0.48, 65,536 0.60 / 0.58 / 0.61 / 0.64, 262,144 1.35 /
// 1.22 / 1.22 / 1.30).
constexpr int kParkSteps = 512;
// Lone-thread to team time per step attempt. Dopri8, two batches of 65,536 uneven
// orbits, s: 0.76 and 0.83 with 2.5, 0.62 and 0.67 with 3.0, 0.59 and 0.58 with 3.5,
// 0.56 and 0.56 with 4.0 and 4.5; 262,144 of them 1.36 with 2.5 and 3.0, 1.22 above.
constexpr float kTeamRatio5 = 2.7f, kTeamRatio8 = 4.0f;

__global__ void k_sched_keys(const OrbitResume* __restrict__ r, int64_t n, unsigned* __restrict__ hist,
                             int* __restrict__ bucket) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (r[i].paused) {
      const double p = r[i].progress;
      const double key = (double)r[i].nsteps * (1.0 - p) / fmax(p, 1e-12);
      int b = (int)(6.0f * log2f(1.0f + (float)key));
      b = b < 0 ? 0 : (b >= kBuckets ? kBuckets - 1 : b);
      bucket[i] = b;
      atomicAdd(&hist[b], 1u);
    } else {
      bucket[i] = -1;
    }
  }
}

// Step attempts of an orbit in bucket b: its lower edge times 2^(part / 6).
__device__ __forceinline__ float bucket_work(int b, float part) { return exp2f(((float)b + part) / 6.0f) - 1.0f; }

// Bucket cursors, most remaining work first, and the number of SMs that get a
// team (one warp).
//
// A team's attempt takes 1 / ratio of a lone thread's, but an SM runs 16 orbits
// on a team and 128 without. With t teams taking the 16 t longest orbits, the
// batch ends no earlier than its longest orbit on a team, the longest other one
// on a thread, and the whole work at the SMs' joint rate; t is the smallest
// number that minimises the latest of the three. Measured (Dopri5, s): 65,536
// uneven orbits 0.77 with 48 SMs, 0.59 with 64, 0.60 with 80 and 96, and 0.57 with
// this choice; 262,144 of them 1.19 with 32, 1.22 with 64, 1.50 with 96, and 1.14.
__global__ void k_sched_scan(const unsigned* __restrict__ hist, unsigned* __restrict__ cursor,
                             unsigned long long* __restrict__ qlen, unsigned* __restrict__ teams, int sms,
                             int fixed_teams, float ratio) {
  const int lane = threadIdx.x;
  if (lane == 0) {
    unsigned acc = 0;
    for (int b = kBuckets - 1; b >= 0; --b) {
      cursor[b] = acc;
      acc += hist[b];
    }
    *qlen = acc;
  }
  if (fixed_teams >= 0) {
    if (lane == 0) *teams = (unsigned)fixed_teams;
    return;
  }
  float total = 0.f, longest = 0.f;
  for (int b = 0; b < kBuckets; ++b) {
    const float w = bucket_work(b, 0.5f);
    total += (float)hist[b] * w;
    if (hist[b]) longest = w;
  }
  float best = 3.4e38f;
  int best_t = 0;
  for (int t = lane; t < sms; t += 32) {
    unsigned left = 16u * (unsigned)t;  // orbits the teams take
    int b = kBuckets - 1;
    while (b > 0 && left >= hist[b]) left -= hist[b--];  // b: bucket of the longest one on a thread
    const float tail = bucket_work(b, 1.0f) * ratio;
    const float rate = (float)(sms - t) * (128.f / ratio) + (float)t * 16.f;
    const float end = fmaxf(fmaxf(t > 0 ? longest : longest * ratio, tail), total / rate);
    if (end < best) {
      best = end;
      best_t = t;
    }
  }
  for (int m = 16; m >= 1; m >>= 1) {
    const float e = __shfl_xor_sync(0xffffffffu, best, m);
    const int t = __shfl_xor_sync(0xffffffffu, best_t, m);
    if (e < best || (e == best && t < best_t)) {
      best = e;
      best_t = t;
    }
  }
  if (lane == 0) *teams = (unsigned)best_t;
}

__global__ void k_sched_scatter(const int* __restrict__ bucket, int64_t n, unsigned* __restrict__ cursor,
                                int32_t* __restrict__ order) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int b = bucket[i];
    if (b >= 0) order[atomicAdd(&cursor[b], 1u)] = (int32_t)i;
  }
}

constexpr size_t kSchedHeader = 1024;
static_assert(16 + 8 * kBuckets + 4 <= kSchedHeader, "schedule header");

struct SchedLayout {
  size_t header, resume, bucket, order, total;
};

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

static SchedLayout sched_layout(int64_t n) {
  SchedLayout L{};
  L.header = 0;  // queue counter, queue length, hist[kBuckets], cursor[kBuckets], teams
  L.resume = kSchedHeader;
  L.bucket = L.resume + align256(sizeof(OrbitResume) * (size_t)n);
  L.order = L.bucket + align256(sizeof(int) * (size_t)n);
  L.total = L.order + align256(sizeof(int32_t) * (size_t)n);
  return L;
}

static void grid_for(int64_t n, int block, unsigned* grid) {
  int64_t g = (n + block - 1) / block;
  const int64_t cap = (int64_t)device_sm_count() * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  *grid = (unsigned)g;
}

}  // namespace gal

using namespace gal;


extern "C" {

int32_t gal_abi_version(void) { return 1; }

const char* gal_last_error(void) { return g_last_error.c_str(); }

const char* gal_status_string(int32_t st) {
  switch (st) {
    case GAL_OK: return "ok";
    case GAL_ERR_INVALID_ARGUMENT: return "invalid argument";
    case GAL_ERR_UNSUPPORTED: return "unsupported";
    case GAL_ERR_CUDA: return "CUDA error";
    case GAL_ERR_WORKSPACE: return "workspace too small";
    case GAL_ERR_TOO_LARGE: return "size beyond the supported maximum";
    case GAL_ERR_HOST_ALLOC: return "host allocation failed";
    default: return "unknown status";
  }
}

gal_status gal_potential_create(const gal_component* comps, int32_t n, double G, gal_potential** out) {
  return no_throw([&]() -> gal_status {
    if (!out) return fail(GAL_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    gal_status st = validate_components(comps, n);
    if (st != GAL_OK) return st;
    if (!(G > 0.0) || !std::isfinite(G)) return fail(GAL_ERR_INVALID_ARGUMENT, "G must be finite and > 0");
    std::unique_ptr<gal_potential> holder(new gal_potential());
    gal_potential* p = holder.get();
    p->comps.assign(comps, comps + n);
    p->G = G;
    p->n = n;
    p->is_mw = milky_way_shape(comps, n);
    p->mw = p->is_mw ? mw_params(comps, G) : MWParams{};
    std::vector<DevComp> h(n);
    for (int i = 0; i < n; ++i) h[i] = fold(comps[i], G);
    cudaError_t e = cudaMalloc(&p->d_comps, sizeof(DevComp) * n);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(component table)");
    e = cudaMemcpy(p->d_comps, h.data(), sizeof(DevComp) * n, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      cudaFree(p->d_comps);
      return cuda_fail(e, "cudaMemcpy(component table)");
    }
    e = build_fixed(p);
    if (e != cudaSuccess) {
      cudaFree(p->d_comps);
      cudaFree(p->d_fixed);
      return cuda_fail(e, "fixed-point table");
    }
    *out = holder.release();
    return GAL_OK;
  });
}

gal_status gal_potential_destroy(gal_potential* p) {
  if (!p) return GAL_OK;
  cudaError_t e = cudaFree(p->d_comps);
  if (p->d_fixed) {
    const cudaError_t e1 = cudaFree(p->d_fixed);
    if (e == cudaSuccess) e = e1;
  }
  if (p->d_lin) {
    const cudaError_t e2 = cudaFree(p->d_lin);
    if (e == cudaSuccess) e = e2;
  }
  delete p;
  return e == cudaSuccess ? GAL_OK : cuda_fail(e, "cudaFree(component table)");
}

gal_status gal_potential_set_linear(gal_potential* p, const double* slopes) {
  return no_throw([&]() -> gal_status {
    if (!p) return fail(GAL_ERR_INVALID_ARGUMENT, "potential is NULL");
    if (slopes) {
      for (int i = 0; i < 3 * p->n; ++i)
        if (!std::isfinite(slopes[i])) return fail(GAL_ERR_INVALID_ARGUMENT, "non-finite slope");
    }
    bool any = false;
    std::vector<DevLinear> h(p->n);
    for (int i = 0; i < p->n; ++i) {
      const gal_component& c = p->comps[i];
      DevLinear& L = h[i];
      L.kind = c.kind;
      L.m0 = c.m;
      L.l10 = c.l1;
      L.l20 = c.l2;
      L.G = p->G;
      L.dm = slopes ? slopes[3 * i] : 0.0;
      L.dl1 = slopes ? slopes[3 * i + 1] : 0.0;
      L.dl2 = slopes ? slopes[3 * i + 2] : 0.0;
      L.active = (L.dm != 0.0 || L.dl1 != 0.0 || L.dl2 != 0.0) ? 1 : 0;
      any = any || L.active;
    }
    if (p->d_lin) {
      cudaError_t e = cudaFree(p->d_lin);
      p->d_lin = nullptr;
      if (e != cudaSuccess) return cuda_fail(e, "cudaFree(linear table)");
    }
    (void)any;
    if (slopes) {  // time-dependent even when every slope is zero: the adjoint then gives d/d(slope)
      cudaError_t e = cudaMalloc(&p->d_lin, sizeof(DevLinear) * p->n);
      if (e != cudaSuccess) {
        p->d_lin = nullptr;
        return cuda_fail(e, "cudaMalloc(linear table)");
      }
      e = cudaMemcpy(p->d_lin, h.data(), sizeof(DevLinear) * p->n, cudaMemcpyHostToDevice);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy(linear table)");
    }
    // the specialised Milky Way model has constant parameters
    p->is_mw = !p->d_lin && milky_way_shape(p->comps.data(), p->n);
    return GAL_OK;
  });
}

gal_status gal_potential_update(gal_potential* p, const gal_component* comps, int32_t n, gal_stream_t stream) {
  return no_throw([&]() -> gal_status {
    if (!p) return fail(GAL_ERR_INVALID_ARGUMENT, "potential is NULL");
    if (n != p->n) return fail(GAL_ERR_INVALID_ARGUMENT, "component count differs from the handle's");
    gal_status st = validate_components(comps, n);
    if (st != GAL_OK) return st;
    for (int i = 0; i < n; ++i)
      if (comps[i].kind != p->comps[i].kind) return fail(GAL_ERR_INVALID_ARGUMENT, "component kinds differ");
    std::vector<DevComp> h(n);
    for (int i = 0; i < n; ++i) h[i] = fold(comps[i], p->G);
    // pageable source: the call returns once the bytes are staged, so h may go out of scope
    cudaError_t e = cudaMemcpyAsync(p->d_comps, h.data(), sizeof(DevComp) * n, cudaMemcpyHostToDevice,
                                    (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(component table)");
    e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
    p->comps.assign(comps, comps + n);
    p->is_mw = !p->d_lin && milky_way_shape(comps, n);
    p->mw = milky_way_shape(comps, n) ? mw_params(comps, p->G) : MWParams{};
    e = build_fixed(p);
    if (e != cudaSuccess) return cuda_fail(e, "fixed-point table");
    if (p->d_lin) {  // new values at t = 0, same slopes
      std::vector<DevLinear> L(n);
      e = cudaMemcpy(L.data(), p->d_lin, sizeof(DevLinear) * n, cudaMemcpyDeviceToHost);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy(linear table)");
      for (int i = 0; i < n; ++i) {
        L[i].m0 = comps[i].m;
        L[i].l10 = comps[i].l1;
        L[i].l20 = comps[i].l2;
      }
      e = cudaMemcpy(p->d_lin, L.data(), sizeof(DevLinear) * n, cudaMemcpyHostToDevice);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy(linear table)");
    }
    return GAL_OK;
  });
}

int32_t gal_potential_num_components(const gal_potential* p) { return p ? p->n : 0; }
int32_t gal_potential_is_milky_way(const gal_potential* p) { return p && p->is_mw ? 1 : 0; }

int32_t gal_potential_is_time_dependent(const gal_potential* p) { return time_dependent(p) ? 1 : 0; }

gal_status gal_eval_points(const gal_potential* p, int32_t what, const double* x, int64_t point_stride,
                           int64_t axis_stride, double t, int64_t n, double* out, gal_stream_t stream) {
  if (!p || (!x && n) || (!out && n) || n < 0) return fail(GAL_ERR_INVALID_ARGUMENT, "bad pointer or size");
  if (what < GAL_EVAL_POTENTIAL || what > GAL_EVAL_HESSIAN) return fail(GAL_ERR_INVALID_ARGUMENT, "unknown quantity");
  if (n == 0) return GAL_OK;
  const Points pts{x, point_stride, axis_stride};
  const cudaStream_t s = (cudaStream_t)stream;
  const int block = what == GAL_EVAL_HESSIAN ? 128 : 256;
  unsigned grid;
  grid_for(n, block, &grid);
  const size_t smem = sizeof(DevComp) * p->n;
  auto room = [&](const void* kernel) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  };
  const double sign = what == GAL_EVAL_ACCELERATION ? -1.0 : 1.0;
  switch (what) {
    case GAL_EVAL_POTENTIAL:
      room((const void*)k_eval_phi);
      k_eval_phi<<<grid, block, smem, s>>>(p->d_comps, p->d_lin, t, p->n, pts, n, out);
      break;
    case GAL_EVAL_HESSIAN:
      if (p->is_mw) {
        k_eval_hessian_mw<<<grid, block, 0, s>>>(p->d_comps, pts, n, out);
      } else {
        room((const void*)k_eval_hessian);
        k_eval_hessian<<<grid, block, smem, s>>>(p->d_comps, p->d_lin, t, p->n, pts, n, out);
      }
      break;
    default:
      if (p->is_mw) {
        k_eval_gradient_mw<<<grid, block, 0, s>>>(MWPot{p->mw}, pts, n, out, sign);
      } else {
        room((const void*)k_eval_gradient_table);
        k_eval_gradient_table<<<grid, block, smem, s>>>(p->d_comps, p->d_lin, t, p->n, pts, n, out, sign);
      }
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GAL_OK : cuda_fail(e, "potential evaluation launch");
}

gal_status gal_eval_gradient(const gal_potential* p, const double* x, double t, int64_t n, double* out,
                             gal_stream_t stream) {
  return gal_eval_points(p, GAL_EVAL_GRADIENT, x, 1, n, t, n, out, stream);
}

gal_status gal_eval_acceleration(const gal_potential* p, const double* x, double t, int64_t n, double* out,
                                 gal_stream_t stream) {
  return gal_eval_points(p, GAL_EVAL_ACCELERATION, x, 1, n, t, n, out, stream);
}

gal_status gal_eval_potential(const gal_potential* p, const double* x, double t, int64_t n, double* phi,
                              gal_stream_t stream) {
  return gal_eval_points(p, GAL_EVAL_POTENTIAL, x, 1, n, t, n, phi, stream);
}

gal_status gal_eval_hessian(const gal_potential* p, const double* x, double t, int64_t n, double* out,
                            gal_stream_t stream) {
  return gal_eval_points(p, GAL_EVAL_HESSIAN, x, 1, n, t, n, out, stream);
}

gal_status gal_integrate_workspace_size(const gal_solver_config* cfg, int64_t n, size_t* bytes) {
  if (!bytes || !cfg || n < 0) return fail(GAL_ERR_INVALID_ARGUMENT, "bad workspace query");
  *bytes = cfg->schedule ? sched_layout(n).total : 256;  // one 8-byte work-queue counter, padded
  return GAL_OK;
}

gal_status gal_integrate_workspace_size_saves(const gal_solver_config* cfg, int64_t n, int64_t total_saves,
                                              size_t* bytes) {
  if (total_saves < 0) return fail(GAL_ERR_INVALID_ARGUMENT, "bad workspace query");
  const gal_status st = gal_integrate_workspace_size(cfg, n, bytes);
  if (st == GAL_OK && cfg->method == 8) *bytes = align256(*bytes) + sizeof(double) * (size_t)total_saves;
  return st;
}

gal_status gal_set_team(int32_t blocks) {
  if (blocks < -1 || blocks > 1024) return fail(GAL_ERR_INVALID_ARGUMENT, "team blocks must be in [-1, 1024]");
  g_team_blocks.store(blocks, std::memory_order_relaxed);
  return GAL_OK;
}

gal_status gal_set_split_fraction(double fraction) {
  if (!(fraction >= 1e-3 && fraction <= 0.9)) return fail(GAL_ERR_INVALID_ARGUMENT, "fraction must be in [0.001, 0.9]");
  g_split_ppm.store((int)(fraction * 1e6 + 0.5), std::memory_order_relaxed);
  return GAL_OK;
}

gal_status gal_set_table_lanes(int32_t lanes) {
  if (lanes != 0 && lanes != 1 && lanes != 32) return fail(GAL_ERR_INVALID_ARGUMENT, "lanes must be 0, 1 or 32");
  g_table_lanes.store(lanes, std::memory_order_relaxed);
  return GAL_OK;
}

gal_status gal_set_launch(int32_t method, int32_t adaptive, int32_t block_threads, int32_t blocks_per_sm,
                          int32_t variant) {
  if ((method != 5 && method != 8) || block_threads < 0 || block_threads > 256 || (block_threads % 32) ||
      blocks_per_sm < 0 || variant < 0 || variant > 2 || (variant != 2 && block_threads > 128))
    return fail(GAL_ERR_INVALID_ARGUMENT, "bad launch shape");
  std::lock_guard<std::mutex> lock(g_shape_mu);
  g_shape[method == 8][adaptive ? 1 : 0] = LaunchShape{block_threads, blocks_per_sm, variant, 0};
  return GAL_OK;
}

gal_status gal_integrate(const gal_potential* p, const gal_solver_config* cfg, const double* y0, const double* t0,
                         const double* t1, const int64_t* save_offsets, const double* save_ts, int64_t n_saves,
                         double* out, int32_t* status, int64_t* steps, const int32_t* order, int64_t n,
                         void* workspace, size_t workspace_bytes, gal_stream_t stream) {
  if (!p) return fail(GAL_ERR_INVALID_ARGUMENT, "potential is NULL");
  gal_status st = validate_cfg(cfg);
  if (st != GAL_OK) return st;
  if (n < 0) return fail(GAL_ERR_INVALID_ARGUMENT, "n < 0");
  if (n == 0) return GAL_OK;
  if (n > (int64_t)2147483647) return fail(GAL_ERR_TOO_LARGE, "at most 2^31-1 orbits per call");
  if (!y0 || !t0 || !t1) return fail(GAL_ERR_INVALID_ARGUMENT, "y0/t0/t1 NULL");
  if (n_saves < 0) return fail(GAL_ERR_INVALID_ARGUMENT, "n_saves < 0");
  if ((save_offsets || n_saves > 0) && (!save_ts || !out)) return fail(GAL_ERR_INVALID_ARGUMENT, "saves need save_ts and out");
  size_t need = 0;
  gal_integrate_workspace_size(cfg, n, &need);
  if (!workspace || workspace_bytes < need) return fail(GAL_ERR_WORKSPACE, "workspace too small");
  // CSR saves: n_saves is the total count (save_offsets[n]); shared grid: saves per orbit
  const int64_t total = save_offsets ? n_saves : n_saves * n;
  IntegrateArgs a{};
  a.adaptive = cfg->adaptive;
  a.force_dtmin = cfg->force_dtmin;
  a.max_steps = cfg->max_steps;
  a.dt0 = cfg->dt0;
  a.rtol = cfg->rtol;
  a.atol = cfg->atol;
  a.dtmin = cfg->dtmin;
  a.dtmax = cfg->dtmax;
  const double morder = cfg->method == 8 ? 8.0 : 5.0;
  a.c1 = (cfg->icoeff + cfg->pcoeff + cfg->dcoeff) / morder;
  a.c2 = -(cfg->pcoeff + 2.0 * cfg->dcoeff) / morder;
  a.c3 = cfg->dcoeff / morder;
  a.i_controller = (cfg->pcoeff == 0.0 && cfg->dcoeff == 0.0 && cfg->icoeff == 1.0) ? 1 : 0;
  a.safety = cfg->safety;
  a.factormin = cfg->factormin;
  a.factormax = cfg->factormax;
  a.y0 = y0;
  a.t0 = t0;
  a.t1 = t1;
  a.save_offsets = save_offsets;
  a.save_ts = save_ts;
  a.n_saves = n_saves;
  a.out = out;
  a.out_stride = total;
  a.status = status;
  a.steps = steps;
  a.order = order;
  a.n = n;
  a.lin = p->d_lin;
  a.fixed = p->fixed;
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = static_cast<char*>(workspace);
  a.queue = reinterpret_cast<unsigned long long*>(ws);
  a.phase = 0;
  a.split_frac = 0.0;
  a.resume = nullptr;
  a.queue_len = nullptr;
  const LaunchShape shape = launch_shape(cfg->method, cfg->adaptive);
  // Dopri8 saves as one parallel pass afterwards (put_deferred_save) when the
  // workspace has an entry per save. Not for several lanes per orbit, whose component
  // sums a per-save thread would not repeat bit for bit, and not for saves in
  // host memory, which would cross the bus three times.
  if (cfg->method == 8 && total > 0 && workspace_bytes >= align256(need) + sizeof(double) * (size_t)total &&
      (p->is_mw || !dopri8_inline_saves(a, shape, p->n))) {
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, out) != cudaSuccess) {
      cudaGetLastError();
    } else if (attr.type == cudaMemoryTypeDevice) {
      a.defer = reinterpret_cast<double*>(ws + align256(need));
      const cudaError_t em = cudaMemsetAsync(a.defer, 0xff, sizeof(double) * (size_t)total, s);  // NaN: not deferred
      if (em != cudaSuccess) return cuda_fail(em, "clearing the save scratch");
    }
  }
  auto finish = [&](cudaError_t e, const char* what) -> gal_status {
    if (e != cudaSuccess) return cuda_fail(e, what);
    if (!a.defer) return GAL_OK;
    e = launch_deferred_saves8(a, p->is_mw, p->mw, p->d_comps, p->n, s);
    return e == cudaSuccess ? GAL_OK : cuda_fail(e, "deferred saves launch");
  };
  auto launch = [&]() {
    return cfg->method == 8 ? launch_integrate_dopri8(a, p->is_mw, p->mw, p->d_comps, p->n, shape, s)
                            : launch_integrate_dopri5(a, p->is_mw, p->mw, p->d_comps, p->n, shape, s);
  };
  const int sms = device_sm_count();
  const int team_blocks = g_team_blocks.load(std::memory_order_relaxed);
  // Few orbits: all of them on teams, in one pass. A team block's step takes a
  // third of a lone thread's time or less, at 16 orbits per four warps instead
  // of 128; two blocks fit an SM, so 9,728 orbits are two turns of the chip.
  // Measured, constant step, 100 steps, ms on teams / one thread per orbit:
  // Dopri8 1.93 / 6.14 at 2,432 orbits, 2.50 / 6.12 at 4,864, 4.76 / 6.13 at
  // 9,728, 6.99 / 6.13 at 12,160; Dopri5 1.00 / 2.71, 1.26 / 2.71, 2.28 / 2.73,
  // 3.28 / 2.73. Tables at 4,864 and 9,728 orbits, teams' time of the single
  // threads', constant (adaptive) Dopri8: power law with cutoff, disk and halo 0.47
  // and 0.86 (0.48, 0.61), the power law alone 0.50 and 0.94 (0.68, 0.85), the six
  // components of MilkyWayPotential2022 0.33 and 0.63 (0.30, 0.38), sixteen
  // components 0.29 and 0.56 (0.26, 0.34); one component of any other kind 0.51-0.52
  // and 0.98 (0.49, 0.51-0.75), which with Dopri5 is 0.54-0.58 and 1.00-1.02.
  if (team_blocks != 0 && n <= (int64_t)kTeamOrbitsPerSm * sms &&
      (p->is_mw || (p->n <= kTeamMaxComps && shape.table_lanes == 0))) {
    cudaError_t e = cudaMemsetAsync(ws, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return cuda_fail(e, "clearing the work queue");
    int64_t blocks = (n + kTeamLanes - 1) / kTeamLanes;
    if (blocks > 2 * sms) blocks = 2 * sms;
    e = cfg->method == 8 ? launch_integrate_team8(a, p->is_mw, p->mw, p->d_comps, p->n, (int)blocks, s)
                         : launch_integrate_team(a, p->is_mw, p->mw, p->d_comps, p->n, (int)blocks, s);
    return finish(e, "integrate kernel launch (teams)");
  }
  if (!cfg->schedule) {
    cudaError_t e = cudaMemsetAsync(ws, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return cuda_fail(e, "clearing the work queue");
    return finish(launch(), "integrate kernel launch");
  }
  // two phases: a part of every span (at most a tenth by default), then longest remaining work first
  const SchedLayout L = sched_layout(n);
  auto* qlen = reinterpret_cast<unsigned long long*>(ws + 8);
  auto* hist = reinterpret_cast<unsigned*>(ws + 16);
  auto* cursor = reinterpret_cast<unsigned*>(ws + 16 + 4 * kBuckets);
  auto* teams = reinterpret_cast<unsigned*>(ws + 16 + 8 * kBuckets);
  auto* resume = reinterpret_cast<OrbitResume*>(ws + L.resume);
  auto* bucket = reinterpret_cast<int*>(ws + L.bucket);
  auto* order2 = reinterpret_cast<int32_t*>(ws + L.order);
  cudaError_t e = cudaMemsetAsync(ws, 0, L.resume + sizeof(OrbitResume) * (size_t)n, s);
  if (e != cudaSuccess) return cuda_fail(e, "clearing the schedule scratch");
  a.split_frac = 1e-6 * g_split_ppm.load(std::memory_order_relaxed);
  a.park_steps = kParkSteps;
  a.resume = resume;
  e = launch();
  if (e != cudaSuccess) return cuda_fail(e, "integrate kernel launch (first pass)");
  unsigned grid;
  grid_for(n, 256, &grid);
  k_sched_keys<<<grid, 256, 0, s>>>(resume, n, hist, bucket);
  k_sched_scan<<<1, 32, 0, s>>>(hist, cursor, qlen, teams, sms, team_blocks < sms - 1 ? team_blocks : sms - 1,
                                cfg->method == 8 ? kTeamRatio8 : kTeamRatio5);
  k_sched_scatter<<<grid, 256, 0, s>>>(bucket, n, cursor, order2);
  e = cudaMemsetAsync(ws, 0, sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "ordering the parked orbits");
  a.phase = 1;
  a.order = order2;
  a.queue_len = qlen;
  if (p->is_mw && team_blocks != 0 && sms > 1) {
    e = cfg->method == 8 ? launch_integrate_mixed8(a, p->mw, teams, sms, s)
                         : launch_integrate_mixed(a, p->mw, teams, sms, s);
    return finish(e, "integrate kernel launch (second pass, teams)");
  }
  return finish(launch(), "integrate kernel launch (second pass)");
}

int32_t gal_tableau(int32_t method, double* c, double* a, double* b, double* e) {
  if (method != 5 && method != 8) return 0;
  for (int i = 0; i < 13; ++i) {
    c[i] = b[i] = e[i] = 0.0;
    for (int j = 0; j < 13; ++j) a[13 * i + j] = 0.0;
  }
  auto copy = [&](auto tb) {
    using TB = decltype(tb);
    for (int i = 0; i < TB::S; ++i) {
      c[i] = TB::C[i];
      b[i] = TB::B[i];
      e[i] = TB::E[i];
      for (int j = 0; j < TB::S; ++j) a[13 * i + j] = TB::A[i][j];
    }
    return TB::S;
  };
  return method == 5 ? copy(Dopri5{}) : copy(Dopri8{});
}

gal_status gal_fp64_peak_probe(int64_t iters, double* ms, double* flops, gal_stream_t stream) {
  if (iters < 1 || !ms || !flops) return fail(GAL_ERR_INVALID_ARGUMENT, "bad probe arguments");
  const int block = 256;
  const unsigned grid = (unsigned)device_sm_count() * 8;
  double* sink = nullptr;
  cudaError_t e = cudaMalloc(&sink, block * sizeof(double));
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(probe)");
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  k_fp64_probe<<<grid, block, 0, (cudaStream_t)stream>>>(iters / 8 + 1, 1.0, sink);  // warm-up
  cudaEventRecord(a, (cudaStream_t)stream);
  k_fp64_probe<<<grid, block, 0, (cudaStream_t)stream>>>(iters, 1.0, sink);
  cudaEventRecord(b, (cudaStream_t)stream);
  e = cudaEventSynchronize(b);
  float t = 0.f;
  cudaEventElapsedTime(&t, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(sink);
  if (e != cudaSuccess) return cuda_fail(e, "probe");
  *ms = t;
  *flops = 2.0 * 8.0 * (double)iters * (double)grid * (double)block;
  return GAL_OK;
}

// The adjoint entry points live in adjoint.cu.

}  // extern "C"
