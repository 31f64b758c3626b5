// Kernel entry points and launcher for one Runge-Kutta method (included once per
// method by integrate_dopri5.cu / integrate_dopri8.cu so the two compile in parallel).
#pragma once

#include "launch.h"
#include "vjp.cuh"

namespace gal {

constexpr int kMaxBlock = 256;

// Register variants of the Milky Way kernel (threads per block <= MAXT):
//   0: 128 threads, 3 blocks per SM  -> at most 168 registers, 12 warps per SM
//   1: 128 threads, 4 blocks per SM  -> at most 128 registers, 16 warps per SM (spills)
//   2: 256 threads, 1 block per SM   -> up to 255 registers
// The autotuner picks per workload; results do not depend on it.
template <class TB, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_integrate_mw(IntegrateArgs a, MWParams p) {
  const MWPot pot{p};
  integrate_loop<TB>(a, pot);
}

template <class TB>
cudaError_t mw_occupancy(int variant, int block, int* per_sm) {
  switch (variant) {
    case 1: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_integrate_mw<TB, 128, 4>, block, 0);
    case 2: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_integrate_mw<TB, 256, 1>, block, 0);
    default: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_integrate_mw<TB, 128, 3>, block, 0);
  }
}

template <class TB>
void mw_launch(int variant, unsigned grid, int block, cudaStream_t stream, const IntegrateArgs& a, const MWParams& p) {
  switch (variant) {
    case 1: k_integrate_mw<TB, 128, 4><<<grid, block, 0, stream>>>(a, p); break;
    case 2: k_integrate_mw<TB, 256, 1><<<grid, block, 0, stream>>>(a, p); break;
    default: k_integrate_mw<TB, 128, 3><<<grid, block, 0, stream>>>(a, p); break;
  }
}

template <class TB, bool TIMED>
__global__ void __launch_bounds__(kMaxBlock) k_integrate_table(IntegrateArgs a, const DevComp* comps, int ncomp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s_comps = reinterpret_cast<DevComp*>(smem_raw);
  for (int i = threadIdx.x; i < ncomp; i += blockDim.x) s_comps[i] = comps[i];
  __syncthreads();
  if constexpr (TIMED) {
    integrate_loop<TB>(a, TimedTablePot{s_comps, ncomp, a.lin});
  } else {
    integrate_loop<TB>(a, TablePot{s_comps, ncomp});
  }
}

// The partial steps that the integration deferred (put_deferred_save): one
// thread per save, all independent. Entries of a.defer without a start time
// (NaN) are saves that were written in place. The arithmetic is the inline
// sub-step's, so saves are the same bits either way. For a static field
// (dir tau_k - tau) dir = ts - t, t = dir tau: exact, the sign is +-1.
template <class TB, class Pot>
__device__ __forceinline__ void deferred_saves(const IntegrateArgs& a, const Pot& pot) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.out_stride;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double t = a.defer[i];
    if (isnan(t)) continue;
    const double hs = (a.save_offsets ? a.save_ts[i] : a.save_ts[i / a.n]) - t;
    double y[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) y[j] = a.out[j * a.out_stride + i];
    rk_step_plain<TB>(pot, y, hs, t);
#pragma unroll
    for (int j = 0; j < 6; ++j) a.out[j * a.out_stride + i] = y[j];
  }
}

template <class TB>
__global__ void __launch_bounds__(128) k_deferred_saves_mw(IntegrateArgs a, MWParams p) {
  deferred_saves<TB>(a, MWPot{p});
}

template <class TB, bool TIMED>
__global__ void __launch_bounds__(128) k_deferred_saves_table(IntegrateArgs a, const DevComp* comps, int ncomp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s_comps = reinterpret_cast<DevComp*>(smem_raw);
  for (int i = threadIdx.x; i < ncomp; i += blockDim.x) s_comps[i] = comps[i];
  __syncthreads();
  if constexpr (TIMED) {
    deferred_saves<TB>(a, TimedTablePot{s_comps, ncomp, a.lin});
  } else {
    deferred_saves<TB>(a, TablePot{s_comps, ncomp});
  }
}

// One warp per block while that gives every SM sub-partition at most one warp.
template <class TB>
cudaError_t launch_deferred_saves(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                  cudaStream_t stream) {
  const int block = a.out_stride > 128LL * device_sm_count() ? 128 : 32;
  const int64_t cap = 64LL * device_sm_count();
  int64_t grid = (a.out_stride + block - 1) / block;
  if (grid > cap) grid = cap;
  if (mw) {
    k_deferred_saves_mw<TB><<<(unsigned)grid, block, 0, stream>>>(a, p);
    return cudaGetLastError();
  }
  const size_t smem = sizeof(DevComp) * (size_t)ncomp;
  auto kernel = a.lin ? k_deferred_saves_table<TB, true> : k_deferred_saves_table<TB, false>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kernel<<<(unsigned)grid, block, smem, stream>>>(a, comps, ncomp);
  return cudaGetLastError();
}

// One warp per orbit (composites with many components): the lanes split the
// components and every lane ends each gradient with the same sum.
template <class TB, bool TIMED>
__global__ void __launch_bounds__(kMaxBlock) k_integrate_table_warp(IntegrateArgs a, const DevComp* comps, int ncomp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DevComp* s_comps = reinterpret_cast<DevComp*>(smem_raw);
  for (int i = threadIdx.x; i < ncomp; i += blockDim.x) s_comps[i] = comps[i];
  __syncthreads();
  integrate_loop<TB, WarpTablePot<TIMED>, 32>(a, WarpTablePot<TIMED>{s_comps, ncomp, a.lin});
}

// Whether a component table runs one warp per orbit: always or never when
// asked (table_lanes 32 / 1); automatically when the table has many components
// and the batch is too small to give every SM sub-partition a warp of 32
// orbits, so that one thread per orbit would leave FP64 pipes idle.
inline bool use_warp_per_orbit(const LaunchShape& shape, int64_t n, int ncomp) {
  if (shape.table_lanes == 32) return true;
  if (shape.table_lanes == 1 || ncomp < kWarpMinComponents) return false;
  return (n + 31) / 32 < 4LL * device_sm_count();
}

// Whether the spheres of a table are evaluated in fixed point: for constant steps
// (an adaptive controller turns another rounding into other steps), unless one
// thread per orbit is asked for. Below 32 spheres nothing is gained over teams and
// single threads.
inline bool use_fixed(const IntegrateArgs& a, const LaunchShape& shape) {
  return !a.adaptive && !a.lin && shape.table_lanes != 1 && a.fixed.n >= kWarpMinComponents;
}

// Four orbits per block of 128 threads and as many blocks per SM as fit (the
// launch shapes tuned for one thread per orbit do not apply).
template <class TB>
cudaError_t launch_integrate_warp(const IntegrateArgs& a, const DevComp* comps, int ncomp, cudaStream_t stream) {
  const int block = 128;
  const size_t smem = sizeof(DevComp) * (size_t)ncomp;
  auto kernel = a.lin ? k_integrate_table_warp<TB, true> : k_integrate_table_warp<TB, false>;
  cudaError_t err;
  if (smem > 48 * 1024) {
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
  }
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) per_sm = 1;
  const int warps = block / 32;
  int64_t grid = (int64_t)per_sm * device_sm_count();
  const int64_t need = (a.n + warps - 1) / warps;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  kernel<<<(unsigned)grid, block, smem, stream>>>(a, comps, ncomp);
  return cudaGetLastError();
}

// Constant-step orbits in a table with many Plummer spheres (fixed_plummer.cuh).
// At most 128 registers, so that four blocks share an SM: the stage slopes that
// spill cost nothing beside hundreds of spheres per gradient, and integer work
// needs several warps per sub-partition to hide its latency. As many lanes per
// orbit as those blocks have room for. 16,384 orbits, Milky Way plus 512 spheres,
// 100 Dopri5 steps: 308 ms with the spheres in FP64 on one warp per orbit, 74 ms
// here, FP64 pipe 87 % busy (68 ms with positions and centres rounded to one grid for the whole table,
// whose error near a sphere grew with the table's extent).
template <class TB>
__global__ void __launch_bounds__(128, 4) k_integrate_fixed(IntegrateArgs a, const DevComp* comps, int lanes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FixedOthers others;
  FixedPlummer* s_f = reinterpret_cast<FixedPlummer*>(smem_raw);
  DevComp* s_o = reinterpret_cast<DevComp*>(s_f + a.fixed.n);
  for (int i = threadIdx.x; i < a.fixed.n; i += blockDim.x) s_f[i] = a.fixed.f[i];
  for (int i = threadIdx.x; i < a.fixed.nother; i += blockDim.x) s_o[i] = comps[a.fixed.at[a.fixed.n + i]];
  if (threadIdx.x == 0) others = *a.fixed.others;
  __syncthreads();
  integrate_loop<TB, FixedTablePot, 0>(a, FixedTablePot{s_f, s_o, &others, comps, a.fixed, lanes});
}

template <class TB>
cudaError_t launch_integrate_fixed(const IntegrateArgs& a, const DevComp* comps, int min_lanes, cudaStream_t stream) {
  const int block = 128;
  const int64_t room = 16LL * 32 * device_sm_count();  // lanes of four blocks per SM
  int lanes = min_lanes;
  while (lanes < 32 && 2 * lanes * a.n <= room) lanes *= 2;
  const size_t smem = sizeof(FixedPlummer) * (size_t)a.fixed.n + sizeof(DevComp) * (size_t)a.fixed.nother;
  auto kernel = k_integrate_fixed<TB>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (int64_t)per_sm * device_sm_count();
  const int64_t need = (a.n * lanes + block - 1) / block;
  if (grid > need) grid = need;
  kernel<<<(unsigned)grid, block, smem, stream>>>(a, comps, lanes);
  return cudaGetLastError();
}

template <class TB>
cudaError_t launch_integrate(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                             LaunchShape shape, cudaStream_t stream) {
  if (!mw && use_fixed(a, shape)) return launch_integrate_fixed<TB>(a, comps, shape.table_lanes == 32 ? 32 : 1, stream);
  if (!mw && use_warp_per_orbit(shape, a.n, ncomp)) return launch_integrate_warp<TB>(a, comps, ncomp, stream);
  const int block = shape.block_threads > 0 ? shape.block_threads : 128;
  if (block > kMaxBlock || block % 32 != 0) return cudaErrorInvalidValue;
  const size_t smem = mw ? 0 : sizeof(DevComp) * (size_t)ncomp;
  int per_sm = shape.blocks_per_sm;
  cudaError_t err;
  if (mw && shape.variant != 2 && block > 128) return cudaErrorInvalidValue;
  if (per_sm <= 0) {
    if (mw)
      err = mw_occupancy<TB>(shape.variant, block, &per_sm);
    else if (a.lin)
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_integrate_table<TB, true>, block, smem);
    else
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_integrate_table<TB, false>, block, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
  }
  int64_t grid = (int64_t)per_sm * device_sm_count();
  const int64_t need = (a.n + block - 1) / block;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  if (mw) {
    mw_launch<TB>(shape.variant, (unsigned)grid, block, stream, a, p);
  } else {
    auto kernel = a.lin ? k_integrate_table<TB, true> : k_integrate_table<TB, false>;
    if (smem > 48 * 1024) {
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (err != cudaSuccess) return err;
    }
    kernel<<<(unsigned)grid, block, smem, stream>>>(a, comps, ncomp);
  }
  return cudaGetLastError();
}

}  // namespace gal
