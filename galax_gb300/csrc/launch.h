// Host-side launchers shared between the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include "integrate.cuh"

namespace gal {

struct LaunchShape {
  int block_threads;  // 0 = default
  int blocks_per_sm;  // 0 = occupancy maximum
  int variant;        // Milky Way kernel: 0 = up to 255 registers, 1 = at most 128 (more warps)
  int table_lanes;    // component tables: 0 = automatic, 1 = one thread per orbit, 32 = one warp per orbit
};

// Component tables with at least this many components may run one warp per orbit.
constexpr int kWarpMinComponents = 32;

cudaError_t launch_integrate_dopri5(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps,
                                    int ncomp, LaunchShape shape, cudaStream_t stream);
cudaError_t launch_integrate_dopri8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps,
                                    int ncomp, LaunchShape shape, cudaStream_t stream);

// Four-warp teams (16 orbits per block) for a Milky Way Dopri5 batch: queue
// positions [0, 16 blocks) in stripes, then base + atomicAdd(a.queue). smem:
// dynamic shared memory requested (unused) to keep other kernels off the
// blocks' SMs.
cudaError_t launch_integrate_team(const IntegrateArgs& a, const MWParams& p, long long base, int blocks, size_t smem,
                                  cudaStream_t stream);
// The one-thread Milky Way Dopri5 kernel, `block` threads per block, `grid`
// blocks, each requesting `smem` bytes (unused) so that blocks of this launch
// and of the team launch never share an SM.
cudaError_t launch_integrate_dopri5_exclusive(const IntegrateArgs& a, const MWParams& p, int variant, int block,
                                              int grid, size_t smem, cudaStream_t stream);
// The same two launches for a Dopri8 batch.
cudaError_t launch_integrate_team8(const IntegrateArgs& a, const MWParams& p, long long base, int blocks, size_t smem,
                                   cudaStream_t stream);
cudaError_t launch_integrate_dopri8_exclusive(const IntegrateArgs& a, const MWParams& p, int variant, int block,
                                              int grid, size_t smem, cudaStream_t stream);
// Dopri8 saves left to a.defer (put_deferred_save), after the integration on the same stream.
cudaError_t launch_deferred_saves8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   cudaStream_t stream);
// Whether such a batch runs one warp per orbit, whose sums have another order than one thread's.
bool dopri8_warp_per_orbit(const LaunchShape& shape, int64_t n, int ncomp);
// Batches of at most this many orbits per SM run on teams alone.
constexpr int kTeamOrbitsPerSm = 4 * kTeamLanes;
constexpr size_t kExclusiveSmem = 120 * 1024;

int device_sm_count();

}  // namespace gal
