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

// A batch on `blocks` four-warp teams (16 orbits per block; at most
// kTeamMaxComps components).
cudaError_t launch_integrate_team(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                  int blocks, cudaStream_t stream);
cudaError_t launch_integrate_team8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   int blocks, cudaStream_t stream);
// The second pass of a Milky Way batch on `blocks` SMs, *teams (device memory) of them
// with a team and the others with one thread per orbit. Every block requests
// kExclusiveSmem bytes of dynamic shared memory, which it does not use, so that
// no two share an SM.
cudaError_t launch_integrate_mixed(const IntegrateArgs& a, const MWParams& p, const unsigned* teams, int blocks,
                                   cudaStream_t stream);
cudaError_t launch_integrate_mixed8(const IntegrateArgs& a, const MWParams& p, const unsigned* teams, int blocks,
                                    cudaStream_t stream);
// Dopri8 saves left to a.defer (put_deferred_save), after the integration on the same stream.
cudaError_t launch_deferred_saves8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   cudaStream_t stream);
// Whether a table's batch runs several lanes per orbit, whose sums one thread per save would not repeat.
bool dopri8_inline_saves(const IntegrateArgs& a, const LaunchShape& shape, int ncomp);
// Batches of at most this many orbits per SM run on teams alone.
constexpr int kTeamOrbitsPerSm = 4 * kTeamLanes;
constexpr size_t kExclusiveSmem = 120 * 1024;

int device_sm_count();

}  // namespace gal
