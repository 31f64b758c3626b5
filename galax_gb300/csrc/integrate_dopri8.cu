// Dopri8 instantiation of the orbit-integration kernels, and the four-warp
// team kernel for the longest orbits of a two-pass Milky Way batch.
#include "integrate_kernels.cuh"
#include "integrate_team.cuh"

namespace gal {
cudaError_t launch_integrate_dopri8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps,
                                    int ncomp, LaunchShape shape, cudaStream_t stream) {
  return launch_integrate<Dopri8>(a, mw, p, comps, ncomp, shape, stream);
}

cudaError_t launch_deferred_saves8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   cudaStream_t stream) {
  return launch_deferred_saves<Dopri8>(a, mw, p, comps, ncomp, stream);
}

bool dopri8_warp_per_orbit(const LaunchShape& shape, int64_t n, int ncomp) {
  return use_warp_per_orbit(shape, n, ncomp);
}

cudaError_t launch_integrate_team8(const IntegrateArgs& a, const MWParams& p, long long base, int blocks, size_t smem,
                                  cudaStream_t stream) {
  if (smem > 0) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_integrate_mw_team<Dopri8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_integrate_mw_team<Dopri8><<<(unsigned)blocks, 128, smem, stream>>>(a, p, base);
  return cudaGetLastError();
}

cudaError_t launch_integrate_dopri8_exclusive(const IntegrateArgs& a, const MWParams& p, int variant, int block,
                                              int grid, size_t smem, cudaStream_t stream) {
  if (variant != 2 && block > 128) block = 128;  // variants 0 and 1 are built for at most 128 threads
  return mw_launch_exclusive<Dopri8>(variant, (unsigned)grid, block, smem, stream, a, p);
}
}  // namespace gal
