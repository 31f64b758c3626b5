// Dopri5 instantiation of the orbit-integration kernels, and the four-warp
// team kernels for small batches and for the longest orbits of a two-pass batch
// in the Milky Way model.
#include "integrate_kernels.cuh"
#include "integrate_team.cuh"

namespace gal {
cudaError_t launch_integrate_dopri5(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps,
                                    int ncomp, LaunchShape shape, cudaStream_t stream) {
  return launch_integrate<Dopri5>(a, mw, p, comps, ncomp, shape, stream);
}

cudaError_t launch_integrate_team(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   int blocks, cudaStream_t stream) {
  if (mw) k_integrate_mw_team<Dopri5><<<(unsigned)blocks, 128, 0, stream>>>(a, p);
  else if (a.lin) k_integrate_table_team<Dopri5, true><<<(unsigned)blocks, 128, 0, stream>>>(a, comps, ncomp);
  else k_integrate_table_team<Dopri5, false><<<(unsigned)blocks, 128, 0, stream>>>(a, comps, ncomp);
  return cudaGetLastError();
}

cudaError_t launch_integrate_mixed(const IntegrateArgs& a, const MWParams& p, const unsigned* teams, int blocks,
                                   cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(k_integrate_mw_mixed<Dopri5>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExclusiveSmem);
  if (e != cudaSuccess) return e;
  k_integrate_mw_mixed<Dopri5><<<(unsigned)blocks, 128, kExclusiveSmem, stream>>>(a, p, teams);
  return cudaGetLastError();
}
}  // namespace gal
