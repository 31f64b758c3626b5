// Dopri8 instantiation of the orbit-integration kernels, and the four-warp
// team kernels for small batches and for the longest orbits of a two-pass batch
// in the Milky Way model.
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

bool dopri8_inline_saves(const IntegrateArgs& a, const LaunchShape& shape, int ncomp) {
  return use_fixed(a, shape) || use_warp_per_orbit(shape, a.n, ncomp);
}

cudaError_t launch_integrate_team8(const IntegrateArgs& a, bool mw, const MWParams& p, const DevComp* comps, int ncomp,
                                   int blocks, cudaStream_t stream) {
  if (mw) k_integrate_mw_team<Dopri8><<<(unsigned)blocks, 128, 0, stream>>>(a, p);
  else if (a.lin) k_integrate_table_team<Dopri8, true><<<(unsigned)blocks, 128, 0, stream>>>(a, comps, ncomp);
  else k_integrate_table_team<Dopri8, false><<<(unsigned)blocks, 128, 0, stream>>>(a, comps, ncomp);
  return cudaGetLastError();
}

cudaError_t launch_integrate_mixed8(const IntegrateArgs& a, const MWParams& p, const unsigned* teams, int blocks,
                                   cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(k_integrate_mw_mixed<Dopri8>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExclusiveSmem);
  if (e != cudaSuccess) return e;
  k_integrate_mw_mixed<Dopri8><<<(unsigned)blocks, 128, kExclusiveSmem, stream>>>(a, p, teams);
  return cudaGetLastError();
}
}  // namespace gal
