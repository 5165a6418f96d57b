// Step-kernel instantiations for CTAs of PMF_TY owned rows with reconstruction PMF_RECON. The
// Makefile compiles this file once per pair, so that the pairs build in parallel.
#include "step_pick.cuh"

namespace pmf {
template <> StepKernelInfo step_kernel_info_of<PMF_TY, PMF_RECON>(int rsol, bool ct, bool comp, int src) {
  return StepKernelInfo{detail::pick_rs<PMF_TY, PMF_RECON>(rsol, ct, comp, src), StepSmem<PMF_TY>::BYTES,
                        step_threads<PMF_TY>()};
}
template <> BatchKernel batch_kernel_of<PMF_TY, PMF_RECON>(int rsol, bool ct, bool comp) {
  return detail::pick_batch_rs<PMF_TY, PMF_RECON>(rsol, ct, comp);
}
}  // namespace pmf
