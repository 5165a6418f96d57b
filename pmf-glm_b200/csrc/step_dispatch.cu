// Host-side dispatch over the instantiated tile heights and reconstructions.
#include "dispatch.h"

namespace pmf {
BatchKernel batch_kernel(int ty, int recon, int rsol, bool ct, bool comp) {
#define PMF_CASE(TY, RECON) \
  if (ty == TY && recon == RECON) return batch_kernel_of<TY, RECON>(rsol, ct, comp);
  PMF_FOR_EACH_TILE(PMF_CASE)
#undef PMF_CASE
  return nullptr;
}

StepKernelInfo step_kernel_info(int ty, int recon, int rsol, bool ct, bool comp, int src) {
#define PMF_CASE(TY, RECON) \
  if (ty == TY && recon == RECON) return step_kernel_info_of<TY, RECON>(rsol, ct, comp, src);
  PMF_FOR_EACH_TILE(PMF_CASE)
#undef PMF_CASE
  return StepKernelInfo{nullptr, 0, 0};
}
}  // namespace pmf
