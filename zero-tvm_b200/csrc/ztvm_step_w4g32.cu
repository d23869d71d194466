#include "ztvm_step.cuh"

namespace ztvm {
cudaError_t launch_step_w4g32(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st) {
  return launch_step_format<4, true, false>(p, al, smem, grid, together, st);
}
}  // namespace ztvm
