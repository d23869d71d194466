#include "ztvm_step.cuh"

namespace ztvm {
cudaError_t launch_step_w8(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st) {
  return launch_step_format<8, false, true>(p, al, smem, grid, together, st);
}
}  // namespace ztvm
