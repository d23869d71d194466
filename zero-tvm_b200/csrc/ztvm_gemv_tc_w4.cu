#include "ztvm_gemv_tc.cuh"

namespace ztvm {
bool gemv_tc_fits_w4(const GemvParams& p, int sm_count) { return tc_fits<4, false>(p, sm_count); }
cudaError_t launch_gemv_tc_w4(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half) { return launch_tc_format<4, false, true>(p, sm_count, st, half); }
}  // namespace ztvm
