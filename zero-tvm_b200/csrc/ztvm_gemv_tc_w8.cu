#include "ztvm_gemv_tc.cuh"

namespace ztvm {
bool gemv_tc_fits_w8(const GemvParams& p, int sm_count) { return tc_fits<8, false>(p, sm_count); }
cudaError_t launch_gemv_tc_w8(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half) { return launch_tc_format<8, false, true>(p, sm_count, st, half); }
}  // namespace ztvm
