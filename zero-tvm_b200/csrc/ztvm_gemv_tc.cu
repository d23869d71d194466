// Which problems the persistent decode GEMV takes, and its instances per weight format (one file each: they compile in parallel).
#include "ztvm_kernels.h"

namespace ztvm {

bool gemv_tc_fits_w4(const GemvParams& p, int sm_count);
cudaError_t launch_gemv_tc_w4(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half);
bool gemv_tc_fits_w4sym(const GemvParams& p, int sm_count);
cudaError_t launch_gemv_tc_w4sym(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half);
bool gemv_tc_fits_w4g32(const GemvParams& p, int sm_count);
cudaError_t launch_gemv_tc_w4g32(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half);
bool gemv_tc_fits_w8(const GemvParams& p, int sm_count);
cudaError_t launch_gemv_tc_w8(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half);

bool gemv_tc_supported(const GemvParams& p, int bits, int sm_count) {
  if (bits == 3 || p.M < 1 || p.M > 8 || p.K % 64u || p.K == 0 || p.N == 0) return false;
  if (!(p.group_shift == 6 || (p.group_shift == 5 && bits == 4 && !p.B)) || (bits == 8 && !p.B)) return false;
  if (p.pair_rows && (p.N != 2 * p.pair_rows || p.out_f32 || p.n_more)) return false;
  if (p.x_row_stride % 8 || (reinterpret_cast<uintptr_t>(p.X) & 15u)) return false;
  if ((reinterpret_cast<uintptr_t>(p.W) & 15u) || ((reinterpret_cast<uintptr_t>(p.S) | reinterpret_cast<uintptr_t>(p.B)) & 7u)) return false;
  // One row: over a K that ends in part of a slice the last K tile leaves most warps idle, and groups of 32 fold twice as
  // often; the CUDA-core kernel, which deals K in 32-code units, is faster there (9000 x 2112: 5.6 against 7.0 us;
  // 14717 x 5056: 13.9 against 20 us; groups of 32, 3072 x 8192: 8.0 against 8.7 us). From two rows on the matrix unit
  // wins everywhere (14717 x 5056, 4 rows: 20.9 against 42.5 us).
  if (bits == 4 && p.M == 1 && (p.K % 256u || p.group_shift == 5) && !p.pair_rows) return false;
  if (bits == 8) return gemv_tc_fits_w8(p, sm_count);
  return p.group_shift == 5 ? gemv_tc_fits_w4g32(p, sm_count) : p.B ? gemv_tc_fits_w4(p, sm_count) : gemv_tc_fits_w4sym(p, sm_count);
}

cudaError_t launch_gemv_tc(const GemvParams& p, int bits, int sm_count, cudaStream_t st, HalfSm* half) {
  if (bits == 8) return launch_gemv_tc_w8(p, sm_count, st, half);
  return p.group_shift == 5 ? launch_gemv_tc_w4g32(p, sm_count, st, half) : p.B ? launch_gemv_tc_w4(p, sm_count, st, half) : launch_gemv_tc_w4sym(p, sm_count, st, half);
}

}  // namespace ztvm
