// One step of the kernel that streams expert weights (ztvm_moe_tc.cu): a tile of 16 weight rows x 256 codes
// times up to eight activation rows, one per column of mma.sync.m16n8k16. Codes enter as f16 subnormals masked where they sit
// (ztvm_frag.cuh), a run of 64 is folded with its scale and bias by f32 FMAs.
#pragma once
#include "ztvm_frag.cuh"
#include "ztvm_stream_mma.cuh"

namespace ztvm {

// The codes of the sixteen rows, then per row its four scales and its four biases.
template <int BITS>
struct MtTile {
  static constexpr int kRowBytes = 32 * BITS;                       // 256 codes
  static constexpr int kCodes = 16 * kRowBytes, kBytes = kCodes + 16 * 16;
  // Place of 16-byte piece j of row `row`. 4-bit: a row's runs are permuted by the row so that fragment loads touch all banks.
  __device__ __forceinline__ static uint32_t piece(uint32_t row, uint32_t j) {
    return row * kRowBytes + (BITS == 4 ? (((j >> 1) ^ (row & 3u)) << 5) + ((j & 1u) << 4) : j * 16u);
  }
};

// B fragments of a slice of four runs: lane (g, c) has row g's 16 activations of each run from xr on (`on`: there is a row g). xs: sums
// per run of the rows of columns 2c, 2c + 1.
template <int BITS>
__device__ __forceinline__ void mt_fragments(const __half* xr, bool on, int c, uint32_t (&xf)[4][8], float (&xs)[4][2]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
    if (on) {
      const uint4* const q = reinterpret_cast<const uint4*>(xr + 64 * r);
      x0 = q[0];
      x1 = q[1];
    }
    Frag<BITS>::b(x0, x1, xf[r]);
    float sum = 0.f;
    const uint32_t xw[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 a = __half22float2(u32_as_h2(xw[i])), b = __half22float2(u32_as_h2(xw[i + 1]));
      sum += (a.x + a.y) + (b.x + b.y);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    xs[r][0] = __shfl_sync(0xffffffffu, sum, (2 * c) * 4);
    xs[r][1] = __shfl_sync(0xffffffffu, sum, (2 * c + 1) * 4);
  }
}

// acc[h][v] += rows g + 8 h of the tile at `st` times the activations of column 2c + v.
template <int BITS>
__device__ __forceinline__ void mt_multiply(uint32_t st, int g, int c, const uint32_t (&xf)[4][8], const float (&xs)[4][2], float (&acc)[2][2]) {
  using T = MtTile<BITS>;
  using F = Frag<BITS>;
  const float kZero[4] = {0.f, 0.f, 0.f, 0.f};
  const uint32_t sb_at = st + T::kCodes + (uint32_t)g * 16u;
  const uint4 sg = tc_lds128(sb_at), sh = tc_lds128(sb_at + 128u);   // rows g, g + 8: four scales, four biases
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    uint32_t ag[8], ah[8];                 // rows g and g + 8
    if constexpr (BITS == 4) {
      const uint32_t at = st + (uint32_t)g * 128u + (((uint32_t)r ^ ((uint32_t)g & 3u)) << 5) + ((uint32_t)c << 3);
      F::a(typename F::Raw{tc_lds64(at)}, ag);
      F::a(typename F::Raw{tc_lds64(at + 1024u)}, ah);
    } else {
      const uint32_t at = st + (uint32_t)g * T::kRowBytes + (uint32_t)r * F::kRunBytes + F::lane_byte(c), at8 = at + 8u * T::kRowBytes;
      F::a(typename F::Raw{tc_lds32(at), tc_lds32(at + 4u), (c & 1) != 0}, ag);
      F::a(typename F::Raw{tc_lds32(at8), tc_lds32(at8 + 4u), (c & 1) != 0}, ah);
    }
    float d0[4], d1[4];
    tc_mma(d0, ag[0], ah[0], ag[1], ah[1], xf[r][0], xf[r][1], kZero);
    tc_mma(d1, ag[4], ah[4], ag[5], ah[5], xf[r][4], xf[r][5], kZero);
    tc_mma(d0, ag[2], ah[2], ag[3], ah[3], xf[r][2], xf[r][3], d0);
    tc_mma(d1, ag[6], ah[6], ag[7], ah[7], xf[r][6], xf[r][7], d1);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 w = h ? sh : sg;
      const float2 s2 = __half22float2(u32_as_h2(r & 2 ? w.y : w.x)), b2 = __half22float2(u32_as_h2(r & 2 ? w.w : w.z));
      const float s = (r & 1 ? s2.y : s2.x) * F::kUnit, b = r & 1 ? b2.y : b2.x;
      // (two-wide FMAs would want the scale and the bias twice each, side by side: more moves than they save)
#pragma unroll
      for (int v = 0; v < 2; ++v)
        acc[h][v] = fmaf(b, xs[r][v], fmaf(s, fmaf(d0[2 * h + v], F::kRatio, d1[2 * h + v]), acc[h][v]));
    }
  }
}

}  // namespace ztvm
