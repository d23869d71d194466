// Batched exact-code matmul on the warp matrix unit: y[t, n] = sum_k x[t, k] * (s q + b)[n, k] for tens to thousands of
// activation rows, dense or grouped by expert, where the weights may not be rounded to f16 first:
//   * router logits (moe_router_logits.wgsl: f32 sums over exact codes feed a softmax and a top-k),
//   * 8-bit projections of 9 to 32 rows, and of any more with f32 results (int8_affine_batched.wgsl),
//   * 3-bit expert matmuls that the streaming kernel leaves (int4_matmul.gen.ts:229-254, :409-448), and 4-bit ones of few pairs per expert over a ragged K.
// Those used to run as slabs of eight rows (or, for experts, one GEMV per pair) on the CUDA cores.
//
// Codes enter the MMA as f16 subnormals masked in place (ztvm_frag.cuh): no dequantisation, exact products, one f32
// accumulator pair per run of 64 codes that is folded with the run's scale and bias by f32 FMAs
//   acc += s * dot + b * sum(x)                                             (int4_matmul.gen.ts:388-408)
// An A fragment costs a handful of ANDs and is used for NBW blocks of eight tokens, so with many tokens the bound is
// the warp-level tensor rate; with few it is the weight stream.
//
// CTA: eight warps as WM x WN x WK; a warp owns 32 weight rows x 8 NBW tokens (n blocks wn, wn + WN, ...: live blocks
// spread evenly when the tile is not full) and every WK-th run. Stages of RUNS runs (weights ROWS x 64 RUNS codes,
// activations TOK x 64 RUNS f16) go through a cp.async ring, swizzled so that fragment loads hit all banks. The sums
// of x that multiply the biases come from the matrix unit as well, one stage ahead of their use.
#include <cstring>

#include "ztvm_frag.cuh"
#include "ztvm_kernels.h"
#include "ztvm_moe_plan.cuh"
#include "ztvm_stream_mma.cuh"

namespace ztvm {

struct BatchParams {
  const uint32_t* W;
  const __half* S;
  const __half* B;
  const __half* X;
  void* Y;
  uint32_t N, M, KP, SPR, out_f32;
  uint32_t x_row_stride, y_row_stride;
  // grouped form
  uint32_t slots, in_slot_stride, out_slot_stride, in_tok_stride, out_tok_stride;
  MoeScratch sc;
};

template <int BITS, int WM, int WN, int WK, int NBW, int RUNS>
struct BatchCfg {
  static_assert(WM * WN * WK == 8, "eight warps");
  static constexpr int kRows = WM * 32, kTok = WN * NBW * 8;
  static constexpr int kRowBytes = RUNS * Frag<BITS>::kRunBytes;
  static constexpr int kWBytes = kRows * kRowBytes, kXBytes = kTok * RUNS * 128;
  // scales and biases of a row in a stage: the aligned 4-byte words around its RUNS values
  static constexpr int kSbSlot = RUNS * 2 + 4, kSbBytes = 2 * kRows * kSbSlot;
  static constexpr int kStageBytes = (kWBytes + kXBytes + kSbBytes + 127) / 128 * 128;
  static constexpr int kStages = 4 * kStageBytes <= 104 * 1024 ? 4 : 3;   // two CTAs per SM
  static constexpr int kOffXs = kStages * kStageBytes;                 // float [2][RUNS][kTok]
  static constexpr int kOffRow = kOffXs + 2 * RUNS * kTok * 4;         // uint64 [2][kTok]: input / output row offsets (grouped form)
  static constexpr int kTotal = kOffRow + 2 * kTok * 8;
  static constexpr int kOutPitch = kRows + 4;
  static_assert(kTok * kOutPitch * 4 <= kOffXs, "the output tile reuses the ring");
};

__device__ __forceinline__ void bm_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f), "f"(0.f), "f"(0.f), "f"(0.f));
}
__device__ __forceinline__ void bm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// W16: weight rows are whole 16-byte pieces (always, but for 3-bit rows of an odd number of runs).
template <int BITS, int WM, int WN, int WK, int NBW, int RUNS, bool MOE, bool W16>
__global__ void __launch_bounds__(256, NBW == 8 ? 1 : 2)
batch_mma_kernel(const BatchParams p) {
  using C = BatchCfg<BITS, WM, WN, WK, NBW, RUNS>;
  using F = Frag<BITS>;
  extern __shared__ __align__(128) uint8_t bm_smem[];
  const uint32_t sm = (uint32_t)__cvta_generic_to_shared(bm_smem);
  float* const xs_sm = reinterpret_cast<float*>(bm_smem + C::kOffXs);
  unsigned long long* const in_off = reinterpret_cast<unsigned long long*>(bm_smem + C::kOffRow);
  unsigned long long* const out_off = in_off + C::kTok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, c = lane & 3;
  const int wm = warp % WM, wn = (warp / WM) % WN, wk = warp / (WM * WN);

  const uint32_t n0 = blockIdx.y * C::kRows;      // token tiles run fastest: they share the row block's weights in L2
  const uint32_t* W = p.W;
  const __half *S = p.S, *B = p.B;
  uint32_t ntok, t0 = blockIdx.x * C::kTok;
  uint32_t sb_odd0 = 0u;             // tables start on 8-byte boundaries; an expert's slice may start on an odd group
  if constexpr (MOE) {
    asm volatile("griddepcontrol.wait;" ::: "memory");     // the plan comes from the kernel before
    if (blockIdx.x >= *p.sc.ntiles) return;
    const uint32_t* tile = p.sc.tiles + (size_t)blockIdx.x * 3;
    const uint32_t expert = tile[0], first = tile[1];
    ntok = tile[2];
    sb_odd0 = expert & p.N & p.SPR & 1u;
    W += (size_t)expert * p.N * p.KP;
    S += (size_t)expert * p.N * p.SPR;
    B += (size_t)expert * p.N * p.SPR;
    for (uint32_t t = tid; t < ntok; t += 256) {
      const uint32_t pair = p.sc.sorted[first + t];
      const uint32_t tok = pair / p.slots, slot = pair - tok * p.slots;
      in_off[t] = (size_t)tok * p.in_tok_stride + (size_t)slot * p.in_slot_stride;
      out_off[t] = (size_t)tok * p.out_tok_stride + (size_t)slot * p.out_slot_stride;
    }
    __syncthreads();
  } else {
    ntok = p.M - t0 < (uint32_t)C::kTok ? p.M - t0 : (uint32_t)C::kTok;
  }
  const uint32_t stages = (p.SPR + RUNS - 1) / RUNS;

  // ---- producer: this thread's pieces of a stage. Where they come from and go to is worked out once; a stage costs an add
  // and a copy per piece (computing rows and pieces afresh took more issue slots than the multiplications). -------------
  constexpr uint32_t WP = W16 ? 16 : 8, CH = C::kRowBytes / WP, NW = (C::kRows * CH + 255) / 256;
  const uint8_t* const w_tile = reinterpret_cast<const uint8_t*>(W + (size_t)n0 * p.KP);
  uint32_t w_off[NW], w_dst[NW], w_on = 0;
#pragma unroll
  for (uint32_t i = 0; i < NW; ++i) {
    const uint32_t idx = tid + 256u * i, row = idx / CH, q = idx - row * CH, run = q * WP / F::kRunBytes;
    const uint32_t sw = BITS == 3 ? 0u : BITS == 8 ? row & 1u : RUNS == 2 ? (row >> 1) & 1u : row & 3u;
    w_off[i] = row * (p.KP * 4u) + q * WP;
    w_dst[i] = row * C::kRowBytes + (BITS == 3 ? q * WP : (run ^ sw) * F::kRunBytes + q * WP % F::kRunBytes);
    if (idx < (uint32_t)C::kRows * CH && n0 + row < p.N) w_on |= 1u << i;
  }
  auto issue_w = [&](uint32_t st) {
    const uint32_t dst0 = sm + (st % C::kStages) * C::kStageBytes;
    const uint8_t* const src0 = w_tile + (size_t)st * C::kRowBytes;
    const uint32_t live = p.SPR - st * RUNS;                       // runs that exist from here on
#pragma unroll
    for (uint32_t i = 0; i < NW; ++i)
      if ((w_on >> i & 1u) && (live >= (uint32_t)RUNS || ((tid + 256u * i) % CH) * WP / F::kRunBytes < live)) {
        if constexpr (W16) cp_async16_s(dst0 + w_dst[i], src0 + w_off[i]);
        else cp_async8_s(dst0 + w_dst[i], src0 + w_off[i]);
      }
  };
  // scales and biases: thread = (table, row)
  constexpr uint32_t NSB = (2 * C::kRows + 255) / 256;
  const uint32_t spr_odd = p.SPR & 1u;
  auto issue_sb = [&](uint32_t st) {
    const uint32_t dst0 = sm + (st % C::kStages) * C::kStageBytes + C::kWBytes + C::kXBytes;
    const uint32_t g0 = st * RUNS, have = p.SPR - g0 < (uint32_t)RUNS ? p.SPR - g0 : (uint32_t)RUNS;
#pragma unroll
    for (uint32_t i = 0; i < NSB; ++i) {
      const uint32_t idx = tid + 256u * i, row = idx % C::kRows;
      if (idx >= 2u * C::kRows || n0 + row >= p.N) continue;
      const __half* src = (idx >= (uint32_t)C::kRows ? B : S) + (size_t)(n0 + row) * p.SPR + g0;
      const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(src) >> 1) & 1u, end = 2u * (odd + have);
#pragma unroll
      for (uint32_t w = 0; w <= (uint32_t)RUNS / 2; ++w)
        if (w * 4u < end)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst0 + idx * C::kSbSlot + w * 4u),
                       "l"(src - odd + 2 * w), "r"(end - w * 4u < 4u ? end - w * 4u : 4u) : "memory");
    }
  };
  // activations: thread = (token mod XT, 16-byte piece)
  constexpr uint32_t XC = RUNS * 8, XT = 256 / XC, NX = C::kTok / XT;
  static_assert(C::kTok % XT == 0 && XT % 8 == 0, "tokens of a thread share their swizzle");
  const uint32_t x_q = tid % XC, x_tok = tid / XC;
  const uint32_t x_dst = C::kWBytes + x_tok * (RUNS * 128) + ((x_q ^ (x_tok & 7u)) << 4);
  const __half* x_src[MOE ? NX : 1];
  uint32_t x_on = 0;
#pragma unroll
  for (uint32_t i = 0; i < NX; ++i) {
    const uint32_t tok = x_tok + XT * i;
    if (tok < ntok) x_on |= 1u << i;
    if constexpr (MOE) x_src[i] = p.X + (tok < ntok ? in_off[tok] : 0ull) + x_q * 8;
  }
  if constexpr (!MOE) x_src[0] = p.X + (size_t)(t0 + x_tok) * p.x_row_stride + x_q * 8;
  const size_t x_step = (size_t)XT * p.x_row_stride;
  auto issue_x = [&](uint32_t st) {
    const uint32_t dst0 = sm + (st % C::kStages) * C::kStageBytes + x_dst;
    if ((x_q >> 3) >= p.SPR - st * RUNS) return;                   // past the last run
#pragma unroll
    for (uint32_t i = 0; i < NX; ++i)
      if (x_on >> i & 1u)
        cp_async16_s(dst0 + i * (XT * RUNS * 128), (MOE ? x_src[MOE ? i : 0] : x_src[0] + i * x_step) + (size_t)st * (RUNS * 64));
  };
  // A landed stage's activations, a warp per (run, eight tokens): their sums per token by the matrix unit (rows of ones), and
  // the pairs of values put into the order of the code pairs, in place, so that the main loop loads B registers as they are.
  auto prepare_x = [&](uint32_t st) {
    uint8_t* const src0 = bm_smem + (st % C::kStages) * C::kStageBytes + C::kWBytes;
    float* const dst = xs_sm + (st & 1u) * (RUNS * C::kTok);
    constexpr uint32_t kOnes = 0x3C003C00u;
#pragma unroll 1
    for (uint32_t i = warp; i < (uint32_t)RUNS * (C::kTok / 8); i += 8) {
      const uint32_t nb = i % (C::kTok / 8), run = i / (C::kTok / 8);
      if (nb * 8 >= ntok) continue;
      uint8_t* const row = src0 + (nb * 8 + (uint32_t)g) * (RUNS * 128);
      uint4* const p0 = reinterpret_cast<uint4*>(row + (((run * 8 + 2 * c) ^ (uint32_t)g) << 4));
      uint4* const p1 = reinterpret_cast<uint4*>(row + (((run * 8 + 2 * c + 1) ^ (uint32_t)g) << 4));
      uint32_t b[8];
      F::b(*p0, *p1, b);
      float d[4];
      bm_mma0(d, kOnes, kOnes, kOnes, kOnes, b[0], b[1]);
      bm_mma(d, kOnes, kOnes, kOnes, kOnes, b[2], b[3]);
      bm_mma(d, kOnes, kOnes, kOnes, kOnes, b[4], b[5]);
      bm_mma(d, kOnes, kOnes, kOnes, kOnes, b[6], b[7]);
      if (g == 0) *reinterpret_cast<float2*>(dst + run * C::kTok + nb * 8 + 2 * c) = make_float2(d[0], d[1]);
      if constexpr (BITS != 8) {
        *p0 = make_uint4(b[0], b[1], b[2], b[3]);
        *p1 = make_uint4(b[4], b[5], b[6], b[7]);
      }
    }
  };

  // 3-bit codes by permuted bytes (codes3_inplace16) or shifted to bit 0 first. Permuted, tiles of 16 pairs take 2 to 5 % less time on 85 of 102 shapes and up to
  // 9 % more on the others, all of 1.3 to 2.5 waves of CTAs (257 experts of 512 x 2048, 4 pairs each, 56.8 us shifted, 55.0; 33 of 1472 x 2816, 10 pairs, 37.1,
  // 40.2); tiles of 64 take 1 % less. With tiles of 32 it gained nothing on average and cost up to 10 % (33 of 1472 x 2816, 14 pairs, 50.1, 55.1).
  constexpr bool kShifted = BITS == 3 && C::kTok == 32;
  constexpr int RPW = RUNS / WK;
  static_assert(RPW >= 1 && RPW * WK == RUNS, "runs per warp");
  float acc[2][NBW][4];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int j = 0; j < NBW; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[t][j][e] = 0.f;

#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s)
    if ((uint32_t)s < stages) { issue_w((uint32_t)s); issue_sb((uint32_t)s); }
  if constexpr (!MOE) asm volatile("griddepcontrol.wait;" ::: "memory");   // weights first, then what a kernel before may have written
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s) {
    if ((uint32_t)s < stages) issue_x((uint32_t)s);
    tc_commit();
  }
  asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 2) : "memory");
  __syncthreads();
  prepare_x(0);

  for (uint32_t st = 0; st < stages; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 3) : "memory");   // stage st + 1 has landed
    __syncthreads();                                                              // stage st - 1 is free, the activations of stage st are prepared
    if (st + C::kStages - 1 < stages) { issue_w(st + C::kStages - 1); issue_sb(st + C::kStages - 1); issue_x(st + C::kStages - 1); }
    tc_commit();
    if (st + 1 < stages) prepare_x(st + 1);

    const uint8_t* const wst = bm_smem + (st % C::kStages) * C::kStageBytes;
    const uint8_t* const xst = wst + C::kWBytes;
    const float* const xs = xs_sm + (st & 1u) * (RUNS * C::kTok);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const uint32_t run = (uint32_t)(r * WK + wk);
      if (st * RUNS + run >= p.SPR) break;
      float sc[4], bi[4];              // of rows g, g + 8, g + 16, g + 24
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t row = (uint32_t)(wm * 32 + g + 8 * h);
        const uint32_t odd = (sb_odd0 + ((n0 + row) & spr_odd)) & 1u;        // a stage starts on an even group
        const uint8_t* const at = xst + C::kXBytes + row * C::kSbSlot + (odd + run) * 2u;
        sc[h] = __half2float(*reinterpret_cast<const __half*>(at)) * F::kUnit;
        bi[h] = __half2float(*reinterpret_cast<const __half*>(at + C::kRows * C::kSbSlot));
      }
      uint32_t a[2][2][8];             // [row tile][row g | g + 8][register]
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t row = (uint32_t)(wm * 32 + t * 16 + h * 8 + g);
          uint32_t pos = run;
          if constexpr (BITS == 4) pos = run ^ (RUNS == 2 ? (row >> 1) & 1u : row & 3u);
          if constexpr (BITS == 8) pos = run ^ (row & 1u);
          const typename F::Raw v = F::load(wst + row * C::kRowBytes + pos * F::kRunBytes + F::lane_byte(c), c);
          if constexpr (kShifted) F::a_shifted(v, a[t][h]);
          else F::a(v, a[t][h]);
        }
#pragma unroll
      for (int j = 0; j < NBW; ++j) {
        const uint32_t nb = (uint32_t)(wn + WN * j);
        if (nb * 8 >= ntok) break;     // warp-uniform: the rest of the tile is empty
        const uint8_t* const xrow = xst + (nb * 8 + (uint32_t)g) * (RUNS * 128);
        const uint4 b0 = *reinterpret_cast<const uint4*>(xrow + (((run * 8 + 2 * c) ^ (uint32_t)g) << 4));
        const uint4 b1 = *reinterpret_cast<const uint4*>(xrow + (((run * 8 + 2 * c + 1) ^ (uint32_t)g) << 4));
        const float2 xsv = *reinterpret_cast<const float2*>(xs + run * C::kTok + nb * 8 + 2 * c);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          float d0[4], d1[4];          // 8-bit codes have one class: a single chain
          bm_mma0(d0, a[t][0][0], a[t][1][0], a[t][0][1], a[t][1][1], b0.x, b0.y);
          bm_mma(d0, a[t][0][2], a[t][1][2], a[t][0][3], a[t][1][3], b0.z, b0.w);
          if constexpr (F::kTwoClasses) bm_mma0(d1, a[t][0][4], a[t][1][4], a[t][0][5], a[t][1][5], b1.x, b1.y);
          else bm_mma(d0, a[t][0][4], a[t][1][4], a[t][0][5], a[t][1][5], b1.x, b1.y);
          bm_mma(F::kTwoClasses ? d1 : d0, a[t][0][6], a[t][1][6], a[t][0][7], a[t][1][7], b1.z, b1.w);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float v = F::kTwoClasses ? fmaf(d0[e], F::kRatio, d1[e]) : d0[e];
            acc[t][j][e] = fmaf(bi[2 * t + (e >> 1)], (e & 1) ? xsv.y : xsv.x, fmaf(sc[2 * t + (e >> 1)], v, acc[t][j][e]));
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- results: turned round in shared memory (a lane holds one row of two tokens, y wants consecutive rows of one token);
  // the K shares of the warps are added in a fixed order ---------------------------------------------------------------
  float* const out = reinterpret_cast<float*>(bm_smem);
#pragma unroll
  for (int k = 0; k < WK; ++k) {
    if (wk == k) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int j = 0; j < NBW; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 v = make_float2(acc[t][j][2 * h], acc[t][j][2 * h + 1]);
            float* d = out + (size_t)((wn + WN * j) * 8 + 2 * c) * C::kOutPitch + wm * 32 + t * 16 + h * 8 + g;
            d[0] = k ? d[0] + v.x : v.x;
            d[C::kOutPitch] = k ? d[C::kOutPitch] + v.y : v.y;
          }
    }
    __syncthreads();
  }
  const uint32_t rows = p.N - n0 < (uint32_t)C::kRows ? p.N - n0 : (uint32_t)C::kRows;
  if (p.out_f32) {
    for (uint32_t i = tid; i < ntok * C::kRows; i += 256) {
      const uint32_t t = i / C::kRows, r = i % C::kRows;
      if (r < rows) reinterpret_cast<float*>(p.Y)[(MOE ? (size_t)out_off[t] : (size_t)(t0 + t) * p.y_row_stride) + n0 + r] = out[t * C::kOutPitch + r];
    }
    return;
  }
  for (uint32_t i = tid; i < ntok * (C::kRows / 8); i += 256) {
    const uint32_t t = i / (C::kRows / 8), r = (i % (C::kRows / 8)) * 8;
    if (r >= rows) continue;
    const float* v = out + t * C::kOutPitch + r;
    __half* y = reinterpret_cast<__half*>(p.Y) + (MOE ? (size_t)out_off[t] : (size_t)(t0 + t) * p.y_row_stride) + n0 + r;
    if (r + 8 <= rows && (reinterpret_cast<uintptr_t>(y) & 15u) == 0) {
      uint4 o;
      o.x = h2_as_u32(__floats2half2_rn(v[0], v[1])); o.y = h2_as_u32(__floats2half2_rn(v[2], v[3]));
      o.z = h2_as_u32(__floats2half2_rn(v[4], v[5])); o.w = h2_as_u32(__floats2half2_rn(v[6], v[7]));
      *reinterpret_cast<uint4*>(y) = o;
    } else {
      for (uint32_t e = 0; e < 8 && r + e < rows; ++e) y[e] = __float2half_rn(v[e]);
    }
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------
template <int BITS, int WM, int WN, int WK, int NBW, int RUNS, bool MOE, bool W16 = true>
static cudaError_t launch_cfg(const BatchParams& p, uint32_t token_tiles, cudaStream_t st) {
  using C = BatchCfg<BITS, WM, WN, WK, NBW, RUNS>;
  auto kern = batch_mma_kernel<BITS, WM, WN, WK, NBW, RUNS, MOE, W16>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 16 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kTotal);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(token_tiles, (p.N + C::kRows - 1) / C::kRows);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = C::kTotal;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

static bool batch_common_ok(const GemvParams& g) {
  if (g.group_shift != 6 || !g.B || g.K % 64u || g.K == 0 || g.N == 0 || g.N > 64u * 65535u) return false;
  const uintptr_t lows = reinterpret_cast<uintptr_t>(g.X) | reinterpret_cast<uintptr_t>(g.W);
  return (lows & 15u) == 0;
}

static BatchParams batch_params(const GemvParams& g) {
  BatchParams p;
  memset(&p, 0, sizeof(p));
  p.W = g.W; p.S = g.S; p.B = g.B; p.X = g.X; p.Y = g.Y;
  p.N = g.N; p.M = g.M; p.KP = g.KP; p.SPR = g.SPR; p.out_f32 = g.out_f32;
  p.x_row_stride = g.x_row_stride; p.y_row_stride = g.y_row_stride;
  return p;
}

bool batch_mma_supported(const GemvParams& g, int bits) {
  return (bits == 8 || bits == 4) && batch_common_ok(g) && g.x_row_stride % 8u == 0 && g.M > 0;
}

template <int BITS>
static cudaError_t launch_dense(const BatchParams& p, int sm_count, cudaStream_t st) {
  // Tile by the work of the busiest SM: tiles dealt to it x their area x what a tile costs per element of its area. Larger
  // tiles unpack a code and load an activation for more products (4096 x 4096 x 1024: 128 x 128 tiles 183 us, 128 x 64
  // 201 us); the smallest, whose warps split K four ways, fill the chip with few rows.
  const uint64_t sm = (uint64_t)sm_count;
  auto cost = [&](uint32_t rows, uint32_t tok, uint32_t weight) {
    const uint64_t tiles = (uint64_t)((p.N + rows - 1) / rows) * ((p.M + tok - 1) / tok);
    return (tiles + sm - 1) / sm * rows * tok * weight;
  };
  const uint64_t big = p.M > 64 ? cost(128, 128, 88) : ~0ull, mid = p.M > 32 ? cost(128, 64, 100) : ~0ull, small = cost(64, 32, 125);
  if (big <= mid && big <= small) return launch_cfg<BITS, 4, 2, 1, 8, 2, false>(p, (p.M + 127) / 128, st);
  if (mid <= small) return launch_cfg<BITS, 4, 2, 1, 4, 2, false>(p, (p.M + 63) / 64, st);
  return launch_cfg<BITS, 2, 1, 4, 4, 4, false>(p, (p.M + 31) / 32, st);
}
cudaError_t launch_batch_mma(const GemvParams& g, int bits, int sm_count, cudaStream_t st) {
  const BatchParams p = batch_params(g);
  return bits == 8 ? launch_dense<8>(p, sm_count, st) : launch_dense<4>(p, sm_count, st);
}

// Grouped by expert. Tile width by the average number of pairs an expert has: a tile's weights are streamed once for
// its whole token tile, its MMAs run over the token blocks that exist. (4-bit codes come here with few pairs only.)
bool batch_moe_supported(const GemvParams& g, int bits) {
  return (bits == 3 || bits == 4) && batch_common_ok(g) && (g.in_slot_stride | g.in_tok_stride) % 8u == 0 && g.experts <= 1024 && !g.dst_index;
}
uint32_t batch_moe_tile_rows(int bits, uint32_t experts, uint64_t pairs) {
  return bits == 4 || pairs <= 10ull * experts ? 16u : pairs <= 24ull * experts ? 32u : 64u;
}
cudaError_t launch_batch_moe(const GemvParams& g, int bits, uint32_t tokens, uint32_t slots, uint32_t* scratch, cudaStream_t st, bool reuse_plan) {
  const uint32_t P = tokens * slots, tok = batch_moe_tile_rows(bits, g.experts, P);
  BatchParams p = batch_params(g);
  p.slots = slots;
  p.in_slot_stride = g.in_slot_stride; p.out_slot_stride = g.out_slot_stride;
  p.in_tok_stride = g.in_tok_stride; p.out_tok_stride = g.out_tok_stride;
  p.sc = moe_scratch_carve(scratch, g.experts, P);
  cudaError_t e = reuse_plan ? cudaSuccess : launch_moe_plan(g, tokens, slots, p.sc, tok, st);
  if (e != cudaSuccess) return e;
  const uint64_t by_rows = (uint64_t)(P + tok - 1) / tok + g.experts;
  const uint32_t max_tiles = (uint32_t)(by_rows < P ? by_rows : P);   // the kernel reads the real count
  if (bits == 4) return launch_cfg<4, 4, 1, 2, 2, 4, true>(p, max_tiles, st);
  if (p.KP % 4u) {
    if (tok == 16) return launch_cfg<3, 4, 1, 2, 2, 4, true, false>(p, max_tiles, st);
    if (tok == 32) return launch_cfg<3, 4, 1, 2, 4, 4, true, false>(p, max_tiles, st);
    return launch_cfg<3, 4, 2, 1, 4, 2, true, false>(p, max_tiles, st);
  }
  if (tok == 16) return launch_cfg<3, 4, 1, 2, 2, 4, true>(p, max_tiles, st);
  if (tok == 32) return launch_cfg<3, 4, 1, 2, 4, 4, true>(p, max_tiles, st);
  return launch_cfg<3, 4, 2, 1, 4, 2, true>(p, max_tiles, st);
}

}  // namespace ztvm
