// Batched exact-code matmul on the warp matrix unit: y[t, n] = sum_k x[t, k] * (s q + b)[n, k] for tens to thousands of
// activation rows, dense or grouped by expert, where the weights may not be rounded to f16 first:
//   * router logits (moe_router_logits.wgsl: f32 sums over exact codes feed a softmax and a top-k),
//   * 8-bit projections of more than eight rows (int8_affine_batched.wgsl),
//   * 3-bit expert matmuls (int4_matmul.gen.ts:229-254, :409-448).
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
// of x that multiply the biases are formed once per stage from shared memory, one stage ahead of their use.
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
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = 4 * kStageBytes <= 104 * 1024 ? 4 : 3;   // two CTAs per SM
  static constexpr int kOffXs = kStages * kStageBytes;                 // float [2][RUNS][kTok]
  static constexpr int kOffRow = kOffXs + 2 * RUNS * kTok * 4;         // uint64 [2][kTok]: input / output row offsets (grouped form)
  static constexpr int kTotal = kOffRow + 2 * kTok * 8;
  static constexpr int kOutPitch = kRows + 4;
  static_assert(kTok * kOutPitch * 4 <= kOffXs, "the output tile reuses the ring");
};

template <int BITS, int WM, int WN, int WK, int NBW, int RUNS, bool MOE>
__global__ void __launch_bounds__(256, 2)
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
  if constexpr (MOE) {
    asm volatile("griddepcontrol.wait;" ::: "memory");     // the plan comes from the kernel before
    if (blockIdx.x >= *p.sc.ntiles) return;
    const uint32_t* tile = p.sc.tiles + (size_t)blockIdx.x * 3;
    const uint32_t expert = tile[0], first = tile[1];
    ntok = tile[2];
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

  // ---- producer: this thread's pieces of a stage -----------------------------------------------------------------
  auto issue_w = [&](uint32_t st) {
    const uint32_t dst0 = sm + (st % C::kStages) * C::kStageBytes;
    const uint32_t live = p.SPR - st * RUNS;                       // runs that exist from here on
    if constexpr (BITS == 3) {                                     // 24-byte runs: 8-byte pieces unless rows are 16-aligned
      constexpr uint32_t CH = C::kRowBytes / 8;
      for (uint32_t i = tid; i < (uint32_t)C::kRows * CH; i += 256) {
        const uint32_t row = i / CH, q = i - row * CH;
        if (n0 + row < p.N && q / 3 < live)
          cp_async8_s(dst0 + row * C::kRowBytes + q * 8, reinterpret_cast<const uint8_t*>(W + (size_t)(n0 + row) * p.KP) + (size_t)st * C::kRowBytes + q * 8);
      }
    } else {
      constexpr uint32_t CH = C::kRowBytes / 16, CPR = F::kRunBytes / 16;
#pragma unroll
      for (uint32_t i = tid; i < (uint32_t)C::kRows * CH; i += 256) {
        const uint32_t row = i / CH, q = i % CH, run = q / CPR;
        const uint32_t sw = BITS == 4 ? (RUNS == 2 ? (row >> 1) & 1u : row & 3u) : row & 1u;
        if (n0 + row < p.N && run < live)
          cp_async16_s(dst0 + row * C::kRowBytes + (run ^ sw) * F::kRunBytes + (q % CPR) * 16,
                       reinterpret_cast<const uint8_t*>(W + (size_t)(n0 + row) * p.KP) + (size_t)st * C::kRowBytes + q * 16);
      }
    }
  };
  auto issue_x = [&](uint32_t st) {
    const uint32_t dst0 = sm + (st % C::kStages) * C::kStageBytes + C::kWBytes;
    const uint32_t live = p.SPR - st * RUNS;
#pragma unroll
    for (uint32_t i = tid; i < (uint32_t)C::kTok * RUNS * 8; i += 256) {
      const uint32_t tok = i / (RUNS * 8), q = i % (RUNS * 8);
      if (tok < ntok && (q >> 3) < live) {
        const __half* src = MOE ? p.X + in_off[tok] : p.X + (size_t)(t0 + tok) * p.x_row_stride;
        cp_async16_s(dst0 + tok * (RUNS * 128) + ((q ^ (tok & 7u)) << 4), src + (size_t)st * (RUNS * 64) + q * 8);
      }
    }
  };
  // sums of x per (run, token) of a landed stage
  auto sums = [&](uint32_t st) {
    const uint32_t src0 = sm + (st % C::kStages) * C::kStageBytes + C::kWBytes;
    float* dst = xs_sm + (st & 1u) * (RUNS * C::kTok);
    for (uint32_t i = tid; i < (uint32_t)RUNS * C::kTok; i += 256) {
      const uint32_t tok = i % C::kTok, run = i / C::kTok;
      if (tok >= ntok) continue;
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (uint32_t q = 0; q < 8; ++q) {
        const uint4 v = tc_lds128(src0 + tok * (RUNS * 128) + (((run * 8 + q) ^ (tok & 7u)) << 4));
        const float2 a = __half22float2(u32_as_h2(v.x)), b = __half22float2(u32_as_h2(v.y)),
                     d = __half22float2(u32_as_h2(v.z)), e = __half22float2(u32_as_h2(v.w));
        s0 += (a.x + a.y) + (b.x + b.y);
        s1 += (d.x + d.y) + (e.x + e.y);
      }
      dst[i] = s0 + s1;
    }
  };

  // ---- scales and biases of this warp's rows (g, g + 8, g + 16, g + 24) for its runs of the next stage ------------
  constexpr int RPW = RUNS / WK;
  static_assert(RPW >= 1 && RPW * WK == RUNS, "runs per warp");
  const unsigned short* srow[4];
  size_t brow_delta = reinterpret_cast<const unsigned short*>(B) - reinterpret_cast<const unsigned short*>(S);
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const uint32_t row = min(n0 + (uint32_t)(wm * 32 + g + 8 * h), p.N - 1);
    srow[h] = reinterpret_cast<const unsigned short*>(S) + (size_t)row * p.SPR;
  }
  uint32_t sb_nxt[RPW][4];             // scale in the low half, bias in the high half
  auto load_sb = [&](uint32_t st) {
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const uint32_t grp = st * RUNS + (uint32_t)(r * WK + wk);
      if (grp >= p.SPR) continue;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t s = __ldg(srow[h] + grp), b = __ldg(srow[h] + brow_delta + grp);
        sb_nxt[r][h] = s | (b << 16);
      }
    }
  };

  unsigned long long acc[2][NBW][2];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int j = 0; j < NBW; ++j) acc[t][j][0] = acc[t][j][1] = 0ull;
  const float kZero[4] = {0.f, 0.f, 0.f, 0.f};
  const unsigned long long kR = tc_pk(F::kRatio, F::kRatio);

#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s)
    if ((uint32_t)s < stages) issue_w((uint32_t)s);
  load_sb(0);
  if constexpr (!MOE) asm volatile("griddepcontrol.wait;" ::: "memory");   // weights first, then what a kernel before may have written
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s) {
    if ((uint32_t)s < stages) issue_x((uint32_t)s);
    tc_commit();
  }
  asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 2) : "memory");
  __syncthreads();
  sums(0);

  for (uint32_t st = 0; st < stages; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 3) : "memory");   // stage st + 1 has landed
    __syncthreads();                                                              // stage st - 1 is free, sums(st) are visible
    if (st + C::kStages - 1 < stages) { issue_w(st + C::kStages - 1); issue_x(st + C::kStages - 1); }
    tc_commit();
    float sc[RPW][4], bi[RPW][4];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float2 v = __half22float2(u32_as_h2(sb_nxt[r][h]));
        sc[r][h] = v.x * F::kUnit; bi[r][h] = v.y;
      }
    load_sb(st + 1);
    if (st + 1 < stages) sums(st + 1);

    const uint32_t wbase = sm + (st % C::kStages) * C::kStageBytes, xbase = wbase + C::kWBytes;
    const float* xs = xs_sm + (st & 1u) * (RUNS * C::kTok);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const uint32_t run = (uint32_t)(r * WK + wk);
      if (st * RUNS + run >= p.SPR) break;
      uint32_t a[2][2][8];             // [row tile][row g | g + 8][register]
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t row = (uint32_t)(wm * 32 + t * 16 + h * 8 + g);
          uint32_t pos = run;
          if constexpr (BITS == 4) pos = run ^ (RUNS == 2 ? (row >> 1) & 1u : row & 3u);
          if constexpr (BITS == 8) pos = run ^ (row & 1u);
          F::a(F::load(bm_smem + (wbase - sm) + row * C::kRowBytes + pos * F::kRunBytes + F::lane_byte(c), c), a[t][h]);
        }
#pragma unroll
      for (int j = 0; j < NBW; ++j) {
        const uint32_t nb = (uint32_t)(wn + WN * j);
        if (nb * 8 >= ntok) break;     // warp-uniform: the rest of the tile is empty
        const uint32_t xrow = xbase + (nb * 8 + (uint32_t)g) * (RUNS * 128);
        const uint4 x0 = tc_lds128(xrow + (((run * 8 + 2 * c) ^ (uint32_t)g) << 4));
        const uint4 x1 = tc_lds128(xrow + (((run * 8 + 2 * c + 1) ^ (uint32_t)g) << 4));
        uint32_t b[8];
        F::b(x0, x1, b);
        const float2 xsv = *reinterpret_cast<const float2*>(xs + run * C::kTok + nb * 8 + 2 * c);
        const unsigned long long xs2 = tc_pk(xsv.x, xsv.y);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          float d0[4], d1[4];
          tc_mma(d0, a[t][0][0], a[t][1][0], a[t][0][1], a[t][1][1], b[0], b[1], kZero);
          tc_mma(d1, a[t][0][4], a[t][1][4], a[t][0][5], a[t][1][5], b[4], b[5], kZero);
          tc_mma(d0, a[t][0][2], a[t][1][2], a[t][0][3], a[t][1][3], b[2], b[3], d0);
          tc_mma(d1, a[t][0][6], a[t][1][6], a[t][0][7], a[t][1][7], b[6], b[7], d1);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            unsigned long long v;
            if constexpr (F::kTwoClasses) v = tc_ffma2(tc_pk(d0[2 * h], d0[2 * h + 1]), kR, tc_pk(d1[2 * h], d1[2 * h + 1]));
            else v = tc_pk(d0[2 * h] + d1[2 * h], d0[2 * h + 1] + d1[2 * h + 1]);
            const float s = sc[r][2 * t + h], bb = bi[r][2 * t + h];
            unsigned long long q = acc[t][j][h];
            q = tc_ffma2(tc_pk(s, s), v, q);
            acc[t][j][h] = tc_ffma2(tc_pk(bb, bb), xs2, q);
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
            const float2 v = tc_unpk(acc[t][j][h]);
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
template <int BITS, int WM, int WN, int WK, int NBW, int RUNS, bool MOE>
static cudaError_t launch_cfg(const BatchParams& p, uint32_t token_tiles, cudaStream_t st) {
  using C = BatchCfg<BITS, WM, WN, WK, NBW, RUNS>;
  auto kern = batch_mma_kernel<BITS, WM, WN, WK, NBW, RUNS, MOE>;
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
  // 128 x 64 tiles (a larger tile re-reads weights and activations less often) while they give every SM a CTA; with
  // fewer, the K loop is the time and the tiles whose warps split K four ways have the shortest.
  const uint64_t tiles = (uint64_t)((p.N + 127) / 128) * ((p.M + 63) / 64);
  if (p.M > 32 && tiles >= (uint64_t)sm_count) return launch_cfg<BITS, 4, 2, 1, 4, 2, false>(p, (p.M + 63) / 64, st);
  return launch_cfg<BITS, 2, 1, 4, 4, 4, false>(p, (p.M + 31) / 32, st);
}
cudaError_t launch_batch_mma(const GemvParams& g, int bits, int sm_count, cudaStream_t st) {
  const BatchParams p = batch_params(g);
  return bits == 8 ? launch_dense<8>(p, sm_count, st) : launch_dense<4>(p, sm_count, st);
}

// Grouped by expert. Tile width by the average number of pairs an expert has: a tile's weights are streamed once for
// its whole token tile, its MMAs run over the token blocks that exist.
bool batch_moe_supported(const GemvParams& g, int bits) {
  return bits == 3 && batch_common_ok(g) && (g.in_slot_stride | g.in_tok_stride) % 8u == 0 && g.experts <= 1024 && !g.dst_index;
}
uint32_t batch_moe_tile_rows(uint32_t experts, uint64_t pairs) {
  return pairs <= 10ull * experts ? 16u : pairs <= 24ull * experts ? 32u : 64u;
}
cudaError_t launch_batch_moe(const GemvParams& g, uint32_t tokens, uint32_t slots, uint32_t* scratch, cudaStream_t st, bool reuse_plan) {
  const uint32_t P = tokens * slots, tok = batch_moe_tile_rows(g.experts, P);
  BatchParams p = batch_params(g);
  p.slots = slots;
  p.in_slot_stride = g.in_slot_stride; p.out_slot_stride = g.out_slot_stride;
  p.in_tok_stride = g.in_tok_stride; p.out_tok_stride = g.out_tok_stride;
  p.sc = moe_scratch_carve(scratch, g.experts, P);
  cudaError_t e = reuse_plan ? cudaSuccess : launch_moe_plan(g, tokens, slots, p.sc, tok, st);
  if (e != cudaSuccess) return e;
  const uint64_t by_rows = (uint64_t)(P + tok - 1) / tok + g.experts;
  const uint32_t max_tiles = (uint32_t)(by_rows < P ? by_rows : P);   // the kernel reads the real count
  if (tok == 16) return launch_cfg<3, 4, 1, 2, 2, 4, true>(p, max_tiles, st);
  if (tok == 32) return launch_cfg<3, 4, 1, 2, 4, 4, true>(p, max_tiles, st);
  return launch_cfg<3, 4, 2, 1, 4, 2, true>(p, max_tiles, st);
}

}  // namespace ztvm
