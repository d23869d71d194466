// Grouped MoE expert matmul, streaming form, 4-bit and 3-bit codes: the contract of the ids-indirect GEMV
//   y[token, slot, :] = x[token, slot, :] * W[ids[token, slot]]^T        (int4_matmul.gen.ts:229-254)
// for token counts where an expert sees a handful of pairs (a few hundred tokens over 256 experts). There every active
// expert's weights are read and unpacked for a few products each, so it is built like the persistent decode GEMV
// (ztvm_gemv_tc.cuh) rather than like the tensor-core tiles of ztvm_moe_gemm.cu:
//   * the plan (ztvm_moe_plan.cuh) sorts the pairs by expert and cuts each expert's list into chunks of <= 8 pairs:
//     a chunk is the 8 columns of an mma.sync.m16n8k16;
//   * work unit = (chunk, 16 weight rows). The units, in chunk-major order, are split evenly over one CTA per SM;
//     inside a CTA warp (ks, rg) owns K slice ks (256 codes) and walks units rg, rg + RG, ...;
//   * a warp keeps the chunk's activations as B fragments in registers and reloads them when its unit sequence
//     crosses into the next chunk; weights / scales / biases stream through the per-warp cp.async ring;
//   * codes enter the MMA as f16 subnormals masked in place (exact products, ztvm_frag.cuh), each 64-code group is folded with its
//     scale and bias by f32 FMAs, K-slice partials meet in shared memory in a fixed order: the warps of a row group among
//     themselves (a barrier of their own), every third round;
//   * which expert a chunk belongs to and where its pairs' rows lie is looked up once, at the start: with the chains of loads from the plan at
//     every chunk and every meeting 257 experts of 2048 x 512 took 97.5 us at 8 pairs each, now 66; 512 x 2048 68, now 58.
// What bounds it are issue slots (58 % used, DRAM at 25 to 38 %): about 400 instructions per 4096 3-bit codes, half of them the unpacking.
// An expert with more than 8 pairs is streamed once per chunk (the repeats hit L2): the host side sends launches
// with many pairs per expert to the tensor-core tiles instead.
#include "ztvm_moe_plan.cuh"
#include "ztvm_moe_tile.cuh"

namespace ztvm {

constexpr int kMtRounds = 3;                       // rounds between two meetings of the K-slice partials
constexpr int kMtPitch = 20;                       // floats of a pair's 16 rows in a partial: both sides of a meeting hit all banks
constexpr int kMtUnitFloats = 8 * kMtPitch;
constexpr int kMtChunks = 24;                      // chunks of a CTA whose rows are looked up once, at the start

struct MoeTcParams {
  const uint32_t* W;
  const __half* S;
  const __half* B;
  const __half* X;
  __half* Y;
  uint32_t N, KP, SPR, slots;
  uint32_t ks;                                     // slices of a row
  uint32_t in_slot_stride, out_slot_stride, in_tok_stride, out_tok_stride;
  uint32_t pair_out;                               // rows 2i, 2i + 1 of every output lie in one 4-byte word
  MoeScratch sc;
};

template <int BITS>
struct MtCfg {
  using T = MtTile<BITS>;
  static constexpr int kOffPartial = kTcWarps * kTcDepth * T::kBytes;   // float [2][warps][kMtRounds][8 pairs][kMtPitch]
  static constexpr int kOffRows = kOffPartial + 2 * kTcWarps * kMtRounds * kMtUnitFloats * 4;   // uint64 [chunks][in, out][8 pairs]
  static constexpr int kOffExpert = kOffRows + kMtChunks * 16 * 8;                              // uint32 [chunks][expert, pairs]
  static constexpr int kTotal = kOffExpert + kMtChunks * 8;
};

template <int BITS>
__global__ void __launch_bounds__(kTcWarps * 32, 1)
moe_tc_kernel(const MoeTcParams p) {
  extern __shared__ __align__(128) uint8_t mt_smem[];
  using C = MtCfg<BITS>;
  using T = MtTile<BITS>;
  pdl_launch_dependents();
  pdl_wait();                                            // the plan may come from the kernel before
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, c = lane & 3;

  const uint32_t KS = p.ks, RG = (uint32_t)kTcWarps / KS;
  const uint32_t ks = (uint32_t)warp % KS, rg = (uint32_t)warp / KS;
  const uint32_t TPE = (p.N + 15u) / 16u;                    // units per chunk
  const uint32_t nchunks = *p.sc.ntiles;
  const uint64_t U = (uint64_t)nchunks * TPE;
  const uint32_t u0 = (uint32_t)(U * blockIdx.x / gridDim.x), u1 = (uint32_t)(U * (blockIdx.x + 1) / gridDim.x);
  if (u0 == u1) return;
  const uint32_t ec0 = u0 / TPE, my_chunks = (u1 - 1u) / TPE - ec0 + 1u;

  // Experts and rows of this CTA's chunks, so that nothing below waits for a chain of loads from the plan.
  unsigned long long* const rows_tab = reinterpret_cast<unsigned long long*>(mt_smem + C::kOffRows);
  uint32_t* const expert_tab = reinterpret_cast<uint32_t*>(mt_smem + C::kOffExpert);
  auto row_off = [&](uint32_t first, uint32_t col, bool out) -> unsigned long long {
    const uint32_t pair = p.sc.sorted[first + col], tok = pair / p.slots, slot = pair - tok * p.slots;
    return out ? (size_t)tok * p.out_tok_stride + (size_t)slot * p.out_slot_stride : (size_t)tok * p.in_tok_stride + (size_t)slot * p.in_slot_stride;
  };
  for (uint32_t i = threadIdx.x; i < my_chunks * 16u && i < kMtChunks * 16u; i += blockDim.x) {
    const uint32_t* const t = p.sc.tiles + (size_t)(ec0 + (i >> 4)) * 3;
    if ((i & 7u) < t[2]) rows_tab[i] = row_off(t[1], i & 7u, (i & 8u) != 0u);
    if ((i & 15u) < 2u) expert_tab[(i >> 4) * 2u + (i & 15u)] = (i & 15u) ? t[2] : t[0];
  }
  __syncthreads();
  if (rg >= RG) return;                                      // (no barrier of the whole CTA from here on)
  auto chunk_expert = [&](uint32_t ec) { return ec - ec0 < (uint32_t)kMtChunks ? expert_tab[(ec - ec0) * 2u] : p.sc.tiles[(size_t)ec * 3]; };
  auto chunk_pairs = [&](uint32_t ec) { return ec - ec0 < (uint32_t)kMtChunks ? expert_tab[(ec - ec0) * 2u + 1u] : p.sc.tiles[(size_t)ec * 3 + 2]; };
  auto chunk_row = [&](uint32_t ec, uint32_t col, bool out) {
    return ec - ec0 < (uint32_t)kMtChunks ? rows_tab[(ec - ec0) * 16u + (out ? 8u : 0u) + col] : row_off(p.sc.tiles[(size_t)ec * 3 + 1], col, out);
  };
  const uint32_t rounds = ((u1 - u0 + RG - 1) / RG + kMtRounds - 1) / kMtRounds * kMtRounds;

  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(mt_smem) + (uint32_t)warp * (kTcDepth * T::kBytes);
  float* const partial = reinterpret_cast<float*>(mt_smem + C::kOffPartial);

  // ---- producer side: the lane's pieces of a tile ------------------------------------------------------------------
  constexpr int PPR = T::kRowBytes / 16, NP = 16 * PPR / 32;
  uint32_t pc_src[NP], pc_dst[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const uint32_t q = (uint32_t)lane + 32u * i, row = q / PPR, j = q - row * PPR;
    pc_src[i] = row * p.KP + ks * (T::kRowBytes / 4) + j * 4;
    pc_dst[i] = T::piece(row, j);
  }
  const uint32_t sb_row = (uint32_t)lane >> 1, sb_which = (uint32_t)lane & 1;
  const __half* const sb_tab = sb_which ? p.B : p.S;
  const uint32_t sb_dst = T::kCodes + sb_row * 16 + sb_which * 8;
  // the unit the next issue will fetch, as (chunk, tile inside the chunk), and where its pieces lie; looked up once per chunk
  uint32_t i_u = u0 + rg, i_st = ring, i_ec = i_u / TPE, i_tile = i_u - i_ec * TPE;
  const uint32_t ring_end = ring + kTcDepth * T::kBytes;
  const uint32_t* i_src = nullptr;
  const __half* i_sb = nullptr;
  int i_left = 0;                                            // rows of the expert from the tile's first one on; 0: a new chunk
  const size_t src_step = (size_t)RG * 16u * p.KP, sb_step = (size_t)RG * 16u * p.SPR;
  auto issue = [&]() {
    if (i_u < u1) {
      if (i_left <= 0) {
        while (i_tile >= TPE) { i_tile -= TPE; ++i_ec; }
        const size_t row = (size_t)chunk_expert(i_ec) * p.N + (size_t)i_tile * 16;
        i_src = p.W + row * p.KP;
        i_sb = sb_tab + (row + sb_row) * p.SPR + ks * 4;
        i_left = (int)(p.N - i_tile * 16u);
      }
      if (i_left >= 16) {
#pragma unroll
        for (int i = 0; i < NP; ++i) tc_cp16(i_st + pc_dst[i], i_src + pc_src[i]);
      } else {
#pragma unroll
        for (int i = 0; i < NP; ++i)
          if ((int)(((uint32_t)lane + 32u * i) / PPR) < i_left) tc_cp16(i_st + pc_dst[i], i_src + pc_src[i]);
      }
      if ((int)sb_row < i_left) tc_cp8(i_st + sb_dst, i_sb);
      i_u += RG; i_tile += RG; i_left -= (int)RG * 16;
      i_src += src_step; i_sb += sb_step;
    }
    tc_commit();
    i_st = i_st + T::kBytes == ring_end ? ring : i_st + T::kBytes;
  };
#pragma unroll
  for (int i = 0; i < kTcDepth - 1; ++i) issue();

  // ---- consumer side -----------------------------------------------------------------------------------------------
  uint32_t xf[4][8];              // B fragments of the current chunk: column g = its g-th pair
  float xs[4][2];                 // per run: sums of x for the pairs of columns 2c, 2c + 1
  auto load_chunk = [&](uint32_t ec) {
    const bool on = (uint32_t)g < chunk_pairs(ec);
    mt_fragments<BITS>(p.X + (on ? chunk_row(ec, (uint32_t)g, false) : 0ull) + (size_t)ks * kTcSlice + 16 * c, on, c, xf, xs);
  };

  float acc[kMtRounds][2][2];
#pragma unroll
  for (int q = 0; q < kMtRounds; ++q) acc[q][0][0] = acc[q][0][1] = acc[q][1][0] = acc[q][1][1] = 0.f;
  uint32_t c_u = u0 + rg, c_ec = c_u / TPE, c_tile = c_u - c_ec * TPE, st = ring;
  bool c_new = true;

  for (uint32_t blk = 0; blk < rounds / kMtRounds; ++blk) {
#pragma unroll
    for (int q = 0; q < kMtRounds; ++q) {
      issue();
      const bool live = c_u < u1;
      if (live && c_new) {                                     // warp-uniform
        load_chunk(c_ec);
        c_new = false;
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(kTcDepth - 1) : "memory");
      __syncwarp();
      if (live) mt_multiply<BITS>(st, g, c, xf, xs, acc[q]);
      __syncwarp();
      st = st + T::kBytes == ring_end ? ring : st + T::kBytes;
      c_u += RG; c_tile += RG;
      while (c_tile >= TPE) { c_tile -= TPE; ++c_ec; c_new = true; }
    }
    // ---- meeting of the KS warps that share units, in slice order -----------------------------------------------------
    float* const mine = partial + ((blk & 1u) * kTcWarps + (uint32_t)warp) * (kMtRounds * kMtUnitFloats);
#pragma unroll
    for (int q = 0; q < kMtRounds; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mine[q * kMtUnitFloats + 2 * c * kMtPitch + g + 8 * h] = acc[q][h][0];
        mine[q * kMtUnitFloats + (2 * c + 1) * kMtPitch + g + 8 * h] = acc[q][h][1];
        acc[q][h][0] = acc[q][h][1] = 0.f;
      }
    if (KS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1u + rg), "r"(KS * 32u) : "memory"); else __syncwarp();
    const float* const buf = partial + ((blk & 1u) * kTcWarps + rg * KS) * (kMtRounds * kMtUnitFloats);
    for (uint32_t i = ks * 32u + (uint32_t)lane; i < kMtRounds * 64u; i += KS * 32u) {
      const uint32_t r2 = (i & 7u) * 2u, col = (i >> 3) & 7u, q = i >> 6;
      const uint32_t u = u0 + (blk * kMtRounds + q) * RG + rg;
      if (u >= u1) continue;
      const uint32_t ec = u / TPE, n = (u - ec * TPE) * 16u + r2;
      if (col >= chunk_pairs(ec) || n >= p.N) continue;
      float2 v = make_float2(0.f, 0.f);
      for (uint32_t k2 = 0; k2 < KS; ++k2) {
        const float2 a = *reinterpret_cast<const float2*>(buf + k2 * (kMtRounds * kMtUnitFloats) + q * kMtUnitFloats + col * kMtPitch + r2);
        v.x += a.x; v.y += a.y;
      }
      __half* const y = p.Y + chunk_row(ec, col, true) + n;
      const __half2 o = __floats2half2_rn(v.x, v.y);
      if (p.pair_out && n + 1u < p.N) *reinterpret_cast<__half2*>(y) = o;
      else { y[0] = __low2half(o); if (n + 1u < p.N) y[1] = __high2half(o); }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- host side ---------------------------------------------------------------------------------------------
bool moe_tc_supported(const GemvParams& g, int bits) {
  if ((bits != 4 && bits != 3) || g.group_shift != 6 || !g.B) return false;
  if (g.K == 0 || g.K % kTcSlice || g.K / kTcSlice > (uint32_t)kTcWarps || g.N == 0) return false;
  if ((g.in_slot_stride | g.in_tok_stride) % 8 || (reinterpret_cast<uintptr_t>(g.X) & 15u)) return false;
  if ((reinterpret_cast<uintptr_t>(g.W) & 15u) || ((reinterpret_cast<uintptr_t>(g.S) | reinterpret_cast<uintptr_t>(g.B)) & 7u)) return false;
  return g.experts <= 1024;
}

template <int BITS>
static cudaError_t launch_mt(const MoeTcParams& p, int sm_count, cudaStream_t st) {
  using C = MtCfg<BITS>;
  static_assert(C::kTotal <= 227 * 1024, "shared memory of a CTA");
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(moe_tc_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kTotal);
    if (e != cudaSuccess) return e;
    if (dev < 16) attr_set[dev] = true;
  }
  return launch_chained(moe_tc_kernel<BITS>, dim3(sm_count), dim3(kTcWarps * 32), C::kTotal, st, p);
}

cudaError_t launch_moe_tc(const GemvParams& g, int bits, uint32_t tokens, uint32_t slots, uint32_t* scratch, int sm_count,
                          cudaStream_t st, bool reuse_plan) {
  const uint32_t P = tokens * slots;
  MoeScratch sc = moe_scratch_carve(scratch, g.experts, P);
  cudaError_t e = reuse_plan ? cudaSuccess : launch_moe_plan(g, tokens, slots, sc, kMoeTcTileRows, st);
  if (e != cudaSuccess) return e;
  MoeTcParams p;
  p.W = g.W; p.S = g.S; p.B = g.B; p.X = g.X; p.Y = reinterpret_cast<__half*>(g.Y);
  p.N = g.N; p.KP = g.KP; p.SPR = g.SPR; p.slots = slots; p.ks = g.K / kTcSlice;
  p.in_slot_stride = g.in_slot_stride; p.out_slot_stride = g.out_slot_stride;
  p.in_tok_stride = g.in_tok_stride; p.out_tok_stride = g.out_tok_stride;
  p.pair_out = ((reinterpret_cast<uintptr_t>(g.Y) >> 1) | g.out_slot_stride | g.out_tok_stride) % 2u == 0;
  p.sc = sc;
  return bits == 3 ? launch_mt<3>(p, sm_count, st) : launch_mt<4>(p, sm_count, st);
}

}  // namespace ztvm
