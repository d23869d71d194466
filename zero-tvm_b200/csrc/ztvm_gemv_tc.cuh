// Persistent decode GEMV, M = 1..8, with the warp-level matrix unit as the multiplier array (int4_matmul.gen.ts:170-571
// for M = 1, :580-695 for the runtime-M matvec; int8_affine_*.wgsl): 4-bit weights in groups of 64 or 32, 8-bit weights
// in groups of 64, any K that is whole runs of 64 codes.
//
// Why this shape. At HBM rate one SM has to consume ~45 4-bit codes per clock. The CUDA-core paths top out near 54
// (M = 1) and pay M times the FMAs for M > 1; mma.sync.m16n8k16 multiplies 16 weight rows x 16 codes x 8 tokens per
// instruction (measured 73 codes/clk/SM with the unpack below), the same for every M <= 8. So the kernel is built
// around keeping the memory pipe full and the per-tile fixed work small:
//   * grid = one CTA per SM; CTA b owns the contiguous rows [b*N/G, (b+1)*N/G): perfectly balanced in bytes.
//   * K is cut in slices of 128 bytes per row (256 4-bit codes, 128 8-bit codes). Warp (ks, rg) owns slice ks of the
//     current K tile (W slices) and walks the CTA's 16-row tiles rg, rg+RG, ...; with fewer slices than warps the spare
//     warps take other row tiles (RG > 1). The activations of a slice live in registers as ready-made B fragments, loaded
//     once per K tile: no shared-memory traffic for x at all. The warps of a CTA together read whole stretches of rows
//     (warps on row tiles of their own, 128 bytes of every row at a time, reached half the HBM rate).
//   * weights, scales and biases of a (tile, slice) travel global -> shared with per-lane cp.async into a ring of
//     kTcDepth stages per warp (147 KB in flight per SM); no block-level barrier is involved in the streaming itself.
//   * codes masked where they sit are f16 subnormals (ztvm_frag.cuh): the A fragments cost a few ANDs, the products are
//     exact, each scale group is summed inside the matrix unit and folded into the f32 accumulators with
//     round-to-nearest FMAs:  acc += s*unit*(ratio*lo + hi) + b*sum(x).
//   * every kTcRounds rounds the K-slice partials of the warps meet in shared memory (double-buffered, one
//     __syncthreads per meeting, fixed summation order: results are deterministic).
#pragma once
#include <cstdlib>

#include "ztvm_frag.cuh"
#include "ztvm_kernels.h"
#include "ztvm_stream_mma.cuh"

namespace ztvm {

// rounds between two meetings: the partial buffers hold 2 x warps x rounds x 16 rows x NT floats
__host__ __device__ constexpr int tc_rounds(int nt) { return nt <= 4 ? 4 : 2; }


template <int BITS, bool G32, bool AL>
struct TcCfg {
  static constexpr int kRpi = BITS == 8 ? 2 : 4;                      // runs of 64 codes per slice
  static constexpr int kGpr = G32 ? 2 : 1;                            // scale groups per run
  static constexpr int kG = kRpi * kGpr;                              // scale groups per slice
  static constexpr int kSlice = kRpi * 64;
  // scales (or biases) of one row of a slice: as they are, or the aligned 4-byte words around them
  static constexpr int kSbSlot = AL ? kG * 2 : (kG * 2 + 4 + 7) / 8 * 8;
  static constexpr int kTileBytes = kTcTileW + 16 * 2 * kSbSlot;
};
// 4-byte copy of which the first `bytes` (0, 2 or 4) exist; the rest arrives as zeros
__device__ __forceinline__ void tc_cp4_zfill(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// NT = tokens padded to a power of two. The eight columns of an MMA are (group, token) pairs: with NT tokens one
// accumulator collects GPA = 8 / NT scale groups side by side (the B fragment of a column is zero in the MMAs of the
// other groups), so the per-group fold after the MMAs is spread over the lanes of a quad instead of being repeated
// by each of them: lane (g, c) owns columns 2c and 2c + 1.
// AL: K is whole slices and the tables allow a slice's scales to be copied in one piece.
// ONCE: a CTA's tiles are one block of rounds, and its sums stay in registers over all of K and meet once, so that the warps need not wait for one
// another at every K tile. us, 8-bit (K tiles of 2048), 2 to 8 rows: 4096 x 12288, 4 rows 17.1 -> 15.7, 2048 x 6144 7.9 -> 7.4, 1024 x 8000 10.4 -> 9.6;
// 4-bit, groups of 64 (of 4096), 5 to 8 rows: 4096 x 12288 12.4 -> 11.8, 1536 x 9024 10.0 -> 9.8, but 4 rows 2048 x 7936 7.1 -> 7.2, 2 rows 2752 x 7040
// 9.6 -> 9.9; groups of 32 lose by it (3072 x 8192 9.1 -> 9.5). An instance of its own: as a choice at run time the longer-lived sums cost every other
// shape 4 %. A K tile's sums are added up before they join the rest: one running sum over all of K had up to 1.2 times the error (8 rows of 8-bit
// 4096 x 12288, against 64 bits: 1.29e-7, so 1.13e-7, and 1.12e-7 where they meet at every K tile).
// W = warps per CTA: 16 (one CTA per SM, the whole shared memory as its ring) for projections that keep an SM busy for
// tens of microseconds; 8 (registers and shared memory halve) for small ones, so that a CTA of the NEXT launch in the stream
// -- already started under programmatic dependent launch -- can sit beside this launch's and stream its first weights while it
// finishes, instead of waiting for the SM to empty. Two CTAs of ONE launch must not: each has a fixed share of the rows.
template <int BITS, bool G32, int NT, bool AFFINE, bool AL, int W, bool ONCE>
__global__ void __launch_bounds__(W * 32, 16 / W)
gemv_tc_kernel(const GemvParams p) {
  extern __shared__ __align__(128) uint8_t tc_smem[];
  using C = TcCfg<BITS, G32, AL>;
  using F = Frag<BITS>;
  constexpr int RPI = C::kRpi, G = C::kG;
  constexpr int GPA = 8 / NT;                               // groups per accumulator
  constexpr int NA = GPA >= G ? 1 : G / GPA;                // accumulators per tile
  constexpr uint32_t kTile = C::kTileBytes;
  constexpr int kTcRounds = tc_rounds(NT);                  // rounds between two meetings of the K-slice partials
  constexpr int kBlkRows = kTcRounds * 16;                  // rows a warp covers between two meetings
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, c = lane & 3;

  const uint32_t runs = p.K >> 6, slices = (runs + RPI - 1) / RPI;
  const uint32_t KS = slices < (uint32_t)W ? slices : (uint32_t)W;
  const uint32_t RG = (uint32_t)W / KS;
  const uint32_t ks = (uint32_t)warp % KS, rg = (uint32_t)warp / KS;
  const bool warp_active = rg < RG;
  const uint32_t num_kt = (slices + KS - 1) / KS;

  // Rows of this CTA. Plain form: the contiguous rows [r0, r0 + nrows). Paired form (gate rows, then up rows, in one
  // weight): the CTA owns output rows [r0, r0 + prows) and walks their gate and up tiles alternately -- tile 2j holds
  // gate rows r0 + 16 j .., tile 2j + 1 the up rows pair_rows further down -- so that both halves of an output meet in
  // the same block of rounds. `nrows` counts tile slots x 16 there.
  const bool paired = p.pair_rows != 0u;
  const uint32_t out_rows = paired ? p.pair_rows : p.N;
  const uint32_t r0 = (uint32_t)((uint64_t)blockIdx.x * out_rows / gridDim.x);
  const uint32_t r1 = (uint32_t)((uint64_t)(blockIdx.x + 1) * out_rows / gridDim.x);
  const uint32_t prows = r1 - r0;
  const uint32_t ntiles = paired ? 2u * ((prows + 15) / 16) : (prows + 15) / 16;
  const uint32_t nrows = paired ? ntiles * 16u : prows;
  // first weight row of the tile that starts at CTA-relative row `trow`, and how many of its 16 rows exist
  auto tile_row = [&](uint32_t trow) -> uint32_t {
    if (!paired) return r0 + trow;
    const uint32_t t = trow >> 4;
    return (t & 1u) * p.pair_rows + r0 + (t >> 1) * 16u;
  };
  auto tile_live = [&](uint32_t trow) -> uint32_t {
    const uint32_t first = paired ? (trow >> 5) * 16u : trow;
    return prows - first < 16u ? prows - first : 16u;
  };
  uint32_t rounds = (ntiles + RG - 1) / RG;
  rounds = (rounds + kTcRounds - 1) / kTcRounds * kTcRounds;
  const uint32_t total = num_kt * rounds;                   // (K tile, round) steps of every warp

  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(tc_smem) + (uint32_t)warp * (kTcDepth * kTile);
  float* partial = reinterpret_cast<float*>(tc_smem + (W * kTcDepth * kTile));            // [2][warps][kBlkRows][NT]
  float* acc_sm = partial + 2 * W * kBlkRows * NT;                       // [nrows][M], only if num_kt > 1 (ONCE: there, and unused)

  // ---- producer side: one (tile, slice) per step, issued kTcDepth - 1 steps ahead ----------------------------
  const uint32_t cp_row = (uint32_t)lane >> 3, cp_chunk = (uint32_t)lane & 7;   // codes: 4 rows x 8 chunks per pass
  const uint32_t sb_row = (uint32_t)lane >> 1, sb_which = (uint32_t)lane & 1;   // scales / biases: 16 rows x 2
  // a row's runs are permuted by the row so that the fragment loads of a quarter (half) warp touch all banks; with groups of
  // 32 a lane takes words c and 4 + c of a run, and the rows 4-7 (12-15) have the halves of their runs swapped as well
  const uint32_t cp_dst = cp_row * 128 + (BITS == 8 ? ((((cp_chunk >> 2) ^ (cp_row & 1)) << 6) + ((cp_chunk & 3) << 4))
                                                    : ((((cp_chunk >> 1) ^ (cp_row & 3)) << 5) + ((cp_chunk & 1) << 4)));
  const uint32_t sb_dst = kTcTileW + (sb_row * 2 + sb_which) * C::kSbSlot;
  const size_t row4 = (size_t)4 * p.KP;
  uint32_t i_step = 0, i_kt = 0, i_rd = 0;                  // the next step to issue, as (K tile, round)
  // Running addresses of this lane's pieces of the next tile (plain form: rows advance by RG tiles per round, slices
  // by KS per K tile), so a step costs a few adds instead of 64-bit multiplies; the paired form computes its rows.
  const uint32_t* const src_base = p.W + (size_t)(r0 + rg * 16 + cp_row) * p.KP + ks * 32 + cp_chunk * 4;
  const __half* const sb_base = (sb_which ? p.B : p.S) + (size_t)(r0 + rg * 16 + sb_row) * p.SPR + ks * G;
  const size_t src_round = (size_t)RG * 16 * p.KP, sb_round = (size_t)RG * 16 * p.SPR;
  const uint32_t* src_run = src_base;
  const __half* sb_run = sb_base;
  uint32_t i_trow = rg * 16, i_slot = 0;
  auto issue = [&]() {
    if (warp_active && i_step < total) {
      const uint32_t sl = i_kt * KS + ks;
      const uint32_t trow = i_trow;                         // first row of the tile, CTA-relative
      if (sl < slices && trow < nrows) {
        const uint32_t st = ring + i_slot * kTile;
        const uint32_t* src = src_run;
        const __half* sbp = sb_run;
        uint32_t live = nrows - trow < 16u ? nrows - trow : 16u;
        if (paired) {
          const uint32_t wrow = tile_row(trow);
          live = tile_live(trow);
          src = p.W + (size_t)(wrow + cp_row) * p.KP + sl * 32 + cp_chunk * 4;
          sbp = (sb_which ? p.B : p.S) + (size_t)(wrow + sb_row) * p.SPR + sl * G;
        }
        // row + 4 i: the bits that swizzle stay, but for the halves of groups of 32 (bit 2 of the row)
        auto dst = [&](int i) { return st + (G32 && (i & 1) ? cp_dst ^ 16u : cp_dst) + i * 512; };
        auto copy_sb = [&]() {
          if (!AFFINE && sb_which != 0) return;
          if constexpr (AL) {
            if constexpr (G == 8) tc_cp16(st + sb_dst, sbp);
            else if constexpr (G == 4) tc_cp8(st + sb_dst, sbp);
            else tc_cp4_zfill(st + sb_dst, sbp, 4u);
          } else {
            // the aligned words around the row's next G values; what lies past the row's end arrives as zeros
            const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(sbp) >> 1) & 1u, have = (runs - sl * RPI) * C::kGpr;
            const uint32_t end = 2u * (odd + (have < (uint32_t)G ? have : (uint32_t)G));
            const uint8_t* q = reinterpret_cast<const uint8_t*>(sbp - odd);
#pragma unroll
            for (uint32_t w = 0; w <= (uint32_t)G / 2; ++w) {
              const uint32_t n = w * 4u >= end ? 0u : end - w * 4u < 4u ? end - w * 4u : 4u;
              tc_cp4_zfill(st + sb_dst + w * 4u, n ? q + w * 4u : q, n);
            }
          }
        };
        const bool there = AL || cp_chunk < (runs - sl * RPI) * (F::kRunBytes / 16);
        // one test for codes and scales: this kernel is bound by issue slots, and a second one cost 2 to 4 % of a large projection
        // (lm_head 151936 x 4096: 71.0 -> 68.9 us, 8-bit 114.7 -> 111.3 us)
        if (live == 16u) {
          if (there) {
#pragma unroll
            for (int i = 0; i < 4; ++i) tc_cp16(dst(i), src + i * row4);
          }
          copy_sb();
        } else {
          if (there) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (cp_row + 4 * i < live) tc_cp16(dst(i), src + i * row4);
          }
          if (sb_row < live) copy_sb();
        }
      }
    }
    tc_commit();
    ++i_step;
    if (++i_slot == (uint32_t)kTcDepth) i_slot = 0;
    src_run += src_round; sb_run += sb_round; i_trow += RG * 16;
    if (++i_rd == rounds) {
      i_rd = 0; ++i_kt;
      i_trow = rg * 16;
      src_run = src_base + (size_t)i_kt * KS * 32;
      sb_run = sb_base + (size_t)i_kt * KS * G;
    }
  };
#pragma unroll
  for (int i = 0; i < kTcDepth - 1; ++i) issue();

  // everything above reads only weights; activations and outputs belong to the stream order
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // B fragments of this warp's slice: column g of the MMA = (group jn within an accumulator, token tn)
  uint32_t xf[RPI][8];           // [run][register of the run's four MMAs]
  unsigned long long xs2[NA];    // sums of x over the groups that columns 2c, 2c + 1 of accumulator a stand for
  const int jn = g / NT, tn = g % NT;
  auto load_x = [&](uint32_t kt) {
    const uint32_t sl = kt * KS + ks;
    const bool tok_ok = warp_active && sl < slices && (uint32_t)tn < p.M;
    const __half* xr = p.X + (size_t)tn * p.x_row_stride + (size_t)sl * C::kSlice;
    float part[G];
#pragma unroll
    for (int r = 0; r < RPI; ++r) {
      uint4 xv[2];
      float sum[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {      // the lane's two pieces of eight: side by side, or (groups of 32) one in each half
        const int q = r * C::kGpr + (G32 ? u : 0);
        const bool on = tok_ok && (AL || sl * RPI + r < runs) && q % GPA == jn;
        xv[u] = make_uint4(0u, 0u, 0u, 0u);
        if (on) xv[u] = *reinterpret_cast<const uint4*>(xr + 64 * r + (G32 ? 32 * u + 8 * c : 16 * c + 8 * u));
        const float2 a = __half22float2(u32_as_h2(xv[u].x)), b = __half22float2(u32_as_h2(xv[u].y)),
                     d = __half22float2(u32_as_h2(xv[u].z)), e = __half22float2(u32_as_h2(xv[u].w));
        sum[u] = ((a.x + a.y) + (b.x + b.y)) + ((d.x + d.y) + (e.x + e.y));
      }
      F::b(xv[0], xv[1], xf[r]);
      if constexpr (!G32) sum[0] += sum[1];
#pragma unroll
      for (int h = 0; h < C::kGpr; ++h) {
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
        sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);          // every lane of quad g: sum over group q of token tn
        part[r * C::kGpr + h] = sum[h];
      }
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      float r2[2];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int col = 2 * c + v, want = a * GPA + col / NT;   // the group this lane folds for that column
        float r = 0.f;
#pragma unroll
        for (int q = 0; q < G; ++q) {
          const float t = __shfl_sync(0xffffffffu, part[q], col * 4);
          if (q == want) r = t;
        }
        r2[v] = r;
      }
      xs2[a] = tc_pk(r2[0], r2[1]);
    }
  };
  load_x(0);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  unsigned long long acc[kTcRounds][2];   // per round and row half: the two columns of this lane, packed
#pragma unroll
  for (int q = 0; q < kTcRounds; ++q) acc[q][0] = acc[q][1] = 0ull;
  unsigned long long tot[ONCE ? kTcRounds : 1][2];   // ONCE: over the K tiles before
  if constexpr (ONCE) {
#pragma unroll
    for (int q = 0; q < kTcRounds; ++q) tot[q][0] = tot[q][1] = 0ull;
  }
  const unsigned long long kR = tc_pk(F::kTwoClasses ? F::kRatio : 1.f, F::kTwoClasses ? F::kRatio : 1.f);
  const float kZero[4] = {0.f, 0.f, 0.f, 0.f};
  const uint32_t swz = BITS == 8 ? (uint32_t)g & 1u : (uint32_t)g & 3u;
  // where this lane finds the scale of the group it folds (columns past the last group fold zeros with any scale)
  const uint32_t sc_off = 2u * (NT == 1 ? (2u * c) % G : (2u * c / NT) % G);

  uint32_t step = 0, meet = 0;   // meet: running count of meetings, its parity picks the partial buffer
  for (uint32_t kt = 0; kt < num_kt; ++kt) {
    if (kt) load_x(kt);
    const bool slice_ok = warp_active && kt * KS + ks < slices;
    for (uint32_t blk = 0; blk < rounds / kTcRounds; ++blk, ++meet) {
#pragma unroll
      for (int q = 0; q < kTcRounds; ++q, ++step) {
        issue();
        asm volatile("cp.async.wait_group %0;" ::"n"(kTcDepth - 1) : "memory");
        __syncwarp();
        const uint32_t trow = ((blk * kTcRounds + q) * RG + rg) * 16;
        if (slice_ok && trow < nrows) {
          const uint32_t st = ring + (step % kTcDepth) * kTile;
          const uint32_t live_runs = AL ? (uint32_t)RPI : runs - (kt * KS + ks) * RPI;
          // rows g and g + 8 have one parity, tiles start on even offsets from the CTA's first row
          const uint32_t sb_odd = AL ? 0u : (((paired ? tile_row(trow) : r0) + (uint32_t)g) & p.SPR & 1u) * 2u;
          float clo[NA][4], chi[NA][4];
          auto fold = [&](int a) {
            // column 2c + v of accumulator a is one (group, token)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t rowp = st + kTcTileW + (uint32_t)(g + 8 * h) * 2u * C::kSbSlot + sc_off + (uint32_t)(a * GPA) * 2u + sb_odd;
              float s[2], b[2];
              if constexpr (NT == 1) {      // columns 2c, 2c + 1 are two groups
                auto two = [&](uint32_t q, float (&o)[2]) {
                  if constexpr (AL) {
                    const float2 v = __half22float2(u32_as_h2(tc_lds32(q)));
                    o[0] = v.x; o[1] = v.y;
                  } else {
                    o[0] = __half2float(__ushort_as_half((unsigned short)tc_lds16(q)));
                    o[1] = __half2float(__ushort_as_half((unsigned short)tc_lds16(q + 2u)));
                  }
                };
                two(rowp, s);
                if (AFFINE) two(rowp + C::kSbSlot, b);
              } else {                      // both columns belong to one group
                s[0] = s[1] = __half2float(__ushort_as_half((unsigned short)tc_lds16(rowp)));
                if (AFFINE) b[0] = b[1] = __half2float(__ushort_as_half((unsigned short)tc_lds16(rowp + C::kSbSlot)));
              }
              if (!AFFINE) { b[0] = -7.f * s[0]; b[1] = -7.f * s[1]; }
              // unit * (ratio * lo + hi), then the scale and the bias term, two columns per instruction
              const unsigned long long t2 = tc_ffma2(tc_pk(clo[a][2 * h], clo[a][2 * h + 1]), kR, tc_pk(chi[a][2 * h], chi[a][2 * h + 1]));
              unsigned long long r = acc[q][h];
              r = tc_ffma2(tc_pk(s[0] * F::kUnit, s[1] * F::kUnit), t2, r);
              r = tc_ffma2(tc_pk(b[0], b[1]), xs2[a], r);
              acc[q][h] = r;
            }
          };
#pragma unroll
          for (int r = 0; r < RPI; ++r) {
            uint32_t ag[8], ah[8];          // rows g and g + 8
            if (!AL && (uint32_t)r >= live_runs) {
#pragma unroll
              for (int k = 0; k < 8; ++k) ag[k] = ah[k] = 0u;
            } else {
              typename F::Raw vg, vh;
              if constexpr (BITS == 8) {
                const uint32_t q8 = st + (uint32_t)g * 128 + (((uint32_t)r ^ swz) << 6) + ((uint32_t)c << 4);
                vg.w = tc_lds128(q8); vh.w = tc_lds128(q8 + 1024u);
              } else if constexpr (G32) {
                const uint32_t q4 = st + (uint32_t)g * 128 + (((uint32_t)r ^ swz) << 5) + ((uint32_t)c << 2) + (((uint32_t)g & 4u) << 2);
                vg.w = make_uint2(tc_lds32(q4), tc_lds32(q4 ^ 16u));
                vh.w = make_uint2(tc_lds32(q4 + 1024u), tc_lds32((q4 ^ 16u) + 1024u));
              } else {
                const uint32_t q4 = st + (uint32_t)g * 128 + (((uint32_t)r ^ swz) << 5) + ((uint32_t)c << 3);
                vg.w = tc_lds64(q4); vh.w = tc_lds64(q4 + 1024u);
              }
              F::a(vg, ag); F::a(vh, ah);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int gq = r * C::kGpr + (G32 ? h : 0), a = NA == 1 ? 0 : gq / GPA;
              const bool first = gq % GPA == 0 && (G32 || h == 0) && (NA > 1 || gq == 0);
              if (first) {
                tc_mma(clo[a], ag[2 * h], ah[2 * h], ag[2 * h + 1], ah[2 * h + 1], xf[r][2 * h], xf[r][2 * h + 1], kZero);
                tc_mma(chi[a], ag[4 + 2 * h], ah[4 + 2 * h], ag[5 + 2 * h], ah[5 + 2 * h], xf[r][4 + 2 * h], xf[r][5 + 2 * h], kZero);
              } else {
                tc_mma(clo[a], ag[2 * h], ah[2 * h], ag[2 * h + 1], ah[2 * h + 1], xf[r][2 * h], xf[r][2 * h + 1], clo[a]);
                tc_mma(chi[a], ag[4 + 2 * h], ah[4 + 2 * h], ag[5 + 2 * h], ah[5 + 2 * h], xf[r][4 + 2 * h], xf[r][5 + 2 * h], chi[a]);
              }
              if ((G32 || h == 1) && ((NA > 1 && (gq + 1) % GPA == 0) || (NA == 1 && gq == G - 1))) fold(a);
            }
          }
        }
        __syncwarp();   // every lane is done with the stage before the next issue refills it
      }
      if constexpr (ONCE) {
#pragma unroll
        for (int q = 0; q < kTcRounds; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(tot[q][h]) : "l"(acc[q][h]));
            acc[q][h] = 0ull;
          }
        if (kt + 1 < num_kt) continue;
      }
      // ---- meeting: K-slice partials of the block's rows -> shared, then one fixed-order sum per output --------
      float* mine = partial + ((size_t)((meet & 1u) * W + (uint32_t)warp) * kBlkRows) * NT;
#pragma unroll
      for (int q = 0; q < kTcRounds; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 av = tc_unpk(ONCE ? tot[ONCE ? q : 0][h] : acc[q][h]);
          float v0 = slice_ok || ONCE ? av.x : 0.f, v1 = slice_ok || ONCE ? av.y : 0.f;
          acc[q][h] = 0ull;
          float* dst = mine + (q * 16 + g + 8 * h) * NT;
          if constexpr (NT == 1) {          // the quad's columns are groups of token 0
            v0 += v1;
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
            if constexpr (G > 4) v0 += __shfl_xor_sync(0xffffffffu, v0, 2);   // (columns 4..7 are empty with fewer groups)
            if (c == 0) dst[0] = v0;
          } else if constexpr (NT == 2) {   // lane c holds group c of tokens 0, 1
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1); v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
            v0 += __shfl_xor_sync(0xffffffffu, v0, 2); v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
            if (c == 0) *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
          } else if constexpr (NT == 4) {   // lanes c and c ^ 2 hold the two groups of tokens 2(c & 1) + v
            v0 += __shfl_xor_sync(0xffffffffu, v0, 2); v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
            if (c < 2) *reinterpret_cast<float2*>(dst + 2 * c) = make_float2(v0, v1);
          } else {
            *reinterpret_cast<float2*>(dst + 2 * c) = make_float2(v0, v1);
          }
        }
      __syncthreads();
      const float* buf = partial + (size_t)(meet & 1u) * W * kBlkRows * NT;
      const uint32_t outs = (uint32_t)kTcRounds * RG * 16u * p.M;
      // the meeting's sums are taken by a different warp each time, so no warp falls behind the others for good
      for (uint32_t i = (threadIdx.x + (uint32_t)(W * 32) - 32u * (meet & (uint32_t)(W - 1))) & (uint32_t)(W * 32 - 1); i < outs; i += blockDim.x) {
        const uint32_t tok = i % p.M, br = i / p.M;           // br: row inside the block's R*RG tiles
        const uint32_t r16 = br & 15u, tb = br >> 4;
        const uint32_t q = tb / RG, rgi = tb - q * RG;
        const uint32_t row = ((blk * kTcRounds + q) * RG + rgi) * 16 + r16;
        if (row >= nrows || r16 >= tile_live(row & ~15u)) continue;
        float v = 0.f;
        for (uint32_t k2 = 0; k2 < KS; ++k2) v += buf[((size_t)(rgi * KS + k2) * kBlkRows + q * 16 + r16) * NT + tok];
        if (num_kt > 1 && !ONCE) {
          float* a = acc_sm + (size_t)row * p.M + tok;
          if (kt) v += *a;
          if (kt + 1 < num_kt) { *a = v; continue; }
        }
        if (paired) {
          // The thread that holds an up row (odd tile) finishes the output: the gate row's sum is one tile back, in the
          // same block (tiles per block are even and blocks start on even tiles). Its own thread wrote nothing.
          const uint32_t tile = row >> 4;
          if ((tile & 1u) == 0u) continue;
          const uint32_t tg = tb - 1u, qg = tg / RG, rgg = tg - qg * RG;
          float gsum = 0.f;
          for (uint32_t k2 = 0; k2 < KS; ++k2) gsum += buf[((size_t)(rgg * KS + k2) * kBlkRows + qg * 16 + r16) * NT + tok];
          if (num_kt > 1 && !ONCE && kt) gsum += acc_sm[(size_t)(row - 16u) * p.M + tok];
          const float silu = gsum * (1.0f / (1.0f + expf(-gsum)));
          reinterpret_cast<__half*>(p.Y)[(size_t)tok * p.y_row_stride + r0 + (tile >> 1) * 16u + r16] = __float2half_rn(v * silu);
          continue;
        }
        const size_t o = (size_t)tok * p.y_row_stride + r0 + row;
        if (p.out_f32) {
          reinterpret_cast<float*>(p.Y)[o] = v;
          for (uint32_t k2 = 0; k2 < p.n_more; ++k2) reinterpret_cast<float*>(p.y_more[k2])[o] = v;   // peers (NVLink stores)
        } else {
          const __half hv = __float2half_rn(v);
          reinterpret_cast<__half*>(p.Y)[o] = hv;
          for (uint32_t k2 = 0; k2 < p.n_more; ++k2) reinterpret_cast<__half*>(p.y_more[k2])[o] = hv;
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- host side --------------------------------------------------------------------------------------------
// Shared-memory accumulators (only when K spans several K tiles of W slices) must fit beside the ring.
template <int BITS>
inline uint32_t tc_slices(const GemvParams& p) { return ((p.K >> 6) + (BITS == 8 ? 2 : 4) - 1) / (BITS == 8 ? 2 : 4); }
inline unsigned tc_grid_for(const GemvParams& p, int sm_count) {
  const uint32_t out_rows = p.pair_rows ? p.pair_rows : p.N;
  return out_rows < (uint32_t)sm_count ? out_rows : (unsigned)sm_count;
}
// rows of the cross-K-tile accumulators of one CTA (paired form: gate and up tile slots, 16 rows each)
inline uint64_t tc_acc_rows(const GemvParams& p, unsigned grid) {
  const uint32_t out_rows = p.pair_rows ? p.pair_rows : p.N;
  const uint64_t rows = ((uint64_t)out_rows + grid - 1) / grid + 1;
  return p.pair_rows ? 2 * ((rows + 15) / 16) * 16 : rows;
}
template <int BITS, bool G32>
inline bool tc_aligned(const GemvParams& p) {
  using C = TcCfg<BITS, G32, true>;
  const uintptr_t tables = reinterpret_cast<uintptr_t>(p.S) | reinterpret_cast<uintptr_t>(p.B);
  return p.K % C::kSlice == 0 && (tables & (C::kG * 2u - 1u)) == 0;
}
inline int tc_tokens(const GemvParams& p) { return p.M == 1 ? 1 : p.M == 2 ? 2 : p.M <= 4 ? 4 : 8; }
template <int BITS, bool G32>
inline size_t tc_smem(const GemvParams& p, int sm_count, int warps) {
  const int nt = tc_tokens(p);
  size_t n = (size_t)warps * kTcDepth * (tc_aligned<BITS, G32>(p) ? TcCfg<BITS, G32, true>::kTileBytes : TcCfg<BITS, G32, false>::kTileBytes);
  n += (size_t)2 * warps * tc_rounds(nt) * 16 * nt * 4;
  if (tc_slices<BITS>(p) > (uint32_t)warps) n += tc_acc_rows(p, tc_grid_for(p, sm_count)) * p.M * 4;
  return n;
}
constexpr size_t tc_smem_limit(int warps) { return warps == 8 ? 112 * 1024 : 227 * 1024; }
// warps per CTA for a problem: 8 while an SM's share of the weights is small, else 16
template <int BITS, bool G32>
inline int tc_warps_for(const GemvParams& p, int sm_count) {
  const bool small = tc_slices<BITS>(p) <= 8u && (uint64_t)p.N * p.KP * 4 / (uint64_t)sm_count <= 384u * 1024u;   // one K tile only
  return small && tc_smem<BITS, G32>(p, sm_count, 8) <= tc_smem_limit(8) ? 8 : 16;
}
template <int BITS, bool G32>
inline bool tc_fits(const GemvParams& p, int sm_count) {
  const int w = tc_warps_for<BITS, G32>(p, sm_count);
  return tc_smem<BITS, G32>(p, sm_count, w) <= tc_smem_limit(w);
}

template <int BITS, bool G32, int NT, bool AFFINE, bool AL, int W, bool ONCE = false>
cudaError_t launch_tc_one(const GemvParams& p, unsigned grid, size_t smem, int sm_count, cudaStream_t st, HalfSm* half) {
  auto kern = gemv_tc_kernel<BITS, G32, NT, AFFINE, AL, W, ONCE>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 16 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(W == 8 ? kOnePerSmSmem : tc_smem_limit(W)));
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(W * 32);
  static_assert(tc_smem_limit(8) <= kOnePerSmSmem, "the padding holds what eight warps use");
  // Shares of a few rows, a router's, may as well sit side by side (94 rows in a recorded MoE token: 35.8 us a step kept apart,
  // 35.3 us)
  const uint32_t out_rows = p.pair_rows ? p.pair_rows : p.N;
  const bool behind = half_sm_behind(*half, p), apart = W == 8 && !behind && out_rows > 4u * grid;
  half->now = W == 8 && grid == (unsigned)sm_count && (behind || apart) ? half_sm_bytes(p) : 0;
  cfg.dynamicSmemBytes = apart ? kOnePerSmSmem : smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int BITS, bool G32, bool AFFINE, bool AL, int W>
cudaError_t launch_tc_w(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half) {
  const unsigned grid = tc_grid_for(p, sm_count);
  const size_t smem = tc_smem<BITS, G32>(p, sm_count, W);
  if constexpr (W == 16 && !G32) {
    const uint64_t rows = ((uint64_t)(p.pair_rows ? p.pair_rows : p.N) + grid - 1) / grid, tiles = p.pair_rows ? 2 * ((rows + 15) / 16) : (rows + 15) / 16;
    if (tc_slices<BITS>(p) > (uint32_t)W && tiles <= (uint64_t)tc_rounds(tc_tokens(p))) {
      switch (tc_tokens(p)) {
        case 1: break;
        case 2: if constexpr (BITS == 8) return launch_tc_one<BITS, G32, 2, AFFINE, AL, W, true>(p, grid, smem, sm_count, st, half); break;
        case 4: if constexpr (BITS == 8) return launch_tc_one<BITS, G32, 4, AFFINE, AL, W, true>(p, grid, smem, sm_count, st, half); break;
        default: return launch_tc_one<BITS, G32, 8, AFFINE, AL, W, true>(p, grid, smem, sm_count, st, half);
      }
    }
  }
  switch (tc_tokens(p)) {
    case 1: return launch_tc_one<BITS, G32, 1, AFFINE, AL, W>(p, grid, smem, sm_count, st, half);
    case 2: return launch_tc_one<BITS, G32, 2, AFFINE, AL, W>(p, grid, smem, sm_count, st, half);
    case 4: return launch_tc_one<BITS, G32, 4, AFFINE, AL, W>(p, grid, smem, sm_count, st, half);
    default: return launch_tc_one<BITS, G32, 8, AFFINE, AL, W>(p, grid, smem, sm_count, st, half);
  }
}
template <int BITS, bool G32, bool AFFINE>
cudaError_t launch_tc_format(const GemvParams& p, int sm_count, cudaStream_t st, HalfSm* half) {
  const bool al = tc_aligned<BITS, G32>(p);
  if (tc_warps_for<BITS, G32>(p, sm_count) == 8)
    return al ? launch_tc_w<BITS, G32, AFFINE, true, 8>(p, sm_count, st, half) : launch_tc_w<BITS, G32, AFFINE, false, 8>(p, sm_count, st, half);
  return al ? launch_tc_w<BITS, G32, AFFINE, true, 16>(p, sm_count, st, half) : launch_tc_w<BITS, G32, AFFINE, false, 16>(p, sm_count, st, half);
}

}  // namespace ztvm
