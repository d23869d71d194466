// A run of one-row matmuls of a decode step in ONE persistent launch (the command-buffer builder of
// src/zero-tvm/engine-core.ts:2194-2202; bodies int4_matmul.gen.ts:170-571 at M = 1, int8_affine_matvec.wgsl).
//
// Why one launch. A decode projection moves 9 to 57 MB, 1.4 to 9 us of HBM time, and as a launch of its own it paid some 4 us
// on top: the CTA of the next launch finds no room until this one's is gone, starts its loads from nothing, and waits for the
// whole grid before it reads its activations (4096 x 4096: 5.4 us; with the loads taken out 3.8 us, with the multiplications
// taken out 3.3 us). Here a warp's loads run on from the last tiles of one matmul into the first of the next -- weights depend on
// nothing -- and a CTA waits for the others only where a matmul reads or overwrites what an earlier one of the run wrote.
//
//   * grid = one CTA per SM (a cooperative launch where any wait is needed: all CTAs are on the chip together). CTA b owns a
//     contiguous share of the rows of every matmul.
//   * a warp's stage is 16 rows x 128 bytes of codes (96 bytes of 3-bit ones) and their scales, fetched by its own lanes
//     (cp.async) into a ring of its own. On 24576 x 4096 in a launch of its own (14.3 us; the kernel for one projection, ztvm_gemv_tc.cuh, 13.7,
//     but its launches do not join): a TMA box per stage 19.8, warps that only fetch for the others 16.0, codes
//     straight from global memory to registers 16.4, e4m3 codes and activations (mma.sync on them is conversions and f16 MMAs here) 18.3.
//   * K is cut into slices of a stage's width. KS of the 16 warps stand side by side along K, RG = 16 / KS groups of them take
//     different row tiles (see step_split).
//   * activations lie in shared memory with the sums of their scale groups; a warp turns its slice into MMA B fragments once per
//     K tile.
//   * codes masked where they sit are f16 subnormals (codes4_inplace, codes3_inplace, codes8_pair01): exact products (3-bit codes put powers
//     of two on their activations, which in one part rounds those below 2^-9, by 2^-20 at most; kTwo's lose nothing); every scale
//     group is summed inside the matrix unit and folded into f32 accumulators, acc += s*(ratio*lo + hi) + b*sum(x). With one
//     token the MMA's columns are the scale groups of the slice: a lane's codes belong to one group, and its activations stand in that
//     group's column.
//   * the unit truncates its sums. Rows that f32 FMAs would otherwise serve (step_two_parts) multiply activations in two parts, in
//     two columns, whose sums are exact.
//   * the K slices of a block of rows meet in shared memory in a fixed order: results are deterministic, and the same whether a
//     matmul runs alone or among others, with or without its activation.
//
// The wait for other CTAs is bounded (about a second); one that runs out raises the status word, and the kernel goes on to its
// end with the data it has, so that all CTAs leave and the counters are handed back clean.
#pragma once
#include "ztvm_frag.cuh"
#include "ztvm_step.h"
#include "ztvm_stream_mma.cuh"
#include "ztvm_tc.cuh"

namespace ztvm {

template <int BITS, bool G32, bool AFFINE, bool AL>
struct StepFmt {
  static constexpr int kRuns = BITS == 8 ? 2 : 4;                   // runs of 64 codes per slice
  static constexpr int kG = kRuns * (G32 ? 2 : 1);                  // scale groups per slice
  static constexpr int kSlice = kRuns * 64;
  static constexpr int kRowBytes = BITS == 3 ? 96 : 128;
  static constexpr int kCodes = 16 * kRowBytes;
  // scales (or biases) of one row of a slice: as they are, or (AL false) the aligned 4-byte words around them
  static constexpr int kSbSlot = AL ? kG * 2 : (kG * 2 + 4 + 7) / 8 * 8;
  static constexpr int kSbRow = (AFFINE ? 2 : 1) * kSbSlot;
  static constexpr int kStage = kCodes + 16 * kSbRow;
  static constexpr int kB = BITS == 3 ? 2 * kCodes3Views : BITS == 8 ? 16 : 32;   // registers of B fragments
  static constexpr bool kTwo = step_two_parts(BITS, G32, AL);
  static constexpr int kSets = kTwo && G32 ? 2 : 1;                 // accumulator sets: two parts of four groups fill the eight columns
};

// kTwo: an activation as two f16 values, x = unit * (whole + rest / 2048), with nothing lost: `unit` takes the group's largest to a whole part
// of 2^10 .. 2^11, and the rest, at most half, keeps the bits below (an f16 of any size has eleven in all). The products of codes and whole
// parts then sum to whole numbers below 2^24, which the matrix unit, that truncates its sums, gives exactly; what it drops of the rests' sum
// is 2^-11 of what it would drop of the activations'.
constexpr float kStepRest = 2048.f;
__device__ __forceinline__ float step_group_unit(uint32_t top) {           // top: bits of the largest f16 magnitude
  const uint32_t e = __float_as_uint(__half2float(__ushort_as_half((unsigned short)top))) >> 23;   // 0: all zeros, 255: not finite
  return e == 0u || e == 255u ? 1.f : __uint_as_float((e - 10u) << 23);
}
__device__ __forceinline__ void step_parts(float x, float& whole, float& rest) {
  whole = rintf(x);
  const float r = (x - whole) * kStepRest;
  rest = r == r ? r : 0.f;                                                 // (infinities: all in `whole`)
}

// Tile row of MMA row g (0..7). The 16-byte pieces of a row lie XORed with row mod 8; these orders make the rows of each phase
// of a fragment load (four rows x 32 bytes, two rows x 64) fall on different banks.
template <int BITS>
__device__ __forceinline__ uint32_t step_row(uint32_t g) {
  if constexpr (BITS == 4) return 2u * (g & 3u) + (g >> 2);
  if constexpr (BITS == 8) return 4u * (g & 1u) + (g >> 1);
  return g;
}

__device__ __forceinline__ uint32_t step_ld_acquire(const uint32_t* a) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ void step_cp4_zfill(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned long long step_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void step_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f), "f"(0.f), "f"(0.f), "f"(0.f));
}
__device__ __forceinline__ void step_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What one CTA and one warp have to do for a matmul. A tile is 16 rows of the weight; in the paired form (gate rows, then up
// rows) eight gate rows and the eight up rows they belong to.
struct StepShare {
  uint32_t r0, rows, tiles, rg, ks;
  uint32_t rounds, nkt;     // of this warp: tiles rg, rg + RG, ..; slices ks, ks + KS, ..
};
__device__ __forceinline__ StepShare step_share(const StepOp& o, uint32_t warp) {
  StepShare s;
  const uint32_t b = blockIdx.x;
  s.rows = o.rows + (b < o.more ? 1u : 0u);
  s.r0 = b * o.rows + (b < o.more ? b : o.more);
  s.tiles = o.pair ? (s.rows + 7u) >> 3 : (s.rows + 15u) >> 4;
  s.rg = (warp * o.ks_inv) >> 16;
  s.ks = warp - s.rg * o.ks;
  s.nkt = o.nkt - ((o.nkt - 1u) * o.ks + s.ks < o.slices ? 0u : 1u);
  s.rounds = s.nkt && s.rg < o.rg && s.rg < s.tiles ? ((s.tiles - s.rg + o.rg - 1u) * o.rg_inv) >> 16 : 0u;
  return s;
}

// AL: K is whole slices and the tables allow a slice's scales to be copied in one piece.
template <int BITS, bool G32, bool AFFINE, bool AL, int MAX>
__global__ void __launch_bounds__(kStepWarps * 32, 1)
step_kernel(const __grid_constant__ StepProgramT<MAX> p) {
  using C = StepFmt<BITS, G32, AFFINE, AL>;
  constexpr int G = C::kG, RPI = C::kRuns, kR = kStepRounds;
  // the sum of a run is kUnit * (kRatio * lo + hi)
  static_assert(AFFINE || C::kTwo, "symmetric sums are taken in units of the products");
  constexpr float kRatio = BITS == 4 ? 16.f : 1.f, kUnit = BITS == 4 ? 1048576.f : 16777216.f;
  extern __shared__ __align__(128) uint8_t step_smem[];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t g = lane >> 2, c = lane & 3u;
  const uint32_t n = p.n;
  // The matmuls' descriptions: read from shared memory (as kernel parameters under a running index each one cost every warp a string of
  // misses of the constant cache, 2 us and more per matmul).
  const StepOp* ops = p.op;
  if constexpr (MAX > 1) {
    const uint4* const from = reinterpret_cast<const uint4*>(p.op);
    uint4* const to = reinterpret_cast<uint4*>(step_smem + p.off_ops);
    for (uint32_t i = tid; i < n * (uint32_t)(sizeof(StepOp) / 16); i += kStepWarps * 32u) to[i] = from[i];
    __syncthreads();
    ops = reinterpret_cast<const StepOp*>(to);
  }
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(step_smem) + warp * (kStepDepth * C::kStage);
  float* const partial = reinterpret_cast<float*>(step_smem + p.off_part);        // [2][warps][kStepPitch]
  uint8_t* const xs = step_smem + p.off_x;
  float* const xsum = reinterpret_cast<float*>(step_smem + p.off_xsum);           // per scale group (kTwo: and the groups' units, behind them)

  // ---- producer: a stage at a time, in the order the warp consumes them ---------------------------------------------
  // This lane's pieces of a stage: 16 bytes (8 where 3-bit rows may start between them) of kPieces rows.
  constexpr uint32_t kPiece = BITS == 3 && !AL ? 8u : 16u, kPer = C::kRowBytes / kPiece, kPieces = 16u * kPer / 32u;
  uint32_t cp_row[BITS == 3 ? kPieces : 1], cp_dst[BITS == 3 ? kPieces : 1];
  const uint32_t cp_col = BITS == 3 ? 0u : (lane & 7u) * 16u;
  if constexpr (BITS == 3) {
#pragma unroll
    for (uint32_t i = 0; i < kPieces; ++i) {
      const uint32_t q = lane + 32u * i;
      cp_row[i] = q / kPer;
      cp_dst[i] = cp_row[i] * 96u + q % kPer * kPiece;
    }
  } else {
    // rows lane / 8 + 4 i: the pieces of rows r and r + 4 swizzle alike but for one bit
    cp_row[0] = lane >> 3;
    cp_dst[0] = cp_row[0] * 128u + (((lane & 7u) ^ cp_row[0]) << 4);
  }
  const uint32_t sb_row = AFFINE ? lane >> 1 : lane & 15u, sb_tab = AFFINE ? lane & 1u : 0u;
  const bool sb_on = AFFINE || lane < 16u;
  const uint32_t sb_dst = C::kCodes + sb_row * C::kSbRow + sb_tab * C::kSbSlot;
  // Where the warp stands: running addresses of this lane's first piece and of its scales, rows from the tile's first one on.
  // What a run of tiles shares is looked up once (a chain of constant loads per stage cost 1.7 us in 10 on 24576 x 4096, loads alone).
  uint32_t p_op = 0, p_kt = 0, p_rbeg = 0, p_left = 0, p_pitch = 0, p_rpt = 16, p_rowstep = 0, p_sstep = 0, p_cut = 0, p_run = 0, p_nkt = 0;
  uint32_t p_rem = 0;
  const uint8_t *p_src = nullptr, *p_sp = nullptr;
  size_t p_half = 0;                         // from a tile's rows 0..7 to its rows 8..15
  auto cut_of = [&](const StepOp& o, uint32_t sl) {          // scales and bytes of slice sl that exist
    const uint32_t have = o.spr - sl * (uint32_t)G, left = o.KP * 4u - sl * (uint32_t)C::kRowBytes;
    return (have < (uint32_t)G ? have : (uint32_t)G) << 16 | (left < (uint32_t)C::kRowBytes ? left : (uint32_t)C::kRowBytes);
  };
  auto p_place = [&]() {                     // a run of tiles starts: K tile p_kt, rounds from p_rbeg on
    const StepOp& o = ops[MAX > 1 ? p_op : 0u];
    const StepShare s = step_share(o, warp);
    const uint32_t sl = p_kt * o.ks + s.ks, t = p_rbeg * o.rg + s.rg;
    p_rpt = o.pair ? 8u : 16u;
    p_pitch = o.KP * 4u;
    p_rowstep = o.rg * p_rpt;
    p_rem = s.rows - t * p_rpt;
    const uint32_t row = s.r0 + t * p_rpt;
    p_half = (size_t)(o.pair ? o.pair : 8u) * p_pitch;
    p_src = reinterpret_cast<const uint8_t*>(o.W) + ((size_t)row * p_pitch + sl * (uint32_t)C::kRowBytes);
    if constexpr (BITS != 3) p_src += cp_row[0] * p_pitch + cp_col;
    const uint32_t srow = row + (sb_row & 7u) + (sb_row >> 3) * (o.pair ? o.pair : 8u);
    p_sp = reinterpret_cast<const uint8_t*>((sb_tab ? o.B : o.S) + ((size_t)srow * o.spr + sl * (uint32_t)G));
    p_sstep = p_rowstep * o.spr * 2u;
    if constexpr (!AL) p_cut = cut_of(o, sl);
    p_nkt = s.nkt;
    p_left = p_run = s.nkt > 1u && s.rounds - p_rbeg > (uint32_t)kR ? (uint32_t)kR : s.rounds - p_rbeg;
  };
  auto p_open = [&]() {                      // the next matmul this warp has a stage of
    p_kt = p_rbeg = 0;
    for (; p_op < n; ++p_op)
      if (step_share(ops[MAX > 1 ? p_op : 0u], warp).rounds) { p_place(); return; }
  };
  auto issue = [&](uint32_t st) {            // st: the stage's place in the ring
    if (p_op < n) {
      if constexpr (BITS == 3) {
#pragma unroll
        for (uint32_t i = 0; i < kPieces; ++i) {
          const uint32_t col = cp_dst[i] - cp_row[i] * 96u, r8 = cp_row[i] & 7u;
          if ((p_rpt == 8u ? r8 : cp_row[i]) < p_rem && (AL || col < (p_cut & 0xffffu))) {
            const uint8_t* const q = p_src + (cp_row[i] >= 8u ? p_half : (size_t)0) + (r8 * p_pitch + col);
            if constexpr (AL) tc_cp16(st + cp_dst[i], q);
            else tc_cp8(st + cp_dst[i], q);
          }
        }
      } else if (AL || cp_col < (p_cut & 0xffffu)) {
        const uint8_t *const q4 = p_src + 4u * p_pitch, *const q8 = p_src + p_half, *const q12 = q8 + 4u * p_pitch;
        const uint32_t d0 = st + cp_dst[0], d4 = st + (cp_dst[0] ^ 64u) + 512u;
        if (p_rem >= p_rpt) {
          tc_cp16(d0, p_src); tc_cp16(d4, q4); tc_cp16(d0 + 1024u, q8); tc_cp16(d4 + 1024u, q12);
        } else {
          const uint32_t r8 = p_rpt == 8u ? 0u : 8u;
          if (cp_row[0] < p_rem) tc_cp16(d0, p_src);
          if (cp_row[0] + 4u < p_rem) tc_cp16(d4, q4);
          if (cp_row[0] + r8 < p_rem) tc_cp16(d0 + 1024u, q8);
          if (cp_row[0] + 4u + r8 < p_rem) tc_cp16(d4 + 1024u, q12);
        }
      }
      if (sb_on && (p_rpt == 8u ? sb_row & 7u : sb_row) < p_rem) {
        const uint32_t dst = st + sb_dst;
        if constexpr (AL) {
          if constexpr (G == 8) tc_cp16(dst, p_sp);
          else if constexpr (G == 4) tc_cp8(dst, p_sp);
          else step_cp4_zfill(dst, p_sp, 4u);
        } else {
          // the aligned words around the row's next G values; what lies past the row's end arrives as zeros
          const uint32_t odd = (uint32_t)reinterpret_cast<uintptr_t>(p_sp) & 2u, end = odd + (p_cut >> 16) * 2u;
          const uint8_t* const q = p_sp - odd;
#pragma unroll
          for (uint32_t w = 0; w <= (uint32_t)G / 2; ++w) {
            const uint32_t k = w * 4u >= end ? 0u : end - w * 4u < 4u ? end - w * 4u : 4u;
            step_cp4_zfill(dst + w * 4u, k ? q + w * 4u : q, k);
          }
        }
      }
      p_src += (size_t)p_rowstep * p_pitch;
      p_sp += p_sstep;
      p_rem -= p_rowstep;
      if (--p_left == 0u) {                  // the run of tiles is done
        if (++p_kt < p_nkt) {                // the same tiles, KS slices on
          const StepOp& o = ops[MAX > 1 ? p_op : 0u];
          const uint32_t back = p_run * p_rowstep;
          p_src += (size_t)(o.ks * (uint32_t)C::kRowBytes) - (size_t)back * p_pitch;
          p_sp += (size_t)(o.ks * (uint32_t)G * 2u) - (size_t)(p_run * p_sstep);
          p_rem += back;
          p_left = p_run;
          if constexpr (!AL) p_cut = cut_of(o, p_kt * o.ks + step_share(o, warp).ks);
        } else {
          const StepShare s = step_share(ops[MAX > 1 ? p_op : 0u], warp);
          p_kt = 0;
          p_rbeg += p_run;
          if (p_rbeg < s.rounds) {
            p_place();
          } else {
            ++p_op;
            p_open();
          }
        }
      }
    }
    tc_commit();
  };
  p_open();
#pragma unroll
  for (uint32_t i = 0; i < (uint32_t)kStepDepth - 1u; ++i) issue(ring + i * C::kStage);

  // everything above reads only weights; activations, outputs and the counters belong to the stream order
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const uint32_t tr = step_row<BITS>(g);                      // tile rows of this lane: tr, tr + 8
  const uint32_t frag = BITS == 3 ? g * 96u + 24u * c : tr * 128u, swz = (tr & 7u) << 4;
  uint32_t st = ring, meet = 0;                               // the stage to consume
  const uint32_t ring_end = ring + kStepDepth * C::kStage;
  bool dead = false;                                          // a wait ran out
  for (uint32_t op = 0; op < n; ++op) {
    const StepOp& o = ops[MAX > 1 ? op : 0u];
    // ---- activations ------------------------------------------------------------------------------------------------
    if (o.wait) {
      if (tid == 0u && !dead) {
        const uint32_t* const cnt = p.counters + (o.wait - 1u);
        const long long t0 = clock64();
        while (step_ld_acquire(cnt) < gridDim.x) {
          if ((unsigned long long)(clock64() - t0) > p.wait_cycles) { dead = true; atomicExch(p.status, 11u); break; }
        }
      }
      __syncthreads();
    }
    // 16-byte pieces; past K, up to whole slices: zeros
    const uint32_t pieces = (o.slices * (uint32_t)C::kSlice + 255u) / 256u * 32u, have = o.K / 8u;
    // (a thread's pieces are asked for three at a time: a long row, one after the other, took a trip to L2 for each)
    auto piece = [&](uint32_t i) {
      return i < have ? __ldcg(reinterpret_cast<const uint4*>(o.X) + i) : make_uint4(0u, 0u, 0u, 0u);      // (other SMs may just have written it)
    };
    constexpr uint32_t kAll = kStepWarps * 32u;
    uint4 v1 = piece(tid), v2 = make_uint4(0u, 0u, 0u, 0u), v3 = v2;
    if (pieces > kAll) { v2 = piece(tid + kAll); v3 = piece(tid + 2u * kAll); }
    for (uint32_t i = tid; i < pieces; i += kAll) {
      const uint4 v = v1;
      v1 = v2; v2 = v3;
      if (pieces > 3u * kAll) v3 = piece(i + 3u * kAll);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      float2 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = __half22float2(u32_as_h2(w[k]));
      float sum = ((x[0].x + x[0].y) + (x[1].x + x[1].y)) + ((x[2].x + x[2].y) + (x[3].x + x[3].y));
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if constexpr (!G32) sum += __shfl_xor_sync(0xffffffffu, sum, 4);
      const bool first = (i & (G32 ? 3u : 7u)) == 0u;
      const uint32_t grp = i / (G32 ? 4u : 8u);
      if constexpr (C::kTwo) {
        uint32_t top = 0u;                                    // the group's largest magnitude, as bits
#pragma unroll
        for (int k = 0; k < 4; ++k) top = max(max(top, w[k] & 0x7fffu), w[k] >> 16 & 0x7fffu);
        top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
        if constexpr (!G32) top = max(top, __shfl_xor_sync(0xffffffffu, top, 4));
        const float unit = step_group_unit(top), scale = 1.f / unit;           // powers of two
        uint32_t whole[4], rest[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float2 a, b;
          step_parts(x[k].x * scale, a.x, b.x);
          step_parts(x[k].y * scale, a.y, b.y);
          whole[k] = h2_as_u32(__floats2half2_rn(a.x, a.y));
          rest[k] = h2_as_u32(__floats2half2_rn(b.x, b.y));
        }
        reinterpret_cast<uint4*>(xs)[i] = make_uint4(whole[0], whole[1], whole[2], whole[3]);
        reinterpret_cast<uint4*>(xs + p.x_bytes)[i] = make_uint4(rest[0], rest[1], rest[2], rest[3]);
        if (first) xsum[p.x_bytes / 64u + grp] = unit;
        if constexpr (!AFFINE) sum *= scale;                  // (symmetric: in units, as the products)
      } else {
        reinterpret_cast<uint4*>(xs)[i] = v;
      }
      if (first) xsum[grp] = sum;
    }
    const StepShare cs = step_share(o, warp);
    const uint32_t pair = o.pair, spr = o.spr, KS = o.ks, RG = o.rg, all_rounds = ((cs.tiles + RG - 1u) * o.rg_inv) >> 16;
    __syncthreads();

    uint32_t xf[C::kB];                                       // B fragments of the slice
    // of columns 2c, 2c + 1, per accumulator set: the sums of x over their groups (0 with a second part) and (kTwo) their units
    unsigned long long xs2[C::kSets], unit2[C::kSets];
    auto load_x = [&](uint32_t sl) {
      // (kTwo: columns 0..3 take the first part of four groups, 4..7 the second)
      const __half* const xr = reinterpret_cast<const __half*>(xs + (C::kTwo && g >= 4u ? p.x_bytes : 0u)) + sl * (uint32_t)C::kSlice;
      const uint32_t gc = C::kTwo ? g & 3u : g;               // the column's group (of its set)
      if constexpr (BITS == 3) {
        // lane (g, c) multiplies the codes of group c, in that group's column; a code's offset in its half goes onto its activation
        __align__(16) __half h[64];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (gc == c) v = *reinterpret_cast<const uint4*>(xr + 64u * c + 8 * i);
          *reinterpret_cast<uint4*>(&h[8 * i]) = v;
        }
        const __half q4 = __float2half(0.25f), q8 = __float2half(0.125f), q32 = __float2half(0.03125f), z = __float2half(0.f);
#pragma unroll
        for (int k = 0; k < kCodes3Views; ++k) {
          const int i = codes3_view_first(k);
          xf[2 * k] = h2_as_u32(__halves2half2(h[i], k < 15 ? __hmul(h[i + 6 < 64 ? i + 6 : 63], q4) : z));
          xf[2 * k + 1] = h2_as_u32(__halves2half2(__hmul(h[i + 1], q8), k < 15 ? __hmul(h[i + 7 < 64 ? i + 7 : 63], q32) : z));
        }
      } else {
        const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int set = 0; set < C::kSets; ++set) {
          constexpr int kRunsPerSet = RPI / C::kSets;
          uint4 v0 = z4, v1 = z4;
          if constexpr (G32) {                                 // (the two pieces of a run are groups of their own)
            v0 = *reinterpret_cast<const uint4*>(xr + 128u * set + 32u * gc + 8u * c);
            v1 = v0;
          } else if (gc < (uint32_t)RPI) {
            v0 = *reinterpret_cast<const uint4*>(xr + 64u * gc + 16u * c);
            v1 = *reinterpret_cast<const uint4*>(xr + 64u * gc + 16u * c + 8u);
          }
          uint32_t b[8];
          Frag<BITS>::b(v0, v1, b);
#pragma unroll
          for (int r = 0; r < kRunsPerSet; ++r)
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              // registers 0, 1, 4, 5 come from the first piece, the others from the second (8-bit: 0..3 and 4..7)
              const bool second = BITS == 8 ? k >= 4 : (k & 2) != 0;
              const uint32_t col = G32 ? 2u * r + (second ? 1u : 0u) : (uint32_t)r;
              xf[(set * kRunsPerSet + r) * 8 + k] = gc == col ? b[k] : 0u;
            }
        }
      }
#pragma unroll
      for (int set = 0; set < C::kSets; ++set) {
        float2 s = make_float2(0.f, 0.f);
        if constexpr (C::kTwo) {
          const float* const at = xsum + sl * (uint32_t)G + 4u * set + 2u * (c & 1u);
          const float2 u = *reinterpret_cast<const float2*>(at + p.x_bytes / 64u);
          const float part = c < 2u ? kUnit : kUnit / kStepRest;
          unit2[set] = tc_pk(u.x * part, u.y * part);
          if (c < 2u) s = *reinterpret_cast<const float2*>(at);
          xs2[set] = AFFINE ? tc_pk(s.x, s.y) : tc_pk(s.x * (1.f / kUnit), s.y * (1.f / kUnit));
        } else {
          if (2u * c < (uint32_t)G) s = *reinterpret_cast<const float2*>(xsum + sl * (uint32_t)G + 2u * c);
          xs2[set] = tc_pk(s.x * (1.f / kUnit), s.y * (1.f / kUnit));  // exact: the accumulators hold results in units of kUnit
        }
      }
    };
    // (AL false) rows whose scales start on an odd group lie one value into their words; tiles start on rows of one parity
    const uint32_t odd_lo = ((cs.r0 + tr) & spr & 1u) * 2u, odd_hi = pair & spr & 1u ? odd_lo ^ 2u : odd_lo;
    // the stage at `st` times the slice, folded into `a`
    auto multiply = [&](unsigned long long (&a)[2]) {
      float lo[C::kSets][4], hi[C::kSets][4];
      const uint32_t at0 = st + frag;
      if constexpr (BITS == 3) {
        uint32_t w[6], u[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const uint2 x = tc_lds64(at0 + 8u * i), y = tc_lds64(at0 + 8u * 96u + 8u * i);
          w[2 * i] = x.x; w[2 * i + 1] = x.y; u[2 * i] = y.x; u[2 * i + 1] = y.y;
        }
#pragma unroll
        for (int k = 0; k < kCodes3Views; ++k) {
          uint32_t w0, w1, u0, u1;
          codes3_inplace(w, k, w0, w1);
          codes3_inplace(u, k, u0, u1);
          if (k == 0) step_mma0(lo[0], w0, u0, w1, u1, xf[2 * k], xf[2 * k + 1]);
          else if (k == 1) step_mma0(hi[0], w0, u0, w1, u1, xf[2 * k], xf[2 * k + 1]);
          else step_mma(k & 1 ? hi[0] : lo[0], w0, u0, w1, u1, xf[2 * k], xf[2 * k + 1]);
        }
      } else {
        using F = Frag<BITS>;
#pragma unroll
        for (int r = 0; r < RPI; ++r) {
          typename F::Raw vg, vh;                              // rows tr, tr + 8 (one swizzle)
          if constexpr (BITS == 8) {
            const uint32_t at = at0 + (((uint32_t)r * 64u + c * 16u) ^ swz);
            vg.w = tc_lds128(at); vh.w = tc_lds128(at + 1024u);
          } else if constexpr (G32) {
            const uint32_t a0 = at0 + (((uint32_t)r * 32u) ^ swz) + c * 4u, a1 = at0 + (((uint32_t)r * 32u + 16u) ^ swz) + c * 4u;
            vg.w = make_uint2(tc_lds32(a0), tc_lds32(a1));
            vh.w = make_uint2(tc_lds32(a0 + 1024u), tc_lds32(a1 + 1024u));
          } else {
            const uint32_t at = at0 + (((uint32_t)r * 32u + (c >> 1) * 16u) ^ swz) + (c & 1u) * 8u;
            vg.w = tc_lds64(at); vh.w = tc_lds64(at + 1024u);
          }
          uint32_t ag[8], ah[8];
          F::a(vg, ag); F::a(vh, ah);
          constexpr int kRunsPerSet = RPI / C::kSets;
          const int set = r / kRunsPerSet;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (r % kRunsPerSet == 0 && h == 0) {
              step_mma0(lo[set], ag[0], ah[0], ag[1], ah[1], xf[r * 8], xf[r * 8 + 1]);
              step_mma0(hi[set], ag[4], ah[4], ag[5], ah[5], xf[r * 8 + 4], xf[r * 8 + 5]);
            } else {
              step_mma(lo[set], ag[2 * h], ah[2 * h], ag[2 * h + 1], ah[2 * h + 1], xf[r * 8 + 2 * h], xf[r * 8 + 2 * h + 1]);
              step_mma(hi[set], ag[4 + 2 * h], ah[4 + 2 * h], ag[5 + 2 * h], ah[5 + 2 * h], xf[r * 8 + 4 + 2 * h], xf[r * 8 + 5 + 2 * h]);
            }
          }
        }
      }
      // column 2c + v of the accumulators is one scale group, or a part of one (columns past the last group fold zeros with any scale)
      const uint32_t sc = st + C::kCodes + tr * C::kSbRow + 2u * (C::kTwo ? 2u * (c & 1u) : (2u * c) % (uint32_t)G);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int set = 0; set < C::kSets; ++set) {
          const uint32_t at = sc + 8u * h * C::kSbRow + 8u * set + (AL ? 0u : h ? odd_hi : odd_lo);
          auto two = [&](uint32_t q) {
            if constexpr (AL) return __half22float2(u32_as_h2(tc_lds32(q)));
            return make_float2(__half2float(__ushort_as_half((unsigned short)tc_lds16(q))),
                               __half2float(__ushort_as_half((unsigned short)tc_lds16(q + 2u))));
          };
          const float2 s = two(at);
          const unsigned long long d = tc_ffma2(tc_pk(lo[set][2 * h], lo[set][2 * h + 1]), tc_pk(kRatio, kRatio), tc_pk(hi[set][2 * h], hi[set][2 * h + 1]));
          const unsigned long long su = C::kTwo ? step_mul2(tc_pk(s.x, s.y), unit2[set]) : tc_pk(s.x, s.y);
          if constexpr (AFFINE) {
            const float2 b = two(at + C::kSbSlot);
            a[h] = tc_ffma2(tc_pk(b.x, b.y), xs2[set], tc_ffma2(su, d, a[h]));
          } else {
            a[h] = tc_ffma2(su, tc_ffma2(tc_pk(-7.f, -7.f), xs2[set], d), a[h]);      // s * sum((q - 7) x)
          }
        }
    };
    if (cs.nkt == 1u) load_x(cs.ks);

    for (uint32_t rb = 0; rb < all_rounds; rb += kR, ++meet) {
      unsigned long long acc[kR][2];
#pragma unroll
      for (int q = 0; q < kR; ++q) acc[q][0] = acc[q][1] = 0ull;
      if (rb < cs.rounds) {
        for (uint32_t kt = 0; kt < cs.nkt; ++kt) {
          if (cs.nkt > 1u) load_x(kt * KS + cs.ks);
#pragma unroll
          for (int q = 0; q < kR; ++q) {
            if (rb + q >= cs.rounds) break;
            issue(st == ring ? ring_end - C::kStage : st - C::kStage);         // into the stage consumed last
            asm volatile("cp.async.wait_group %0;" ::"n"(kStepDepth - 1) : "memory");
            __syncwarp();
            multiply(acc[q]);
            __syncwarp();                                     // every lane is done with the stage before it is refilled
            st = st + C::kStage == ring_end ? ring : st + C::kStage;
          }
        }
      }
      // ---- the K slices of the block meet ----------------------------------------------------------------------------
      const uint32_t nq = all_rounds - rb < (uint32_t)kR ? all_rounds - rb : (uint32_t)kR;
      float* const mine = partial + ((meet & 1u) * kStepWarps + warp) * kStepPitch;
#pragma unroll
      for (int q = 0; q < kR; ++q) {
        if ((uint32_t)q >= nq) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 v2 = tc_unpk(acc[q][h]);
          float v = v2.x + v2.y;
          if constexpr (C::kTwo || G > 2) v += __shfl_xor_sync(0xffffffffu, v, 1);
          if constexpr (C::kTwo || G > 4) v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (c == 0u) mine[q * 16 + tr + 8u * h] = C::kTwo ? v : v * kUnit;
        }
      }
      __syncthreads();
      const float* const buf = partial + (meet & 1u) * (kStepWarps * kStepPitch);
      const uint32_t t0 = rb * RG;                            // first tile of the block
      const uint32_t nt = cs.tiles - t0 < nq * RG ? cs.tiles - t0 : nq * RG;
      auto sum_of = [&](uint32_t tb, uint32_t r16) {          // tb: tile of the block
        const uint32_t q = (tb * o.rg_inv) >> 16, rgi = tb - q * RG;
        const float* const src = buf + rgi * KS * kStepPitch + q * 16u + r16;
        float v = 0.f;
#pragma unroll 4
        for (uint32_t k = 0; k < KS; ++k) v += src[k * kStepPitch];
        return v;
      };
      // A thread per result, beginning with another pair of warps each time: the others are streaming again meanwhile (with all 16
      // warps on the sums 24576 x 4096 took 0.8 us more).
      const uint32_t shift = pair ? 3u : 4u, outs = nt << shift;      // results of a tile: 16, in pairs 8
      for (uint32_t i = (tid + 64u * (meet & 7u)) & (kStepWarps * 32u - 1u); i < outs; i += kStepWarps * 32u) {
        const uint32_t r = i & ((1u << shift) - 1u), tb = i >> shift, row = (t0 << shift) + i;
        if (row >= cs.rows) continue;
        const float v = sum_of(tb, r);
        if (!pair) {
          o.Y[cs.r0 + row] = __float2half_rn(v);
        } else {
          // the activation of the SiLU call that follows, from the rounded values that it would read
          const float vu = sum_of(tb, r + 8u);
          const __half hg = __float2half_rn(v), hu = __float2half_rn(vu);
          __half* const y = o.Y + cs.r0 + row;
          y[0] = hg;
          y[pair] = hu;
          o.H[cs.r0 + row] = __float2half_rn(silu_mul_one(__half2float(hg), __half2float(hu)));
        }
      }
    }
    // ---- for the matmuls that wait for this one ------------------------------------------------------------------------
    if (o.signal) {
      __syncthreads();
      if (tid == 0u) {
        __threadfence();
        atomicAdd(p.counters + op, 1u);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // The last CTA to leave clears the counters for the next launch of this program.
  if (p.counters && tid == 0u && atomicAdd(p.counters + n, 1u) == gridDim.x - 1u) {
    for (uint32_t i = 0; i <= n; ++i) p.counters[i] = 0u;
  }
}

template <int BITS, bool G32, bool AFFINE, bool AL, int MAX>
cudaError_t launch_step_one(const StepProgramT<MAX>& p, size_t smem, int grid, bool together, cudaStream_t st) {
  auto kern = step_kernel<BITS, G32, AFFINE, AL, MAX>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16 || !attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    if (dev < 16) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kStepWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if (together) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  } else {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}
template <int BITS, bool G32, bool AFFINE>
cudaError_t launch_step_format(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st) {
  if (p.n == 1) {
    StepProgramT<1> q;
    q.op[0] = p.op[0];
    q.n = 1; q.x_bytes = p.x_bytes; q.off_part = p.off_part; q.off_x = p.off_x; q.off_xsum = p.off_xsum;
    q.counters = nullptr; q.status = p.status; q.wait_cycles = p.wait_cycles;
    return al ? launch_step_one<BITS, G32, AFFINE, true>(q, smem, grid, false, st) : launch_step_one<BITS, G32, AFFINE, false>(q, smem, grid, false, st);
  }
  return al ? launch_step_one<BITS, G32, AFFINE, true>(p, smem, grid, together, st) : launch_step_one<BITS, G32, AFFINE, false>(p, smem, grid, together, st);
}

}  // namespace ztvm
