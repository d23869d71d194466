// Prefill GEMM, M > 16, 4-bit weights (8-bit ones: below): y[M, N] = x[M, K] * W16[N, K]^T on tcgen05 with the DEQUANTISED WEIGHTS AS THE
// A OPERAND IN TENSOR MEMORY (replaces the matrix-unit GEMMs of int4_matmul.gen.ts:1058-1456; contract of
// ztvm_int4_matmul for M > 16). W16 = f16_rne(fl32(s * q + b)) (or s * (q - 7)), the value the reference's numpy
// dequantiser produces (scripts/make-dsv2-layer-ref.py:108-116); f32 accumulation in tensor memory.
//
// Why this orientation. The weights take the M side of the MMA (128 weight rows = 128 TMEM lanes) and go from the
// dequantisers' registers straight into tensor memory with tcgen05.st; the activations take the N side (up to 256 tokens
// per instruction) and are the only operand read from shared memory: 32 KB per k block instead of 64 + 16 with both
// operands there. D is [weight row][token] in tensor memory.
//
// Roles (640 threads): warp 0 TMA-loads activation tiles (NT tokens x 64 k, 128-byte swizzle); warp 1 allocates tensor
// memory and issues the MMAs; warp 2 TMA-loads packed weight tiles (128 rows x 32 words = four k blocks); warps 3..18
// dequantise: warp w may touch TMEM lanes 32 (w % 4) .. +31, so it owns those 32 weight rows; warp 19 stages scales and biases, eight k
// blocks at a time, as the 8-byte words around each row's groups: rows whose group count is odd (K = 64 x odd) or groups of
// 32 cost the same as aligned groups of 64. (Loading them from global memory in the dequantisers cost a DRAM or L2 latency
// per k block wherever a row's groups did not come as aligned 16-byte vectors: 43 us per 9216 x 3072 launch at 77 rows.)
// Every wait is bounded (status word); on expiry the roles stop and copies in flight are waited for.
//
// Tiles of up to 352 tokens (accumulator 352 + weight slices 128 of the 512 tensor-memory columns; shared memory then has
// room for two packed-weight slots), the tokens dealt evenly to the tiles. A k block costs 0.28 / 0.31 / 0.45 / 0.58 us at
// 64 / 128 / 256 / 352 tokens: at many tokens the MMA's reads and the TMA's writes of the activations share the 128 bytes
// per clock of shared memory, beside a fixed 0.18 us that wider tiles have less often. 24576 x 4096, 1024 tokens: 172 us
// with tiles of 256, 154 us; 6144 x 4096 (192 tiles of 256 on 148 SMs, 144 of 352): 54, 38 us.
//
// 8-bit weights (int8_affine_batched.wgsl multiplies them as f32) may not be rounded, and the MMA truncates its sums (over a K of 6144 3.6e-6
// of the result, all one way). So the slices hold the codes, which f16 has exactly; a k block is one scale group, summed in an
// accumulator of its own and folded in f32 registers, sum += s * acc + b * sum(x): 1.1e-7, as on the warp-level matrix unit (ztvm_batch_mma.cu),
// 1.4e-7. Each of the four teams has its slice, accumulator, sums of activations and f32 sums for itself; they meet at the end.
// Tiles of up to 64 tokens: what bounds them is issue slots (two FMAs and a load per row, token and group, 86 % of the slots of an SM that
// has a tile) at 0.41 to 0.44 us a block. With one accumulator ring for all teams (tiles of 128) every warp waited for every block: 0.5 and
// 0.97 us at 64 and 128 tokens. us against that kernel, 200 tokens: 3072 x 2048 18.1 : 26.4, 12288 x 2048 51.7 : 80.6, 2048 x 6144 28.2 : 44.7; 1000
// tokens 12288 x 2048 196 : 267.
//
// Few tiles (short prompts, small N): the K range is split over a cluster of CTAs. Each CTA keeps the k blocks of its
// share; at the end every CTA sends its f32 partial sums of token slice j to CTA j through distributed shared memory, and
// each reduces and stores its own slice, in CTA order. The sums travel as whole 512-byte rows of a warp, into a place of their own where there is
// room: a CTA then waits for the others to have started, not to have finished (with biases, stores 32 bytes apart into the idle rings, behind a barrier of
// the whole cluster: 4096 x 4096, 128 rows 15.7 us, now 12.5; 200 rows 19.3, 15.1; 3072 x 8192, 128 rows 19.3, 16.0). The exchange stays in the same instance as
// launches without shares, which are up to 1 % slower for its code where K is some 1100: with instances of their own a pass that alternates fetches code anew
// (41 rows of a layer 1280 wide 57.9 -> 61.1 us).
#include "ztvm_kernels.h"
#include "ztvm_stream_mma.cuh"
#include "ztvm_tc.cuh"

namespace ztvm {

constexpr int kTaStages = 4;        // weight slices in tensor memory
constexpr int kTaWChunk = 4;        // k blocks of a slot of the packed-weight ring
constexpr int kTaSbStages = 2;      // scales ring (each stage holds eight k blocks)
constexpr int kTaSbChunk = 8;
constexpr int kTaSbMaxPitch = 40;   // bytes of one row's scales (or biases) in a stage: groups of 32
constexpr int kTaTeamWarps = 4;     // dequantiser warps of a k block (128 rows)
constexpr int kTaDqWarps = 16;      // four teams: team t takes block t of every packed-weight slot, and stage t
constexpr int kTaThreads = 96 + kTaDqWarps * 32 + 32;
constexpr int kTaRows = 128;        // weight rows per CTA = TMEM lanes
constexpr int kTaMaxSplit = 8;

struct GemmTaParams {
  const __half* S;
  const __half* B;   // nullptr: symmetric
  void* Y;
  uint32_t M, N, K, SPR, group_shift, out_f32;
  uint32_t sb_pitch;   // 8 x an odd number: half of the banks apart for neighbouring rows
  uint32_t tile_m;     // tokens of a tile (the last tile of M may hold fewer)
  uint32_t box_rows;   // rows of one activation box: a stage receives whole boxes
  uint32_t* status;
};

template <int NT, int BITS>
struct GemmTaSmem {
  static constexpr int kXBytes = NT * kGemmBK * 2;            // per stage
  static constexpr int kWBytes = kTaRows * 32 * BITS;         // per packed-weight slot: four k blocks, in boxes of 128 bytes a row
  // the widest tile leaves room for two packed-weight slots and for one table of groups of 32 or two of wider groups
  static constexpr int kWStages = NT > 256 ? 2 : BITS == 8 ? 4 : 3;
  static constexpr int kSbBytes = NT > 256 ? 2 * kTaRows * 24 : 2 * kTaRows * kTaSbMaxPitch;
  static constexpr int kOffW = kTaStages * kXBytes;
  static constexpr int kOffSb = kOffW + kWStages * kWBytes;
  static constexpr int kOffBar = kOffSb + kTaSbStages * kSbBytes;
  static constexpr int kOffXsum = kOffBar + 256;              // 8-bit: sums of a block's activations per token, two rounds of the stages
  // Partial sums that the other CTAs of a cluster send: a place of their own where there is room, else the idle rings.
  static constexpr bool kApart = NT <= 128 && BITS == 4;
  static constexpr int kPartBytes = (NT + 56) * kTaRows * 4;
  static constexpr int kOffPart = kApart ? (kOffXsum + 127) / 128 * 128 : 0;
  static constexpr int kTotal = kApart ? kOffPart + kPartBytes : kOffXsum + (BITS == 8 ? 2 * kTaStages * NT * 4 : 0);
  static_assert(kTotal + 1024 <= 227 * 1024 && (kApart || kPartBytes <= kTaStages * kXBytes + kWStages * kWBytes), "shared memory of a CTA");
  static constexpr int kAccs = BITS == 8 ? kTaStages : 1;     // accumulators: 8-bit blocks have one each
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr) : "memory");
}
// acc + the two halves of h
__device__ __forceinline__ float ta_add2(float acc, uint32_t h) {
  asm("{\n\t.reg .f16 a, b, one;\n\tmov.b16 one, 0x3C00;\n\tmov.b32 {a, b}, %1;\n\t"
      "fma.rn.f32.f16 %0, a, one, %0;\n\tfma.rn.f32.f16 %0, b, one, %0;\n\t}" : "+f"(acc) : "r"(h));
  return acc;
}

template <int NT, bool AFFINE, int BITS>
__global__ void __launch_bounds__(kTaThreads, 1)
gemm_ta_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                  const GemmTaParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  using L = GemmTaSmem<NT, BITS>;
  constexpr int kTaWStages = L::kWStages;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t x_ring = base, w_ring = base + L::kOffW, bars = base + L::kOffBar;
  auto bar_full = [&](int s) { return bars + 8u * s; };
  auto bar_empty = [&](int s) { return bars + 8u * (kTaStages + s); };
  auto bar_w_full = [&](int s) { return bars + 8u * (2 * kTaStages + s); };
  auto bar_w_empty = [&](int s) { return bars + 8u * (2 * kTaStages + kTaWStages + s); };
  auto bar_sb_full = [&](int s) { return bars + 8u * (2 * kTaStages + 2 * kTaWStages + s); };
  auto bar_sb_empty = [&](int s) { return bars + 8u * (2 * kTaStages + 2 * kTaWStages + kTaSbStages + s); };
  constexpr int kBarAccum = 2 * kTaStages + 2 * kTaWStages + 2 * kTaSbStages;
  // 8-bit: activations landed (in `full` otherwise)
  auto bar_x = [&](int s) { return BITS == 8 ? bars + 8u * (kBarAccum + 1 + s) : bars + 8u * s; };
  constexpr int kNumBars = kBarAccum + 1 + (BITS == 8 ? kTaStages : 0);
  static_assert(8 * kNumBars + 8 <= 256, "barrier block");
  const uint32_t bar_accum = bars + 8u * kBarAccum;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen_base + L::kOffBar + 8 * kNumBars);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t n0 = blockIdx.x * kTaRows;
  const uint32_t m0 = blockIdx.y * p.tile_m;
  const uint32_t mrows = p.M - m0 < p.tile_m ? p.M - m0 : p.tile_m;     // tokens of this tile
  // k blocks of this CTA: whole scale stages, so that every share starts on a multiple of eight
  const uint32_t split = gridDim.z, kz = blockIdx.z;
  const uint32_t all_kb = p.K / kGemmBK, units = (all_kb + kTaSbChunk - 1) / kTaSbChunk;
  const uint32_t kb_first = kz * units / split * kTaSbChunk;
  const uint32_t kb_last = kz + 1 == split ? all_kb : (kz + 1) * units / split * kTaSbChunk;
  const uint32_t num_kb = kb_last - kb_first;
  constexpr uint32_t kColA = NT * L::kAccs;                      // weight slices start after the accumulator columns
  constexpr uint32_t kTmemCols = kColA + kTaStages * 32 <= 256 ? 256 : 512;
  static_assert(kColA + kTaStages * 32 <= 512, "tensor memory");
  const uint32_t nbox = mrows > p.box_rows ? 2u : 1u, box_bytes = p.box_rows * (uint32_t)(kGemmBK * 2);

  if (threadIdx.x == 32) { tma_prefetch_desc(&tmap_x); tma_prefetch_desc(&tmap_w); }
  auto load_x = [&](uint32_t s, uint32_t kb) {
    mbar_arrive_expect_tx(bar_x((int)s), nbox * box_bytes);
    for (uint32_t b = 0; b < nbox; ++b)
      tma_load_2d(x_ring + s * L::kXBytes + b * box_bytes, &tmap_x, bar_x((int)s), (int)((kb_first + kb) * kGemmBK), (int)(m0 + b * p.box_rows));
  };
  auto load_w = [&](uint32_t s, uint32_t c) {
    mbar_arrive_expect_tx(bar_w_full((int)s), (uint32_t)L::kWBytes);
#pragma unroll
    for (uint32_t b = 0; b < BITS / 4; ++b)
      tma_load_2d(w_ring + s * L::kWBytes + b * (kTaRows * 128), &tmap_w, bar_w_full((int)s), (int)(kb_first * 2u * BITS + c * 8u * BITS + b * 32u), (int)n0);
  };
  // Each TMA producer initialises the barriers its own copies signal and starts its first loads before the block
  // barrier: they fly while tensor memory is allocated.
  if (threadIdx.x == 0) {
    for (int s = 0; s < kTaStages; ++s) {
      // the activation tile (with its byte count) + every warp of the team that writes the slice
      mbar_init(bar_full(s), BITS == 8 ? kTaTeamWarps : 1 + kTaTeamWarps);
      if (BITS == 8) mbar_init(bar_x(s), 1);
      mbar_init(bar_empty(s), BITS == 8 ? 2 : 1);
    }
    for (int s = 0; s < kTaSbStages; ++s) {
      mbar_init(bar_sb_full(s), 32);
      mbar_init(bar_sb_empty(s), kTaDqWarps);
    }
    mbar_init(bar_accum, 1);
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // Programmatic dependent launch: everything before this point (and the weight / scale loads of the other warps)
    // touches nothing the previous kernel in the stream may write; the activations may be its output.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (uint32_t kb = 0; kb < (uint32_t)kTaStages && kb < num_kb; ++kb) load_x(kb, kb);
  }
  if (threadIdx.x == 64) {
    for (int s = 0; s < kTaWStages; ++s) {
      mbar_init(bar_w_full(s), 1);
      mbar_init(bar_w_empty(s), kTaDqWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint32_t nc = (num_kb + kTaWChunk - 1) / kTaWChunk;
    for (uint32_t c = 0; c < (uint32_t)kTaWStages && c < nc; ++c) load_w(c, c);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  // scales: the 8-byte words around the groups of eight k blocks of each row
  const uint32_t sb_groups = (uint32_t)(kTaSbChunk * kGemmBK) >> p.group_shift;       // 16, 8 or 4 per row and stage
  auto load_sb = [&](uint32_t s, uint32_t ch) {
    const uint32_t g0 = ((kb_first + ch * kTaSbChunk) * (uint32_t)kGemmBK) >> p.group_shift;
    const uint32_t have = p.SPR - g0 < sb_groups ? p.SPR - g0 : sb_groups;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t r = (uint32_t)lane + 32u * i;
      const size_t off = (size_t)min(n0 + r, p.N - 1) * p.SPR + g0;
      const uint32_t odd = ((uint32_t)off & 3u) * 2u, end = odd + have * 2u;             // tables start on 8-byte boundaries
#pragma unroll
      for (int tb = 0; tb < (AFFINE ? 2 : 1); ++tb) {
        const uint8_t* src = reinterpret_cast<const uint8_t*>((tb ? p.B : p.S) + off) - odd;
        const uint32_t dst = base + L::kOffSb + s * L::kSbBytes + ((uint32_t)tb * kTaRows + r) * p.sb_pitch;
        for (uint32_t b = 0; b < end; b += 8u)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + b), "l"(src + b), "r"(min(8u, end - b)) : "memory");
      }
    }
  };
  const uint32_t sb_chunks = (num_kb + kTaSbChunk - 1) / kTaSbChunk;
  if (warp == 3 + kTaDqWarps) load_sb(0, 0);       // before the block barrier: weights are not written by the previous kernel
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // That this CTA runs, so that the others of its cluster may write to the place of their sums: nothing was written that they read, so
  // the arrival is relaxed. (As a release it waited for the loads in flight: 4096 x 4096, 128 rows without biases 11.5 us, now 10.9; 2624 x 2624 10.1, 9.7.)
  if (L::kApart && split > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const int quarter = warp & 3;                       // TMEM lanes this warp may touch: [32 * quarter, +32)
  const uint32_t wpart = (uint32_t)(warp - 3) >> 2;   // dequantisers: 0..3
  const uint32_t r_tile = (uint32_t)(quarter * 32 + lane);
  const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
  const bool is_dq = warp >= 3 && warp < 3 + kTaDqWarps;
  bool acc_ok = false;

  if (warp == 0) {
    // ================= TMA producer: activations =================
    if (elect_one()) {
      uint32_t issued = num_kb < (uint32_t)kTaStages ? num_kb : (uint32_t)kTaStages;
      for (uint32_t kb = issued; kb < num_kb; ++kb) {
        const int s = kb % kTaStages;
        const uint32_t ph = (kb / kTaStages) & 1u;
        if (!mbar_wait(bar_empty(s), ph ^ 1u, p.status, 1u, abort_flag)) break;
        load_x((uint32_t)s, kb);
        issued = kb + 1;
      }
      if (*abort_flag) {   // the consumer stopped: wait (bounded) until the copies already issued have landed
        const uint32_t first = issued > (uint32_t)kTaStages ? issued - kTaStages : 0u;
        for (uint32_t kb = first; kb < issued; ++kb) {
          const long long t0 = clock64();
          while (!mbar_try_wait(bar_x(kb % kTaStages), (kb / kTaStages) & 1u) &&
                 (unsigned long long)(clock64() - t0) < kWaitCycles) {}
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer =================
    if (elect_one()) {
      // an instruction takes up to 256 tokens: a wider tile is two column ranges of the accumulator
      const uint32_t cols = (mrows + 15u) & ~15u, cols_a = cols > 256u ? (cols / 2u + 15u) & ~15u : cols;
      const uint32_t idesc = idesc_f16((int)cols_a), idesc_b = idesc_f16((int)(cols - cols_a));
      const uint64_t b0 = smem_desc_sw128(x_ring);
      uint32_t s = 0, ph = 0;
      // The thread is held at each tcgen05.mma until the pipe takes it, so a barrier poll between two k blocks would
      // be a bubble in the pipe: the next block's barrier is polled once before the last MMA of the current block is
      // issued, in the shadow of the MMAs already queued, and waited for afterwards only if that poll failed.
      bool ok = mbar_wait(bar_full(0), 0u, p.status, 2u, abort_flag);
      if constexpr (BITS == 8) {
        // Each block into its stage's accumulator: the team that wrote the slice had folded what was there before.
        for (uint32_t kb = 0; kb < num_kb && ok; ++kb) {
          ok = mbar_wait(bar_x((int)s), ph, p.status, 3u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bdesc = b0 + (uint64_t)(s * (L::kXBytes >> 4));
#pragma unroll
          for (int k = 0; k < kGemmBK / 16; ++k)
            umma_f16_ta(tmem_base + s * NT, tmem_base + kColA + s * 32u + (uint32_t)(8 * k), bdesc + (uint64_t)(2 * k), idesc, k ? 1u : 0u);
          umma_commit(bar_empty((int)s));
          mbar_arrive(bar_empty((int)s));    // (a plain arrival as well: it passes on what the team wrote to shared memory before its own)
          if (++s == (uint32_t)kTaStages) { s = 0; ph ^= 1u; }
          if (kb + 1 < num_kb) ok = mbar_wait(bar_full((int)s), ph, p.status, 2u, abort_flag);
        }
      } else {
      for (uint32_t kb = 0; kb < num_kb && ok; ++kb) {
        tc_fence_after();
        const uint64_t bdesc = b0 + (uint64_t)(s * (L::kXBytes >> 4));
        const uint32_t a_tmem = tmem_base + kColA + s * 32u;
        uint32_t s1 = s + 1u, ph1 = ph;
        if (s1 == (uint32_t)kTaStages) { s1 = 0; ph1 ^= 1u; }
        bool next_ready = true;
#pragma unroll
        for (int k = 0; k < kGemmBK / 16; ++k) {   // 16 k elements: 8 TMEM columns of A, 32 bytes along the swizzled B row
          if (k == kGemmBK / 16 - 1 && kb + 1 < num_kb) next_ready = mbar_try_wait(bar_full((int)s1), ph1);
          umma_f16_ta(tmem_base, a_tmem + (uint32_t)(8 * k), bdesc + (uint64_t)(2 * k), idesc, (kb | (uint32_t)k) ? 1u : 0u);
          if (NT > 256 && cols > cols_a)
            umma_f16_ta(tmem_base + cols_a, a_tmem + (uint32_t)(8 * k), bdesc + (uint64_t)(cols_a * 8u + 2 * k), idesc_b, (kb | (uint32_t)k) ? 1u : 0u);
        }
        umma_commit(bar_empty((int)s));   // the activation tile and the weight slice are free once these MMAs have read them
        if (!next_ready) ok = mbar_wait(bar_full((int)s1), ph1, p.status, 2u, abort_flag);
        s = s1; ph = ph1;
      }
      if (ok) umma_commit(bar_accum);
      }
    }
  } else if (warp == 2) {
    // ================= TMA producer: packed weights =================
    if (elect_one()) {
      const uint32_t num_chunks = (num_kb + kTaWChunk - 1) / kTaWChunk;
      uint32_t issued = num_chunks < (uint32_t)kTaWStages ? num_chunks : (uint32_t)kTaWStages;
      for (uint32_t c = issued; c < num_chunks; ++c) {
        const int s = c % kTaWStages;
        const uint32_t ph = (c / kTaWStages) & 1u;
        if (!mbar_wait(bar_w_empty(s), ph ^ 1u, p.status, 6u, abort_flag)) break;
        load_w((uint32_t)s, c);
        issued = c + 1;
      }
      if (*abort_flag) {
        const uint32_t first = issued > (uint32_t)kTaWStages ? issued - kTaWStages : 0u;
        for (uint32_t c = first; c < issued; ++c) {
          const long long t0 = clock64();
          while (!mbar_try_wait(bar_w_full(c % kTaWStages), (c / kTaWStages) & 1u) &&
                 (unsigned long long)(clock64() - t0) < kWaitCycles) {}
        }
      }
    }
  } else if (!is_dq) {
    // ================= scales and biases =================
    for (uint32_t ch = 0; ch < sb_chunks; ++ch) {
      const uint32_t s = ch % kTaSbStages;
      bool ok = true;
      if (ch >= (uint32_t)kTaSbStages) ok = mbar_wait(bar_sb_empty((int)s), ((ch / kTaSbStages) & 1u) ^ 1u, p.status, 8u, abort_flag, 400u);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (ch) load_sb(s, ch);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_sb_full((int)s)) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ================= dequantisers (warps 3..18) =================
    // Four teams of four warps; thread (quarter, lane) of team t dequantises the 64 codes of weight row 32 quarter + lane
    // in block t of every slot. Issue slots bound this part: a whole row of a block per thread (instead of half, with
    // teams of eight) halves the waits, scale look-ups and guards per code, and four blocks are in flight at once, so a
    // team's chain of wait, load, dequantise, store, arrive may take as long as four blocks.
    static_assert(kTaStages == kTaWChunk && kTaDqWarps == kTaWChunk * kTaTeamWarps, "a team per stage");
    const uint32_t team = wpart;
    const uint8_t* const wrow_sm = gen_base + L::kOffW + (r_tile >> 3) * 1024 + (r_tile & 7) * 128;
    [[maybe_unused]] const uint32_t w_at0 = ((team * 2u) ^ (r_tile & 7)) << 4, w_at1 = ((team * 2u + 1u) ^ (r_tile & 7)) << 4;
    const uint32_t sb_odd = (uint32_t)(((size_t)min(n0 + r_tile, p.N - 1) * p.SPR) & 3u) * 2u;   // (stages start on multiples of four groups)
    const uint8_t* const sb_row = gen_base + L::kOffSb + r_tile * p.sb_pitch + sb_odd;
    const uint32_t b_delta = (uint32_t)kTaRows * p.sb_pitch;
    const uint32_t st_at = tmem_base + lane_base + kColA + team * 32u;
    bool ok = true;
    if constexpr (BITS == 8) {
      static_assert(kTaWStages == 4, "slots of the packed ring by c & 3");
      // Codes go to tensor memory masked where they sit, as f16 subnormals (products q * 2^-24 * x, exact). A team takes its block's
      // accumulator back and folds it into f32 registers: a thread has its weight row and all tokens of the tile. Slice, accumulator
      // and sums of activations are the team's own, so teams wait for nothing but their own MMAs. What round c - 1 left is folded
      // before round c overwrites it; the sums of activations alternate between two places, as a warp may be a round ahead of another.
      float* const xsum = reinterpret_cast<float*>(gen_base + L::kOffXsum) + team * NT;
      unsigned long long sum[NT / 2];
#pragma unroll
      for (int i = 0; i < NT / 2; ++i) sum[i] = 0ull;
      for (uint32_t c = 0;; ++c) {
        if (c > 0) {
          const uint32_t d = c - 1u, sbs = (d >> 1) & 1u;
          if (d * kTaWChunk + team < num_kb) {
            if (ok && (d & 1u) == 0u) ok = mbar_wait(bar_sb_full((int)sbs), (d >> 2) & 1u, p.status, 9u, abort_flag);
            if (ok) ok = mbar_wait(bar_empty((int)team), d & 1u, p.status, 4u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok) {
              const uint8_t* const sp = sb_row + sbs * L::kSbBytes + ((d & 1u) * kTaWChunk + team) * 2u;
              const float sf = __half2float(*reinterpret_cast<const __half*>(sp)), bf = __half2float(*reinterpret_cast<const __half*>(sp + b_delta));
              const unsigned long long s2 = tc_pk(sf * 16777216.f, sf * 16777216.f), b2 = tc_pk(bf, bf);
              const ulonglong2* const xs = reinterpret_cast<const ulonglong2*>(xsum + (d & 1u) * (kTaStages * NT));
#pragma unroll
              for (int h = 0; h < NT / 16; ++h) {
                if (16u * h >= mrows) break;
                uint32_t v[16];
                tmem_ld16(tmem_base + lane_base + team * NT + 16u * h, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const ulonglong2 x = xs[4 * h + i];
                  unsigned long long* const to = sum + 8 * h + 2 * i;
                  to[0] = tc_ffma2(b2, x.x, tc_ffma2(s2, tc_pk(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1])), to[0]));
                  to[1] = tc_ffma2(b2, x.y, tc_ffma2(s2, tc_pk(__uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])), to[1]));
                }
              }
            }
          }
          __syncwarp();
          if (lane == 0 && ((d & 1u) || c * kTaWChunk >= num_kb)) mbar_arrive(bar_sb_empty((int)sbs));
        }
        if (c * kTaWChunk >= num_kb) break;
        if (c * kTaWChunk + team < num_kb) {
          if (ok) ok = mbar_wait(bar_w_full((int)(c & 3u)), (c >> 2) & 1u, p.status, 7u, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (ok) {
            const uint8_t* const wl = wrow_sm + (c & 3u) * L::kWBytes + (team >> 1) * (kTaRows * 128);
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
              uint32_t a[16];
#pragma unroll
              for (uint32_t j = 0; j < 2; ++j) {
                const uint4 w = *reinterpret_cast<const uint4*>(wl + ((((team & 1u) * 4u + 2u * h + j) ^ (r_tile & 7)) << 4));
                const uint32_t q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { a[8 * j + 2 * i] = codes8_pair01(q[i]); a[8 * j + 2 * i + 1] = codes8_pair23(q[i]); }
              }
              tmem_st16(st_at + 16u * h, a);
            }
            // meanwhile: sums of the block's activations, two threads per token
            ok = mbar_wait(bar_x((int)team), c & 1u, p.status, 3u, abort_flag);
            static_assert(NT * 2 == kTaRows, "two threads of a team per token");
            const uint32_t token = r_tile >> 1, part = r_tile & 1u;
            const uint8_t* const xr = gen_base + team * L::kXBytes + token * 128u;
            float x0 = 0.f, x1 = 0.f, x2 = 0.f, x3 = 0.f;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
              const uint4 w = *reinterpret_cast<const uint4*>(xr + (((part * 4u + j) ^ (token & 7u)) << 4));
              x0 = ta_add2(x0, w.x); x1 = ta_add2(x1, w.y); x2 = ta_add2(x2, w.z); x3 = ta_add2(x3, w.w);
            }
            float x = (x0 + x1) + (x2 + x3);
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            if (part == 0u) xsum[(c & 1u) * (kTaStages * NT) + token] = x;
            tmem_st_wait();
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_full((int)team));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_w_empty((int)(c & 3u)));
      }
      // The teams' sums meet in tensor memory, in team order, where the epilogue looks for them.
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
#pragma unroll
        for (int h = 0; h < NT / 16; ++h) {
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) { v[2 * i] = (uint32_t)sum[8 * h + i]; v[2 * i + 1] = (uint32_t)(sum[8 * h + i] >> 32); }
          tmem_st16(tmem_base + lane_base + team * NT + 16u * h, v);
        }
        tmem_st_wait();
      }
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(kTaDqWarps * 32) : "memory");
      tc_fence_after();
      if (ok && team * (NT / 4) < mrows) {
        uint32_t v[16], u[16];
        tmem_ld16(tmem_base + lane_base + team * (NT / 4), v);
#pragma unroll
        for (uint32_t t = 1; t < 4; ++t) {
          tmem_ld16(tmem_base + lane_base + t * NT + team * (NT / 4), u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(u[i]));
        }
        tmem_st16(tmem_base + lane_base + team * (NT / 4), v);
        tmem_st_wait();
      }
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(kTaDqWarps * 32) : "memory");
    } else {
    uint32_t ws = 0, wph = 0, ss = 0, sph = 0;          // slot and phase of the packed ring and of the scales ring
    for (uint32_t c = 0; c * kTaWChunk < num_kb; ++c) {
      if (c * kTaWChunk + team < num_kb) {
        if (ok && (c & 1u) == 0u) ok = mbar_wait(bar_sb_full((int)ss), sph, p.status, 9u, abort_flag);
        if (ok) ok = mbar_wait(bar_w_full((int)ws), wph, p.status, 7u, abort_flag);
        uint32_t a[32];
        if (ok) {
          const uint8_t* const wl = wrow_sm + ws * L::kWBytes;
          const uint4 w0 = *reinterpret_cast<const uint4*>(wl + w_at0), w1 = *reinterpret_cast<const uint4*>(wl + w_at1);
          const uint32_t k0 = ((c & 1u) * kTaWChunk + team) * (uint32_t)kGemmBK;
          const uint8_t* const sp = sb_row + ss * L::kSbBytes + (k0 >> p.group_shift) * 2u;
          const DqGroup dq = dq_group<AFFINE>(*reinterpret_cast<const unsigned short*>(sp),
                                              AFFINE ? *reinterpret_cast<const unsigned short*>(sp + b_delta) : (unsigned short)0);
          DqGroup dq2 = dq;
          if (p.group_shift == 5)                       // the second half of the block is the next group
            dq2 = dq_group<AFFINE>(*reinterpret_cast<const unsigned short*>(sp + 2),
                                   AFFINE ? *reinterpret_cast<const unsigned short*>(sp + b_delta + 2) : (unsigned short)0);
          dequant_block_w16<AFFINE>(w0, w1, dq, dq2, a);
        }
        // the TMEM slice of this stage was last read by the MMAs of the block one slot back
        if (ok && c > 0) {
          ok = mbar_wait(bar_empty((int)team), (c & 1u) ^ 1u, p.status, 4u, abort_flag);
          tc_fence_after();
        }
        if (ok) {
          // 64 weights of this row = 32 TMEM columns (two k-adjacent f16 per column) of this thread's lane
          tmem_st32(st_at, a);
          tmem_st_wait();
        }
        // every lane's stores to tensor memory are complete; one lane signals for the warp (also on abort)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_full((int)team));
      }
      // The slots go back to the producers only after the stores that consumed their words. A team without a block in a
      // short last slot hands them back all the same.
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar_w_empty((int)ws));
        if ((c & 1u) || (c + 1) * kTaWChunk >= num_kb) mbar_arrive(bar_sb_empty((int)ss));
      }
      if (++ws == (uint32_t)kTaWStages) { ws = 0; wph ^= 1u; }
      if (c & 1u) { if (++ss == (uint32_t)kTaSbStages) { ss = 0; sph ^= 1u; } }
    }
    }
    // ---- epilogue: D[weight row][token] in TMEM -> y[token][weight row] ------------------------------------------
    acc_ok = ok && (BITS == 8 || mbar_wait(bar_accum, 0u, p.status, 5u, abort_flag));
    acc_ok = __all_sync(0xffffffffu, acc_ok);            // the loads from tensor memory below are the whole warp's
    tc_fence_after();
    asm volatile("griddepcontrol.wait;" ::: "memory");   // y may still be read by the previous kernel in the stream
    // f16 rows of whole 16-byte pieces: the tile is turned round in the (now idle) activation ring. Phase 1: a thread
    // stores its weight row's 32 tokens of a block as f16 into stage[token][row] (a warp fills 64 consecutive bytes
    // per instruction). Phase 2: half a warp reads one token's 256 bytes and stores them to y in 16-byte pieces.
    // All sixteen warps reach the named barrier (also when a wait ran out: they then skip the memory work).
    static_assert(NT * kTaRows * 2 <= kTaStages * L::kXBytes, "the output stage lives in the activation ring");
    const bool staged = !p.out_f32 && (p.N % 8u) == 0;
    const int ncb = (int)((mrows + 31u) / 32u);
    if (split > 1) {
      // below, with the whole cluster
    } else if (staged) {
      const uint32_t stage = x_ring;
      if (acc_ok) {
#pragma unroll 1
        for (int cb = (int)wpart; cb < ncb; cb += 4) {
          uint32_t v[32];
          tmem_ld32(tmem_base + lane_base + (uint32_t)(cb * 32), v);
          tmem_ld_wait();
          const uint32_t col = stage + (uint32_t)(cb * 32) * (kTaRows * 2u) + r_tile * 2u;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const unsigned short hv = __half_as_ushort(__float2half_rn(__uint_as_float(v[i])));
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(col + (uint32_t)i * (kTaRows * 2u)), "h"(hv) : "memory");
          }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kTaDqWarps * 32) : "memory");
      if (acc_ok) {
        const uint32_t w16 = (uint32_t)(warp - 3);                 // 0..15
        const uint32_t sub = (uint32_t)lane >> 4, piece = (uint32_t)lane & 15u;
        const uint32_t n = n0 + piece * 8u;
        const uint4* const stage_g = reinterpret_cast<const uint4*>(gen_base);
#pragma unroll 4
        for (uint32_t t = w16 * 2u + sub; t < mrows; t += 2u * kTaDqWarps) {
          if (n < p.N)
            *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.Y) + (size_t)(m0 + t) * p.N + n) = stage_g[t * (kTaRows * 2u / 16u) + piece];
        }
      }
    } else if (acc_ok) {
      const uint32_t n = n0 + r_tile;
      // the four warps of a quarter take the 32-token blocks in turn
#pragma unroll 1
      for (int cb = (int)wpart; cb < ncb; cb += 4) {
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_base + (uint32_t)(cb * 32), v);
        tmem_ld_wait();
        const uint32_t m_first = m0 + cb * 32;
        if (n < p.N) {
          if (p.out_f32) {
            float* dst = reinterpret_cast<float*>(p.Y) + (size_t)m_first * p.N + n;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (cb * 32 + i < (int)mrows) dst[(size_t)i * p.N] = __uint_as_float(v[i]);
          } else {
            __half* dst = reinterpret_cast<__half*>(p.Y) + (size_t)m_first * p.N + n;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (cb * 32 + i < (int)mrows) dst[(size_t)i * p.N] = __float2half_rn(__uint_as_float(v[i]));
          }
        }
        __syncwarp();   // lanes past N are back before the next load, which takes the whole warp
      }
    }
  }
  if (split > 1) {
    // ---- K shares meet: token blocks of eight, dealt to the CTAs in runs of `per`; partial sums as [sender][block][half][row][4
    // tokens], so that a warp's stores and loads are contiguous. Every thread of the cluster takes both barriers, whatever became of its waits.
    const uint32_t nb = (mrows + 7u) / 8u, per = (nb + split - 1) / split;
    __syncwarp();
    if constexpr (L::kApart) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else cluster_sync_all();                             // every CTA's MMAs have read its rings for the last time
    if (is_dq && acc_ok) {
      for (uint32_t b = wpart; b < nb; b += 4u) {
        const uint32_t to = b / per;
        if (to == kz) continue;
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_base + b * 8u, v);
        tmem_ld_wait();
        const uint32_t slot = kz < to ? kz : kz - 1u;     // the receiver's own sums stay in its tensor memory
        uint32_t dst;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(base + L::kOffPart + (((slot * per + b - to * per) * 2u * kTaRows + r_tile) * 16u)), "r"(to));
#pragma unroll
        for (int i = 0; i < 2; ++i)
          asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)(kTaRows * 16) * i), "r"(v[4 * i]), "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (is_dq && acc_ok) {
      const uint32_t n = n0 + r_tile;
      for (uint32_t b = kz * per + wpart; b < nb && b < (kz + 1) * per; b += 4u) {
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_base + b * 8u, v);
        tmem_ld_wait();
        if (n < p.N) {
          float r[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) r[i] = 0.f;
          for (uint32_t z = 0; z < split; ++z) {              // in CTA order, wherever this CTA stands in it
            if (z == kz) {
#pragma unroll
              for (int i = 0; i < 8; ++i) r[i] += __uint_as_float(v[i]);
            } else {
              const float4* const got = reinterpret_cast<const float4*>(gen_base + L::kOffPart) + ((z < kz ? z : z - 1u) * per + b - kz * per) * 2u * kTaRows + r_tile;
              const float4 g0 = got[0], g1 = got[kTaRows];
              r[0] += g0.x; r[1] += g0.y; r[2] += g0.z; r[3] += g0.w;
              r[4] += g1.x; r[5] += g1.y; r[6] += g1.z; r[7] += g1.w;
            }
          }
#pragma unroll
          for (uint32_t i = 0; i < 8; ++i) {
            if (b * 8u + i >= mrows) break;
            const size_t o = (size_t)(m0 + b * 8u + i) * p.N + n;
            if (p.out_f32) reinterpret_cast<float*>(p.Y)[o] = r[i];
            else reinterpret_cast<__half*>(p.Y)[o] = __float2half_rn(r[i]);
          }
        }
        __syncwarp();     // lanes past N are back before the next load, which takes the whole warp
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
}

// ---- host side ---------------------------------------------------------------------------------------------
typedef CUresult (*TaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TaEncodeFn ta_encode_fn() {
  static TaEncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<TaEncodeFn>(ptr);
  }
  return fn;
}

template <int NT, bool AFFINE, int BITS>
static cudaError_t ta_kernel_ready() {
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 16 && attr_set[dev]) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(gemm_ta_kernel<NT, AFFINE, BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmTaSmem<NT, BITS>::kTotal + 1024);
  if (e == cudaSuccess && dev < 16) attr_set[dev] = true;
  return e;
}
struct TaLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  TaLaunch(dim3 grid, int smem, cudaStream_t st) {
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kTaThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = grid.z;
    cfg.attrs = attr;
    cfg.numAttrs = grid.z > 1 ? 2 : 1;
  }
};
template <int NT, bool AFFINE, int BITS>
static cudaError_t launch_ta_one(const CUtensorMap& tx, const CUtensorMap& tw, const GemmTaParams& p, uint32_t split, cudaStream_t st) {
  const cudaError_t e = ta_kernel_ready<NT, AFFINE, BITS>();
  if (e != cudaSuccess) return e;
  TaLaunch l(dim3((p.N + kTaRows - 1) / kTaRows, (p.M + p.tile_m - 1) / p.tile_m, split), GemmTaSmem<NT, BITS>::kTotal + 1024, st);
  return cudaLaunchKernelEx(&l.cfg, gemm_ta_kernel<NT, AFFINE, BITS>, tx, tw, p);
}
// Clusters of `split` CTAs that the device holds at once (a cluster sits inside one GPC, so this is less than SMs / split).
template <int NT, int BITS>
static uint32_t ta_clusters(uint32_t split, int sm_count) {
  if (split == 1) return (uint32_t)sm_count;
  static int known[16][kTaMaxSplit + 1] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 16) return 1;
  int n = known[dev][split];
  if (n == 0) {
    TaLaunch l(dim3(1, 1, split), GemmTaSmem<NT, BITS>::kTotal + 1024, nullptr);
    if (ta_kernel_ready<NT, true, BITS>() != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_ta_kernel<NT, true, BITS>, &l.cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 1;
    }
    known[dev][split] = n;
  }
  return (uint32_t)n;
}

bool gemm_ta_supported(int bits, uint32_t group, uint32_t K) {
  if (bits == 8) return group == 64 && K % kGemmBK == 0;
  return bits == 4 && (group == 32 || group == 64 || group == 128) && K % kGemmBK == 0;
}

template <int BITS>
static uint32_t ta_at_once(uint32_t tm, uint32_t z, int sm_count) {
  if (BITS == 8 || tm <= 64u) return ta_clusters<64, BITS>(z, sm_count);
  if (tm <= 128u) return ta_clusters<128, 4>(z, sm_count);
  return tm <= 256u ? ta_clusters<256, 4>(z, sm_count) : ta_clusters<352, 4>(z, sm_count);
}

cudaError_t launch_gemm_ta(const uint32_t* W, const __half* S, const __half* B, const __half* X, void* Y, uint32_t M, uint32_t N, uint32_t K,
                           int bits, uint32_t group_shift, bool out_f32, uint32_t* status, int sm_count, cudaStream_t st) {
  TaEncodeFn enc = ta_encode_fn();
  if (!enc) return cudaErrorNotSupported;
  // Tokens per tile and K shares, by the time of the busiest SM in cycles. 4-bit, fitted to 1980 shapes (512 to 16384 rows, K of 512 to 12288, 17 to 1100
  // tokens) of which every tile and number of shares was timed, 0.2 % from the best of them on average: a k block takes 340 + 1.4 per token, with biases at least
  // 620; a CTA of a launch without shares 7000 to start, fill its rings and store, and the last ones 12 per token; one of a cluster 7500 + 35 per token, 4 per
  // tile, 2.8 per CTA and 320 for every share beyond two, and 100 + 13 per token with tiles of more than 128 tokens, whose sums have no place of their own. More
  // CTAs than half the SMs: 8 % more with biases, 3 % without. The longest share counts: all are whole scale stages but the last. Clusters run in as many waves as
  // the device can place. The tokens are dealt evenly to the tiles. (us: 4096 x 4096, 128 rows with biases, one share 20.7, two 14.4, three 13.5, four 12.5; 9216
  // x 1472, 24 rows with biases, one 9.4, two 10.0; 9216 x 3072, 200 rows without, whole-K tiles of 100 tokens 14.3, two shares of 200 15.0.) (Groups of 32 with
  // biases do not fit beside the widest tile.) 8-bit: tiles of up to 64 tokens, a block 700 + 2 per token, 8500 and 5300 + 12 per token; the exchange more for
  // every share beyond two.
  const uint32_t units = (K / kGemmBK + kTaSbChunk - 1) / kTaSbChunk, n_tiles = (N + kTaRows - 1) / kTaRows;
  const uint32_t widest = bits == 8 ? 64u : B && group_shift == 5 ? 256u : 352u;
  uint32_t tile_m = 0, split = 1;
  uint64_t best = ~0ull;
  for (uint32_t t = 64; t <= widest; t += 32) {
    if (t > 64u && t - 32u >= M) break;
    const uint32_t m_tiles = (M + t - 1) / t, tm = ((M + m_tiles - 1) / m_tiles + 15u) & ~15u;
    const uint64_t tiles = (uint64_t)n_tiles * m_tiles;
    const uint32_t live = M < tm ? M : tm, by_tokens = 340u + live * 14u / 10u;
    const uint32_t block = bits == 8 ? 700u + 2u * live : B && by_tokens < 620u ? 620u : by_tokens;
    for (uint32_t z = 1; z <= (uint32_t)kTaMaxSplit && z <= units; ++z) {
      if (z > 1 && tiles * z > (uint64_t)sm_count) break;
      const uint32_t at_once = bits == 8 ? ta_at_once<8>(tm, z, sm_count) : ta_at_once<4>(tm, z, sm_count);
      const uint64_t waves = (tiles + at_once - 1) / at_once;
      const uint32_t more = z > 2 ? z - 2u : 0u, all = K / kGemmBK;
      uint64_t cost;
      if (bits == 8) {
        cost = waves * ((z == 1 ? all : (units + z - 1) / z * kTaSbChunk) * block + 8500u + (z == 1 ? 0u : 5300u + (12u + 28u * more) * live));
      } else {
        const uint32_t last = all - (z - 1u) * units / z * kTaSbChunk, others = (units / z + (units % z > 1u ? 1u : 0u)) * kTaSbChunk;
        const uint32_t blocks = z == 1 || last > others ? last : others, per_tile = 40u + 28u * z;
        const uint32_t rest = z == 1 ? 7000u : 7500u + 35u * live + per_tile * (uint32_t)tiles / 10u + 320u * more + (tm > 128u ? 100u + 13u * live : 0u);
        cost = waves * (blocks * block + rest) * (2u * tiles * z <= (uint64_t)sm_count ? 100u : B ? 108u : 103u) / 100u + (z == 1 ? 12u * live : 0u);
      }
      if (cost < best) { best = cost; tile_m = tm; split = z; }
    }
  }
  const cuuint32_t estr[2] = {1, 1};
  CUtensorMap tx, tw;
  const cuuint64_t xdims[2] = {K, M};
  const cuuint64_t xstrides[1] = {(cuuint64_t)K * 2};
  // boxes no taller than the tile: a box much taller than the tensor makes every load slow (22 against 13 us per launch at M = 17)
  const uint32_t box_rows = tile_m > 128u ? (tile_m / 2u + 7u) & ~7u : tile_m < M ? tile_m : (M + 7u) & ~7u;
  const cuuint32_t xbox[2] = {(cuuint32_t)kGemmBK, box_rows};
  CUresult r = enc(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(X), xdims, xstrides, xbox, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
  const cuuint64_t wdims[2] = {K / 32 * (uint32_t)bits, N};
  const cuuint64_t wstrides[1] = {(cuuint64_t)(K / 32 * (uint32_t)bits) * 4};
  const cuuint32_t wbox[2] = {32, (cuuint32_t)kTaRows};
  r = enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint32_t*>(W), wdims, wstrides, wbox, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
  GemmTaParams p;
  p.S = S; p.B = B; p.Y = Y;
  p.M = M; p.N = N; p.K = K; p.SPR = K >> group_shift; p.group_shift = group_shift;
  p.out_f32 = out_f32 ? 1u : 0u;
  p.sb_pitch = group_shift == 5 ? 40u : 24u;
  p.tile_m = tile_m; p.box_rows = box_rows;
  p.status = status;
  if (bits == 8) return launch_ta_one<64, true, 8>(tx, tw, p, split, st);
  const bool affine = B != nullptr;
  if (tile_m > 256u) return affine ? launch_ta_one<352, true, 4>(tx, tw, p, split, st) : launch_ta_one<352, false, 4>(tx, tw, p, split, st);
  if (tile_m > 128u) return affine ? launch_ta_one<256, true, 4>(tx, tw, p, split, st) : launch_ta_one<256, false, 4>(tx, tw, p, split, st);
  if (tile_m > 64u) return affine ? launch_ta_one<128, true, 4>(tx, tw, p, split, st) : launch_ta_one<128, false, 4>(tx, tw, p, split, st);
  return affine ? launch_ta_one<64, true, 4>(tx, tw, p, split, st) : launch_ta_one<64, false, 4>(tx, tw, p, split, st);
}

}  // namespace ztvm
