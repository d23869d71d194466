// A run of one-row matmuls as one persistent launch (ztvm_step.cuh): the program a launch is given and its builder.
#pragma once
#include "ztvm_kernels.h"

namespace ztvm {

constexpr int kStepWarps = 16;
constexpr int kStepDepth = 4;       // stages of a warp's ring
constexpr int kStepRounds = 4;      // row tiles of a warp between two meetings of the K slices
constexpr int kStepPitch = 68;      // floats of a warp's partial sums: 64 rows, warps four banks apart
constexpr int kStepMaxOps = 64;

// Whether a row's activations go to the matrix unit in two parts (step_parts), which make the sums of a scale group exact: where f32 FMAs
// serve a matmul by itself. Error of the f32 sums against 64 bits, relative, N(0, 1) activations / a few large ones among small: groups of
// 32, 3000 x 3072, f32 FMAs 0.96e-7 / 1.8e-7, one part 6.5e-7 / 39e-7, two 0.90e-7 / 1.5e-7. Decode of 8 layers, hidden 3072: 241 us on
// the FMAs, 195 with one part, 218 with two.
constexpr bool step_two_parts(int bits, bool g32, bool al) { return bits != 8 && (g32 || !al); }

struct alignas(16) StepOp {
  const uint32_t* W;
  const __half* S;
  const __half* B;           // nullptr: symmetric
  const __half* X;
  __half* Y;
  __half* H;                 // paired form: f16(up * silu(gate)) of the rounded results
  uint32_t rows, more;       // rows dealt to a CTA (in the paired form the gate rows); the first `more` CTAs have one row more
  uint32_t out_rows;         // all of them
  uint32_t pair;             // 0, or the rows from a gate row to its up row
  uint32_t K, KP, spr;       // KP: words of a weight row, spr: scale groups of one
  uint32_t slices;           // of a stage's width, the last one possibly short
  uint32_t ks, rg, nkt;      // warps side by side along K, groups of them on row tiles of their own, K tiles: by K alone
  uint32_t ks_inv, rg_inv;   // 65536 / ks, / rg, rounded up
  uint32_t wait;             // 1 + the last earlier matmul of the run whose buffers this one reads or overwrites, 0: none
  uint32_t signal;           // a later one waits for this one
};

static_assert(sizeof(StepOp) == 112, "kStepMaxOps of them travel as kernel parameters");

// A launch's parameter. One matmul by itself has a type of its own: 7 KB of parameters would be copied for nothing.
template <int MAX>
struct StepProgramT {
  StepOp op[MAX];
  uint32_t n;
  uint32_t off_ops, off_part, off_x, off_xsum;   // in shared memory, behind the ring
  uint32_t x_bytes;          // of the longest activation row (a row in two parts takes two)
  uint32_t* counters;        // n + 1 words, zero between launches; nullptr where no matmul waits
  uint32_t* status;
  uint64_t wait_cycles;      // limit of a wait
};
using StepProgram = StepProgramT<kStepMaxOps>;

// Collects matmuls of one weight format; `add` refuses what the kernel cannot run together with the ones collected.
class StepBuilder {
 public:
  bool add(const GemvParams& p, int bits, int sm_count);
  // h = f16(up * silu(gate)) of the last matmul's result [gate(ffn) | up(ffn)], if that is what was collected last
  bool add_silu(const void* gate_up, void* h, uint32_t rows, uint32_t ffn, int sm_count);
  int size() const { return (int)prog_.n; }
  bool waits() const;
  void clear() { prog_.n = 0; }
  cudaError_t launch(uint32_t* counters, uint32_t* status, uint64_t wait_cycles, int sm_count, cudaStream_t st);

 private:
  struct Span { uintptr_t lo, hi; };
  bool touches(const Span& a, const Span& b) const { return a.lo < b.hi && b.lo < a.hi; }
  bool link(uint32_t i);
  bool layout();
  StepProgram prog_;
  Span x_[kStepMaxOps], y_[kStepMaxOps], h_[kStepMaxOps], w_[kStepMaxOps][3];
  int format_ = 0;           // bits, + 32 with groups of 32
  uint32_t smem_ = 0;        // shared memory of the program
};

// Whether a one-row matmul that no run takes is faster here than on the kernels for one projection.
bool step_alone_faster(int bits, bool affine, uint32_t N, uint32_t K, int sm_count);

cudaError_t launch_step_w4(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st);
cudaError_t launch_step_w4g32(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st);
cudaError_t launch_step_w8(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st);
cudaError_t launch_step_w3(const StepProgram& p, bool al, size_t smem, int grid, bool together, cudaStream_t st);

}  // namespace ztvm
