// Host side of the one-launch decode step (ztvm_step.cuh): which matmuls may share a launch, who waits for whom, how K and the
// rows are dealt to the warps.
#include "ztvm_step.h"

#include <cstring>

namespace ztvm {

namespace {

// Warps along K (ks) and groups of them (rg), by K alone: the order of an output's sum then is the same however the rows are
// dealt, alone or in a run, with or without the activation behind it. The most even deal wins: slices over whole K tiles, times
// warps that have work. A K tile beyond the first costs the activations' fragments anew, so several count three fifths (in a run, us per
// matmul: 9216 x 3072 with 12 warps and one K tile 4.3, with 16 and three 4.75; 5000 x 2112 with 9 and one 4.0, with 15 and three 4.5).
// Fewer than three warps side by side would read rows in pieces of less than 384 bytes.
void step_split(StepOp* o) {
  uint32_t best = 0;
  for (uint32_t ks = (uint32_t)kStepWarps; ks >= 1; --ks) {
    if (ks > o->slices || (ks < 3u && ks < o->slices)) continue;
    const uint32_t rg = (uint32_t)kStepWarps / ks, nkt = (o->slices + ks - 1) / ks;
    const uint32_t busy = 1000u * o->slices * rg / (nkt * (uint32_t)kStepWarps), gain = nkt > 1 ? busy * 3u / 5u : busy;
    if (gain > best) { best = gain; o->ks = ks; o->rg = rg; o->nkt = nkt; }
  }
  o->ks_inv = (65536u + o->ks - 1) / o->ks;
  o->rg_inv = (65536u + o->rg - 1) / o->rg;
}
void step_deal(StepOp* o, int sm_count) {
  o->rows = o->out_rows / (uint32_t)sm_count;
  o->more = o->out_rows % (uint32_t)sm_count;
}

uint32_t slice_codes(int format) { return format == 8 ? 128u : 256u; }
uint32_t groups_per_slice(int format) { return format == 8 ? 2u : format == 4 + 32 ? 8u : 4u; }
// whole slices, and their scales in one aligned piece (rows of 3-bit codes then are whole 16-byte pieces, too)
bool op_aligned(const StepOp& o, int format) {
  const uint32_t g = groups_per_slice(format);
  const uintptr_t tables = reinterpret_cast<uintptr_t>(o.S) | reinterpret_cast<uintptr_t>(o.B);
  return o.spr % g == 0 && (tables & (g * 2u - 1u)) == 0;
}
bool all_aligned(const StepProgram& p, int format) {
  for (uint32_t i = 0; i < p.n; ++i)
    if (!op_aligned(p.op[i], format)) return false;
  return true;
}

}  // namespace

// A launch of its own has nothing to join. Calls one after the other, us, here against the kernels for one projection:
//   8-bit: everywhere (4096 x 4096 5.7 : 6.8, 12000 x 7936 19.4 : 22.5, 1200 x 9024 8.2 : 12.0, 1000 x 576 2.7 : 2.6)
//   3-bit over whole slices: everywhere (1024 x 1024 3.0 : 3.5, 4096 x 4096 5.1 : 5.6, 12000 x 7936 16.3 : 16.8)
//   4-bit with biases, whole slices: long K, which those take in K tiles with a meeting each (1200 x 8960 8.0 : 8.6, 2048 x 12288 7.1 : 9.1),
//     and small ones (4096 x 4096 4.8 : 5.3, 1024 x 4096 3.5 : 4.0; dispatched from Python, 8192 x 2048 4.3 : 5.2; 9216 x 3072 6.4 : 6.1)
//   3-bit in two parts: from a second tile of rows per SM on (3000 x 1600 4.3 : 4.6, 9000 x 2112 7.0 : 10.3, 3072 x 8256 14.7 : 19.9; 1000 x 576
//     3.6 : 2.4, 2048 x 4160 7.6 : 7.5, 512 x 12352 14.1 : 13.3)
//   4-bit in two parts: nowhere by much. K % 256: 1000 x 576 3.0 : 2.1, 9000 x 2112 6.0 : 5.4, 3072 x 8256 11.6 : 8.1, 12000 x 8000 17.7 : 18.8;
//     groups of 32: 8192 x 2048 4.8 : 3.8, 3072 x 8192 7.7 : 7.0, 3072 x 8256 13.2 : 8.0, 4096 x 12288 10.5 : 10.7
bool step_alone_faster(int bits, bool affine, uint32_t N, uint32_t K, int sm_count) {
  if (step_two_parts(bits, !affine, K % 256u == 0)) return bits == 3 && N > 16u * (uint32_t)sm_count;
  return bits != 4 || K >= 7168u || (uint64_t)N * K <= (20u << 20);
}

bool StepBuilder::waits() const {
  for (uint32_t i = 0; i < prog_.n; ++i)
    if (prog_.op[i].wait) return true;
  return false;
}

// Shared memory of the program as it stands; false if its longest activation row does not fit.
bool StepBuilder::layout() {
  StepProgram& p = prog_;
  uint32_t k_most = 0;
  for (uint32_t i = 0; i < p.n; ++i) k_most = k_most < p.op[i].K ? p.op[i].K : k_most;
  const uint32_t k_pad = (k_most + 255u) / 256u * 256u;
  const bool al = all_aligned(p, format_);
  const uint32_t g = groups_per_slice(format_), stage = 16u * ((format_ == 3 ? 96u : 128u) + (format_ == 4 + 32 ? 1u : 2u) * (al ? g * 2u : (g * 2u + 4u + 7u) / 8u * 8u));
  p.off_ops = (uint32_t)(kStepWarps * kStepDepth) * stage;
  p.off_part = p.off_ops + (p.n > 1 ? p.n * (uint32_t)sizeof(StepOp) : 0u);
  p.off_x = p.off_part + 2u * (uint32_t)(kStepWarps * kStepPitch) * 4u;
  const uint32_t parts = step_two_parts(format_ & 31, format_ == 4 + 32, al) ? 2u : 1u;
  p.x_bytes = k_pad * 2u;
  p.off_xsum = p.off_x + parts * p.x_bytes;
  smem_ = p.off_xsum + parts * (k_pad / 32u * 4u);
  return smem_ <= 227u * 1024u;
}

// Waits of matmul i, or false where it may not follow the earlier ones in one launch: its weights are fetched ahead of every wait.
bool StepBuilder::link(uint32_t i) {
  StepProgram& p = prog_;
  uint32_t wait = 0;
  for (uint32_t j = 0; j < i; ++j) {
    for (const Span& w : w_[i])
      if (touches(w, y_[j]) || touches(w, h_[j])) return false;
    if (touches(x_[i], y_[j]) || touches(x_[i], h_[j]) || touches(y_[i], y_[j]) || touches(y_[i], h_[j]) || touches(y_[i], x_[j]) ||
        touches(h_[i], y_[j]) || touches(h_[i], h_[j]) || touches(h_[i], x_[j]))
      wait = j + 1;
    // (an earlier matmul may still be fetching its weights)
    for (const Span& w : w_[j])
      if (touches(w, y_[i]) || touches(w, h_[i])) return false;
  }
  p.op[i].wait = wait;
  for (uint32_t j = 0; j <= i; ++j) p.op[j].signal = 0;
  for (uint32_t j = 1; j <= i; ++j)
    if (p.op[j].wait) p.op[p.op[j].wait - 1].signal = 1;
  return true;
}

bool StepBuilder::add(const GemvParams& g, int bits, int sm_count) {
  StepProgram& p = prog_;
  if (p.n >= (uint32_t)kStepMaxOps || g.M != 1 || g.out_f32 || g.n_more || g.pair_rows || g.K == 0 || g.N == 0 || g.K % 64u) return false;
  const bool sym32 = bits == 4 && g.group_shift == 5 && !g.B;
  if (!sym32 && !(g.group_shift == 6 && g.B && (bits == 4 || bits == 3 || bits == 8))) return false;
  const int format = bits + (sym32 ? 32 : 0);
  if (p.n && format != format_) return false;
  if (g.N > (1u << 22) || (uint64_t)g.N * g.KP * 4 >= (1ull << 32) || (reinterpret_cast<uintptr_t>(g.X) & 15u) || (reinterpret_cast<uintptr_t>(g.W) & 15u) ||
      ((reinterpret_cast<uintptr_t>(g.S) | reinterpret_cast<uintptr_t>(g.B)) & 7u))
    return false;
  const int before = format_;
  format_ = format;
  const uint32_t i = p.n;
  StepOp& o = p.op[i];
  o.W = g.W; o.S = g.S; o.B = g.B; o.X = g.X; o.Y = static_cast<__half*>(g.Y); o.H = nullptr;
  o.out_rows = g.N;
  step_deal(&o, sm_count);
  o.pair = 0;
  o.K = g.K; o.KP = g.KP; o.spr = g.SPR;
  o.slices = (g.K + slice_codes(format) - 1) / slice_codes(format);
  step_split(&o);
  // (one kernel for all of a run, and a matmul's sums are the same in every run)
  if (i && step_two_parts(bits, sym32, op_aligned(o, format)) != step_two_parts(bits, sym32, op_aligned(p.op[0], format))) return false;
  auto span = [](const void* q, uint64_t bytes) { return Span{reinterpret_cast<uintptr_t>(q), reinterpret_cast<uintptr_t>(q) + bytes}; };
  x_[i] = span(g.X, (uint64_t)g.K * 2);
  y_[i] = span(g.Y, (uint64_t)g.N * 2);
  h_[i] = Span{0, 0};
  w_[i][0] = span(g.W, (uint64_t)g.N * g.KP * 4);
  w_[i][1] = span(g.S, (uint64_t)g.N * g.SPR * 2);
  w_[i][2] = g.B ? span(g.B, (uint64_t)g.N * g.SPR * 2) : Span{0, 0};
  p.n = i + 1;
  if (touches(x_[i], y_[i]) || !link(i) || !layout()) {
    p.n = i;
    if (i == 0) format_ = before;
    else link(i - 1);                                          // who signals, without the one refused
    return false;
  }
  return true;
}

bool StepBuilder::add_silu(const void* gate_up, void* h, uint32_t rows, uint32_t ffn, int sm_count) {
  StepProgram& p = prog_;
  if (p.n == 0 || rows != 1) return false;
  const uint32_t i = p.n - 1;
  StepOp& o = p.op[i];
  if (o.pair || o.Y != gate_up || o.out_rows != 2 * ffn) return false;
  const Span hs{reinterpret_cast<uintptr_t>(h), reinterpret_cast<uintptr_t>(h) + (uint64_t)ffn * 2};
  if (touches(hs, y_[i]) || touches(hs, x_[i])) return false;
  for (const Span& w : w_[i])
    if (touches(hs, w)) return false;
  h_[i] = hs;
  if (!link(i)) {
    h_[i] = Span{0, 0};
    link(i);
    return false;
  }
  o.H = static_cast<__half*>(h);
  o.pair = o.out_rows = ffn;
  step_deal(&o, sm_count);
  return true;
}

cudaError_t StepBuilder::launch(uint32_t* counters, uint32_t* status, uint64_t wait_cycles, int sm_count, cudaStream_t st) {
  StepProgram& p = prog_;
  if (p.n == 0) return cudaSuccess;
  if (!layout()) return cudaErrorInvalidValue;
  const bool together = waits();
  p.counters = together ? counters : nullptr;
  p.status = status;
  p.wait_cycles = wait_cycles;
  const bool al = all_aligned(p, format_);
  switch (format_) {
    case 3: return launch_step_w3(p, al, smem_, sm_count, together, st);
    case 8: return launch_step_w8(p, al, smem_, sm_count, together, st);
    case 4: return launch_step_w4(p, al, smem_, sm_count, together, st);
    default: return launch_step_w4g32(p, al, smem_, sm_count, together, st);
  }
}

}  // namespace ztvm
