// Fragments of mma.sync.m16n8k16 for packed codes that are never dequantised: a code masked where it sits in a 16-bit
// half is an f16 subnormal, so an AND is the whole conversion and every product with an f16 activation is exact.
//
// One run = the 64 codes of a row that share a scale (groups of 64). The four lanes c = 0..3 of a quad hold 16 codes of
// the run each (codes 16c .. 16c + 15), i.e. the k slots of four MMAs. `A` gives, for one row, the eight registers
// r[2i], r[2i + 1] = the low and high k half of MMA i; `B` gives the matching eight registers from the lane's 16
// activations. The order of codes inside a run is whatever the masks make cheapest -- A and B agree on it.
//   4-bit  MMAs 0, 1: nibbles at bits 0-3 / 8-11 of a half (q * 2^-24), MMAs 2, 3: bits 4-7 / 12-15 (q * 2^-20)
//   3-bit  MMAs 0, 1: fields at bits 0-2 (q * 2^-24),                   MMAs 2, 3: fields at bits 3-5 (q * 2^-21)
//   8-bit  all four: bytes at bits 0-7 (q * 2^-24)
// so sum x*q = kUnit * (kRatio * d0 + d1) with d0 the sum of MMAs 0, 1 and d1 that of MMAs 2, 3 (8-bit: kUnit * d0).
#pragma once
#include "ztvm_device.cuh"

namespace ztvm {

template <int BITS>
struct Frag;

// x0..x15 of the lane as two 16-byte pieces
template <>
struct Frag<4> {
  static constexpr int kRunBytes = 32;
  static constexpr bool kTwoClasses = true;
  static constexpr float kUnit = 1048576.f, kRatio = 16.f;
  struct Raw { uint2 w; };
  // `p`: the lane's first byte of the run in shared memory
  __device__ __forceinline__ static Raw load(const uint8_t* p, int) { return Raw{*reinterpret_cast<const uint2*>(p)}; }
  __host__ __device__ static constexpr uint32_t lane_byte(int c) { return 8u * (uint32_t)c; }
  __device__ __forceinline__ static void a(const Raw& v, uint32_t (&r)[8]) {
    const Inplace4 p = codes4_inplace(v.w.x), q = codes4_inplace(v.w.y);
    r[0] = p.lo04; r[1] = p.lo26; r[2] = q.lo04; r[3] = q.lo26;
    r[4] = p.hi15; r[5] = p.hi37; r[6] = q.hi15; r[7] = q.hi37;
  }
  __device__ __forceinline__ static void b(const uint4& x0, const uint4& x1, uint32_t (&r)[8]) {
    r[0] = __byte_perm(x0.x, x0.z, 0x5410); r[1] = __byte_perm(x0.y, x0.w, 0x5410);
    r[2] = __byte_perm(x1.x, x1.z, 0x5410); r[3] = __byte_perm(x1.y, x1.w, 0x5410);
    r[4] = __byte_perm(x0.x, x0.z, 0x7632); r[5] = __byte_perm(x0.y, x0.w, 0x7632);
    r[6] = __byte_perm(x1.x, x1.z, 0x7632); r[7] = __byte_perm(x1.y, x1.w, 0x7632);
  }
};

template <>
struct Frag<8> {
  static constexpr int kRunBytes = 64;
  static constexpr bool kTwoClasses = false;
  static constexpr float kUnit = 16777216.f, kRatio = 0.f;
  struct Raw { uint4 w; };
  __device__ __forceinline__ static Raw load(const uint8_t* p, int) { return Raw{*reinterpret_cast<const uint4*>(p)}; }
  __host__ __device__ static constexpr uint32_t lane_byte(int c) { return 16u * (uint32_t)c; }
  __device__ __forceinline__ static void a(const Raw& v, uint32_t (&r)[8]) {
    const uint32_t w[4] = {v.w.x, v.w.y, v.w.z, v.w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { r[2 * j] = codes8_pair01(w[j]); r[2 * j + 1] = codes8_pair23(w[j]); }
  }
  // the activations as they lie in memory
  __device__ __forceinline__ static void b(const uint4& x0, const uint4& x1, uint32_t (&r)[8]) {
    r[0] = x0.x; r[1] = x0.y; r[2] = x0.z; r[3] = x0.w;
    r[4] = x1.x; r[5] = x1.y; r[6] = x1.z; r[7] = x1.w;
  }
};

template <>
struct Frag<3> {
  static constexpr int kRunBytes = 24;
  static constexpr bool kTwoClasses = true;
  static constexpr float kUnit = 2097152.f, kRatio = 8.f;
  struct Raw { uint32_t w0, w1; bool odd; };   // the words around the lane's 48 bits, which start in the middle of the first in odd lanes
  // byte 6c of the run: words 0,1 | 1,2 | 3,4 | 4,5; odd lanes start in the middle of their first word
  __host__ __device__ static constexpr uint32_t lane_byte(int c) { return (6u * (uint32_t)c) & ~3u; }
  __device__ __forceinline__ static Raw load(const uint8_t* p, int c) {
    return Raw{*reinterpret_cast<const uint32_t*>(p), *reinterpret_cast<const uint32_t*>(p + 4), (c & 1) != 0};
  }
  __device__ __forceinline__ static void a(const Raw& v, uint32_t (&r)[8]) { codes3_inplace16(v.w0, v.w1, v.odd, r); }
  __device__ __forceinline__ static void a_shifted(const Raw& v, uint32_t (&r)[8]) { codes3_inplace16_shifted(v.w0, v.w1, v.odd, r); }
  __device__ __forceinline__ static void b(const uint4& x0, const uint4& x1, uint32_t (&r)[8]) {
    r[0] = __byte_perm(x0.x, x1.x, 0x5410); r[1] = __byte_perm(x0.y, x1.y, 0x5410);   // codes (0 | 8), (2 | 10)
    r[2] = __byte_perm(x0.z, x1.z, 0x5410); r[3] = __byte_perm(x0.w, x1.w, 0x5410);   // codes (4 | 12), (6 | 14)
    r[4] = __byte_perm(x0.x, x1.x, 0x7632); r[5] = __byte_perm(x0.y, x1.y, 0x7632);   // the odd codes
    r[6] = __byte_perm(x0.z, x1.z, 0x7632); r[7] = __byte_perm(x0.w, x1.w, 0x7632);
  }
};

__device__ __forceinline__ void cp_async16_s(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8_s(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

}  // namespace ztvm
