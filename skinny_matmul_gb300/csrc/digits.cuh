// digits.cuh -- balanced base-256 digits of FP64 values as FP16 MMA operands, shared by the split
// precision kernels (split.cu, split_tsmm.cu).
//
// An FP64 value x of a row or column with shared exponent field E is the 62-bit fixed-point
// integer F = |x| * 2^(1084 - E) (sign kept apart); G = F + 0x8080...80 holds F's balanced digits
// as bytes (byte i = digit i + 128, most significant first).  A digit d in [-128, 127] is exact in
// FP16, and so is every product of two digits and every FP32 sum of up to 2^10 of them.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace skinny {

constexpr int NDIGITS = 8;

// G = F + 0x8080...80 for the 62-bit fixed-point magnitude F of x relative to exponent field E:
// byte i of G (most significant first) is digit i + 128, so the digits are balanced.
// FAST: E > EMIN_FAST, where zeros and subnormal numbers shift out entirely and need no case of their own
constexpr uint32_t EMIN_FAST = 64;
template <bool FAST = false>
__device__ __forceinline__ void g_words(double x, uint32_t E, uint32_t& gh, uint32_t& gl) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t ef = (hi >> 20) & 0x7FF;
  uint64_t F;
  if constexpr (FAST) {
    const uint64_t m9 =
        ((uint64_t)__funnelshift_l(lo, (hi & 0xFFFFFu) | 0x100000u, 9) << 32) | (uint64_t)(uint32_t)(lo << 9);
    asm("shr.u64 %0, %1, %2;" : "=l"(F) : "l"(m9), "r"(E - ef));  // 0 from 64 on
  } else {
    const uint32_t eff = ef ? ef : 1u;
    const uint64_t mant = ((uint64_t)((hi & 0xFFFFFu) | (ef ? 0x100000u : 0u)) << 32) | lo;
    const uint32_t sh = E - eff;
    F = sh < 64 ? ((mant << 9) >> sh) : 0ull;
  }
  const uint64_t G = F + 0x8080808080808080ull;
  gh = (uint32_t)(G >> 32);
  gl = (uint32_t)G;
}

// signs of elements a, b as FP16 factors (a in the low half), and -1152 times them
struct SignPair {
  uint32_t s, c;
};
// (from the words that hold their sign bits)
__device__ __forceinline__ SignPair sign_pair(uint32_t a, uint32_t b) {
  const uint32_t t = __byte_perm(a, b, 0x7632) & 0x80008000u;
  return {t | 0x3C003C00u, t ^ 0xE480E480u};
}
__device__ __forceinline__ SignPair sign_pair(double a, double b) {
  return sign_pair((uint32_t)__double2hiint(a), (uint32_t)__double2hiint(b));
}
// Two FP16 digit pairs of elements a, b (a in the low halves) from one 32-bit word of their G's: the
// digits of its upper (half 0) or lower bytes, the higher one in d0.  A byte g of G becomes the half
// 1024 + g by pairing it with the byte 0x64, and one HFMA2 subtracts 1152 and applies each element's
// sign: (1024 + g - 1152) * s = (g - 128) * s, exact in FP16.  1.25 instructions a digit.
__device__ __forceinline__ void digit_pairs2(uint32_t ga, uint32_t gb, int lower, SignPair sg, uint32_t& d0,
                                             uint32_t& d1) {
  const uint32_t pair = __byte_perm(ga, gb, lower ? 0x4051 : 0x6273);  // [a.b1, b.b1, a.b0, b.b0] or the upper bytes
  auto dig = [&](uint32_t sel) {
    const uint32_t u = __byte_perm(pair, 0x64646464u, sel);
    const __half2 h = __hfma2(*reinterpret_cast<const __half2*>(&u), *reinterpret_cast<const __half2*>(&sg.s),
                              *reinterpret_cast<const __half2*>(&sg.c));
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  d0 = dig(0x4140);
  d1 = dig(0x4342);
}

// A 64-bit integer W times a power of two as a double, by integer instructions (the FP64 pipe does 1.89
// operations a clock); ex: the biased exponent field of the result when W has its leading one at bit
// 63.  Results below the normal range give 0.  Normalise |W| so that its leading one is bit 63, round on bit 10 (ties
// away from zero), and add the exponent field below the leading one, so that a mantissa carry
// raises the exponent.
__device__ __forceinline__ double window_int(long long W, int ex) {
  const uint32_t sgn = (uint32_t)((unsigned long long)W >> 32) & 0x80000000u;
  const unsigned long long m = (unsigned long long)(W < 0 ? -W : W);
  const int z = __clzll((long long)m);                       // 64 for W == 0
  const unsigned long long n = m << (z & 63);                 // leading one at bit 63 (0 for W == 0)
  const unsigned long long r = (n >> 11) + ((n >> 10) & 1);  // 53 bits, or 2^53 after a carry
  const int ef = ex - z;                                      // biased exponent field of the result
  const uint32_t hi = ((uint32_t)(ef - 1) << 20) + (uint32_t)(r >> 32);
  const bool ok = n != 0 && ef > 0;
  return __hiloint2double(ok ? (int)(hi | sgn) : 0, ok ? (int)(uint32_t)r : 0);
}

}  // namespace skinny
