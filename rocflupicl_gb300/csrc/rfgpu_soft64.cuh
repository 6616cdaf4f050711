// rfgpu_soft64.cuh - double-precision products on the integer pipes.
//
// GB300 issues one warp-wide FP64 operation per 64 cycles and SM quarter, so
// the FP64 path is bound by its count of FP64 operations while the integer
// pipes idle.  A product of two normal doubles needs no FP64 unit: the exact
// 106-bit product of the significands by four 32 x 32 -> 64 bit multiplies,
// normalised and rounded to nearest-even as IEEE 754 defines it: the bits of
// __dmul_rn.  Measured on GB300: 6.2 ns per warp product and SM against
// 9.6 ns on the FP64 pipe, and it runs beside FP64 sums: a loop of 5
// differences, 15 products and 15 sums takes 2.67 ms with these products
// against 4.13 ms with FP64 ones (2.37 ms without any product).
//
// Operands are zero or have biased exponents in [512, 1534], so that every
// product is a normal number; soft_ok() tests that and callers take the FP64
// unit otherwise.  A zero operand gives a zero of the right sign.
#pragma once

namespace rfgpu {

// Left operand: significand shifted to the top of 64 bits; right operand:
// significand in place.  e holds sign and exponent (the bias taken from the
// left one); z masks the result's upper half: all ones, or the sign bit alone
// for a zero operand, which has significand 0 and the exponent of 1.
struct SoftA {
  unsigned m1, m0, e, z;
};
struct SoftB {
  unsigned m1, m0, e, z;
};

__device__ __forceinline__ bool soft_zero(double x) {
  return (((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x)) == 0u;
}
__device__ __forceinline__ bool soft_ok(double x) {
  const unsigned t = (unsigned)__double2hiint(x) & 0x7fffffffu;
  return t - 0x20000000u < 0x3ff00000u || soft_zero(x);
}
__device__ __forceinline__ SoftA soft_a(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const bool zero = soft_zero(x);
  return SoftA{zero ? 0u : __funnelshift_l(l, h, 11) | 0x80000000u, l << 11,
               zero ? h : (h & 0xfff00000u) - (1023u << 20), zero ? 0x80000000u : 0xffffffffu};
}
__device__ __forceinline__ SoftB soft_b(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const bool zero = soft_zero(x);
  return SoftB{zero ? 0u : (h & 0xfffffu) | 0x100000u, l,
               zero ? h | (1023u << 20) : h & 0xfff00000u, zero ? 0x80000000u : 0xffffffffu};
}

__device__ __forceinline__ double soft_mul(const SoftA &a, const SoftB &b) {
  // h:u:p00 = the product of the significands, its leading bit at bit 115 or
  // 116 of 117: h holds the top 52 or 53 bits
  const unsigned long long p00 = (unsigned long long)a.m0 * b.m0;
  const unsigned long long t = (unsigned long long)a.m0 * b.m1 + (unsigned)(p00 >> 32);
  const unsigned long long u = (unsigned long long)a.m1 * b.m0 + (unsigned)t;
  unsigned long long h = (unsigned long long)a.m1 * b.m1 + (unsigned)(t >> 32);
  h += (unsigned)(u >> 32);
  const unsigned h1 = (unsigned)(h >> 32), h0 = (unsigned)h, l1 = (unsigned)u, l0 = (unsigned)p00;
  // one place left when the leading bit is the lower one
  const unsigned s20 = ~h1 & 0x100000u, s = s20 >> 20;
  unsigned r1 = __funnelshift_l(h0, h1, s), r0 = __funnelshift_l(l1, h0, s);
  const unsigned q = __funnelshift_l(l0, l1, s) | ((l0 << s) != 0u ? 1u : 0u);
  // round to nearest, ties to even: a carry out of q + (half - 1) + lowest bit
  const unsigned k = 0x7fffffffu + (r0 & 1u);
  const unsigned E = a.e + b.e - s20;  // the significand's leading bit adds the last 1
  asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %2, %3;\n\taddc.cc.u32 %0, %0, 0;\n\t"
      "addc.u32 %1, %1, %4;\n\t}"
      : "+r"(r0), "+r"(r1)
      : "r"(q), "r"(k), "r"(E));
  return __hiloint2double((int)(r1 & a.z & b.z), (int)r0);
}

}  // namespace rfgpu
