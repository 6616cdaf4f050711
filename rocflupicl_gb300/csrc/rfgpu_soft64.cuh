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

// A double for arithmetic written over a number type, whose products are
// FP64 operations as usual unless asked for as prod(), an integer product, or
// scale<K>(), a product with 2^K done on the exponent.  An operand outside
// their range makes the result NaN instead of taking a branch; NaN reaches
// every result that depends on it, and the caller repeats such a rare
// evaluation on plain doubles.  Comparisons do not hide it: minimum, maximum
// and positive part keep NaN, and `unknown` tells that a branch condition is
// NaN (for plain numbers it is false at compile time, their NaNs being
// results).
struct Sd {
  double v;
  __device__ __forceinline__ Sd() {}
  __device__ __forceinline__ constexpr explicit Sd(double x) : v(x) {}
  friend __device__ __forceinline__ Sd sqrt(Sd a) { return Sd(::sqrt(a.v)); }
  friend __device__ __forceinline__ Sd fabs(Sd a) { return Sd(::fabs(a.v)); }
};
__device__ __forceinline__ Sd operator+(Sd a, Sd b) { return Sd(a.v + b.v); }
__device__ __forceinline__ Sd operator-(Sd a, Sd b) { return Sd(a.v - b.v); }
__device__ __forceinline__ Sd operator-(Sd a) { return Sd(-a.v); }
__device__ __forceinline__ Sd operator/(Sd a, Sd b) { return Sd(a.v / b.v); }
__device__ __forceinline__ Sd operator*(Sd a, Sd b) { return Sd(a.v * b.v); }
template <typename R> __device__ __forceinline__ R prod(R a, R b) { return a * b; }
template <> __device__ __forceinline__ Sd prod(Sd a, Sd b) {
  const double r = soft_mul(soft_a(a.v), soft_b(b.v));
  const unsigned bad = (soft_ok(a.v) ? 0u : 0x7ff80000u) | (soft_ok(b.v) ? 0u : 0x7ff80000u);
  return Sd(__hiloint2double((int)((unsigned)__double2hiint(r) | bad), __double2loint(r)));
}
constexpr double pow2(int k) { return k == 0 ? 1.0 : k > 0 ? 2.0 * pow2(k - 1) : 0.5 * pow2(k + 1); }
template <int K, typename R> __device__ __forceinline__ R scale(R x) { return R(pow2(K)) * x; }
template <int K> __device__ __forceinline__ Sd scale(Sd x) {
  const unsigned h = (unsigned)__double2hiint(x.v), l = (unsigned)__double2loint(x.v);
  const bool ok = (h & 0x7fffffffu) - 0x01000000u < 0x7e000000u;  // exponents 16 .. 2031
  const unsigned r = ok ? h + (unsigned)(K * (1 << 20)) : soft_zero(x.v) ? h : 0x7ff80000u;
  return Sd(__hiloint2double((int)r, (int)l));
}
__device__ __forceinline__ bool operator<(Sd a, Sd b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>(Sd a, Sd b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<=(Sd a, Sd b) { return a.v <= b.v; }
__device__ __forceinline__ bool nan_bits(double x) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  return h > 0x7ff00000u || (h == 0x7ff00000u && __double2loint(x) != 0);
}
__device__ __forceinline__ bool unknown(Sd a) { return nan_bits(a.v); }

}  // namespace rfgpu
