// cgb_pair.cuh — FP32-pair ("double-float") arithmetic for the mixed-precision shape stage.
//
// A value is the unevaluated sum hi + lo of two floats with |lo| <= ulp(hi) / 2, about
// 48 significant bits. Everything here runs on the FP32 pipe, which on GB300 issues 62x
// the FP64 rate, so per-neighbour work in pairs costs a fraction of the same work in FP64.
//
// Published methods, restated:
//  - TwoSum (Knuth, TAOCP vol. 2, sec. 4.2.2; Moller 1965): s = fl(a + b) and the exact
//    rounding error e, a + b = s + e, in six additions, any magnitudes.
//  - FastTwoSum (Dekker 1971): the same in three additions when |a| >= |b|.
//  - TwoProd with a fused multiply-add: p = fl(a b), e = fma(a, b, -p) is exact.
//  - Pair addition and multiplication as in Dekker (1971), "A floating-point technique for
//    extending the available precision", and the double-double library of Hida, Li and
//    Bailey (2001), with float in place of double ("sloppy" addition where operands do not
//    cancel, the two-TwoSum addition where they may).
//  - Reciprocal and square root by one Newton step on the pair (Karp and Markstein 1997,
//    "High-precision division and square root"), seeded by the single-precision result.
//  - Dot products accumulated as in Ogita, Rump and Oishi (2005), "Accurate sum and dot
//    product" (Dot2): the high parts by TwoSum, all rounding errors in a second float.
// All operations use explicitly rounded intrinsics, so the compiler neither contracts nor
// reorders the error-free transforms.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace cgb {

struct fp2 {
  float hi, lo;
};

__device__ __forceinline__ fp2 fp2_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}

__device__ __forceinline__ fp2 fp2_fast_two_sum(float a, float b) {  // |a| >= |b| (or a == 0)
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ fp2 fp2_two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

// Conversions between doubles and floats. Like an addition of doubles, the instructions for them
// issue on the FP64 pipe, at 1/62 of the FP32 rate, so they are done on the bits; only exponents near
// the ends of the float range, infinities and NaN in a pair take the instructions, in volatile asm so
// that they are not executed beside the common path and selected. (Under a predicate they would still
// take their turn on the pipe: fp2_to_double therefore converts several pairs at a time, behind one
// branch.)
__device__ __forceinline__ double fp2_widen(float f) {
  const uint32_t sign = __float_as_uint(f) & 0x80000000u;
  uint32_t m = __float_as_uint(f) & 0x7fffffffu, bias = 0x38000000u;   // exponent from 127 to 1023
  if (m >= 0x7f800000u) bias = 0x70000000u;                            // infinity, NaN: from 255 to 2047
  if (m < 0x00800000u) {                                               // zero; denormals times 2^64
    m = __float_as_uint(__fmul_rn(__uint_as_float(m), 0x1p64f));
    bias = m == 0u ? 0u : 0x34000000u;
  }
  return __hiloint2double(static_cast<int>(((m >> 3) + bias) | sign), static_cast<int>(m << 29));
}

// hi = the double rounded to 24 bits, lo = the other 29 bits rounded to 24.
__device__ __forceinline__ fp2 fp2_from_double(double d) {
  const uint32_t h = static_cast<uint32_t>(__double2hiint(d)), l = static_cast<uint32_t>(__double2loint(d));
  const uint32_t e = (h >> 20) & 0x7ffu, sign = h & 0x80000000u;
  const uint32_t low = l & 0x1fffffffu, up = low >> 28;
  const uint32_t hi = __funnelshift_l(l, h & 0x7fffffffu, 3) - 0xc0000000u + up;   // exponent - 896
  const float lo = __int2float_rn(static_cast<int>(low) - static_cast<int>(up << 29)) * __uint_as_float((e - 948u) << 23);
  fp2 r = {__uint_as_float(hi | sign), __uint_as_float(__float_as_uint(lo) ^ sign)};
  if (((h << 1) | l) == 0u) {
    r = {__uint_as_float(sign), 0.0f};
  } else if (e < 949u || e > 1149u) {   // lo would be denormal, or hi may round to infinity
    asm volatile("{\n\t.reg .f64 a;\n\tcvt.rn.f32.f64 %0, %2;\n\tcvt.f64.f32 a, %0;\n\tsub.rn.f64 a, %2, a;\n\t"
                 "cvt.rn.f32.f64 %1, a;\n\t}" : "=&f"(r.hi), "=f"(r.lo) : "d"(d));
  }
  return r;
}

// hi + lo rounded to double, normalised or not. Normalised, lo in units of the last place of hi as a
// double is rounded to an integer and added to its bits; below a power of two those units are half
// as large.
template <int N>
__device__ __forceinline__ void fp2_to_double(const fp2 (&b)[N], double (&d)[N]) {
  bool rest = false;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const fp2 a = fp2_two_sum(b[k].hi, b[k].lo);
    const uint32_t u = __float_as_uint(a.hi), sign = u & 0x80000000u, m = u & 0x7fffffffu, e = m >> 23;
    float t = __fmul_rn(a.lo, __uint_as_float((306u - e) << 23));   // lo 2^(52 - exponent)
    t = __uint_as_float(__float_as_uint(t) ^ sign);
    if ((u & 0x7fffffu) == 0u && t < 0.0f) t = __fadd_rn(t, t);
    const bool zero = (m | (__float_as_uint(a.lo) << 1)) == 0u;
    const long long bits = __double_as_longlong(__hiloint2double(static_cast<int>((m >> 3) + 0x38000000u), static_cast<int>(m << 29)))
                           + __float2int_rn(t);
    d[k] = __longlong_as_double(bits | static_cast<long long>(static_cast<unsigned long long>(sign) << 32));
    if (zero) d[k] = __hiloint2double(static_cast<int>(__float_as_uint(b[k].hi) & __float_as_uint(b[k].lo) & 0x80000000u), 0);
    rest = rest || (!zero && (e < 52u || e == 255u || !(fabsf(t) <= 268435456.0f)));   // 2^28: half a unit of hi
  }
  if (rest) {
#pragma unroll
    for (int k = 0; k < N; ++k)
      asm volatile("{\n\t.reg .f64 a, b;\n\tcvt.f64.f32 a, %1;\n\tcvt.f64.f32 b, %2;\n\tadd.rn.f64 %0, a, b;\n\t}"
                   : "=d"(d[k]) : "f"(b[k].hi), "f"(b[k].lo));
  }
}

__device__ __forceinline__ double fp2_to_double(fp2 a) {
  const fp2 b[1] = {a};
  double d[1];
  fp2_to_double(b, d);
  return d[0];
}

__device__ __forceinline__ fp2 operator-(fp2 a) { return {-a.hi, -a.lo}; }

// a + b, for operands that do not nearly cancel.
__device__ __forceinline__ fp2 operator+(fp2 a, fp2 b) {
  const fp2 s = fp2_two_sum(a.hi, b.hi);
  return fp2_fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ fp2 operator-(fp2 a, fp2 b) { return a + (-b); }

// a + b with full relative accuracy also under cancellation.
__device__ __forceinline__ fp2 fp2_add_exact(fp2 a, fp2 b) {
  fp2 s = fp2_two_sum(a.hi, b.hi);
  const fp2 t = fp2_two_sum(a.lo, b.lo);
  s = fp2_fast_two_sum(s.hi, __fadd_rn(s.lo, t.hi));
  return fp2_fast_two_sum(s.hi, __fadd_rn(s.lo, t.lo));
}

__device__ __forceinline__ fp2 operator*(fp2 a, fp2 b) {
  const fp2 p = fp2_two_prod(a.hi, b.hi);
  return fp2_fast_two_sum(p.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo)));
}
// By a float that is exact (small integers, powers of two, sides +-1).
__device__ __forceinline__ fp2 operator*(fp2 a, float b) {
  const fp2 p = fp2_two_prod(a.hi, b);
  return fp2_fast_two_sum(p.hi, __fmaf_rn(a.lo, b, p.lo));
}
__device__ __forceinline__ fp2 operator*(float b, fp2 a) { return a * b; }
__device__ __forceinline__ fp2 operator+(fp2 a, float b) {
  const fp2 s = fp2_two_sum(a.hi, b);
  return fp2_fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}
__device__ __forceinline__ fp2 operator+(float b, fp2 a) { return a + b; }
__device__ __forceinline__ fp2 operator-(float b, fp2 a) { return (-a) + b; }
__device__ __forceinline__ fp2 operator-(fp2 a, float b) { return a + (-b); }

__device__ __forceinline__ fp2 fp2_sqr(fp2 a) {
  const fp2 p = fp2_two_prod(a.hi, a.hi);
  return fp2_fast_two_sum(p.hi, __fmaf_rn(2.0f * a.hi, a.lo, p.lo));
}

// 1 / b: x = 1 / b.hi, then x + x (1 - b x) with the residual formed in pairs.
__device__ __forceinline__ fp2 fp2_recip(fp2 b) {
  const float x = __frcp_rn(b.hi);
  // r = 1 - b x, exactly enough: 1 - b.hi x is exact by one FMA, then the b.lo term.
  const float r = __fmaf_rn(-b.lo, x, __fmaf_rn(-b.hi, x, 1.0f));
  return fp2_fast_two_sum(x, __fmul_rn(x, r));
}

// sqrt(a) for a >= 0: y = sqrt(a.hi), then y + (a - y^2) / (2 y).
__device__ __forceinline__ fp2 fp2_sqrt(fp2 a) {
  if (a.hi <= 0.0f) return {0.0f, 0.0f};
  const float y = __fsqrt_rn(a.hi);
  const fp2 y2 = fp2_two_prod(y, y);
  const float r = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, y2.hi), y2.lo), a.lo);
  return fp2_fast_two_sum(y, __fmul_rn(r, __fdividef(0.5f, y)));
}

// Dot-product accumulator (Dot2): acc.hi carries the running sum by TwoSum, acc.lo the
// sum of every rounding error; normalise with fp2_norm once the sum is complete.
__device__ __forceinline__ void fp2_fma_acc(fp2& acc, fp2 a, fp2 b) {
  const fp2 p = fp2_two_prod(a.hi, b.hi);
  const float cross = __fmaf_rn(a.hi, b.lo, __fmul_rn(a.lo, b.hi));
  const fp2 s = fp2_two_sum(acc.hi, p.hi);
  acc.hi = s.hi;
  acc.lo = __fadd_rn(acc.lo, __fadd_rn(s.lo, __fadd_rn(p.lo, cross)));
}

__device__ __forceinline__ fp2 fp2_norm(fp2 a) { return fp2_two_sum(a.hi, a.lo); }

// Comparisons with float constants (exact in float: 0, 0.5, 1).
__device__ __forceinline__ bool fp2_ge(fp2 a, float c) { return a.hi > c || (a.hi == c && a.lo >= 0.0f); }
__device__ __forceinline__ bool fp2_le(fp2 a, float c) { return a.hi < c || (a.hi == c && a.lo <= 0.0f); }
__device__ __forceinline__ bool fp2_is_zero(fp2 a) { return a.hi == 0.0f && a.lo == 0.0f; }

}  // namespace cgb
