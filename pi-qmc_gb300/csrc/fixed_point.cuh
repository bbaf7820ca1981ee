// Correctly rounded FP64 operations on the integer pipe.
//
// An FP64 instruction costs an SM 19 clocks per warp whatever its active lanes, a
// conversion to or from an integer 16, and the sequences of a reciprocal 86, a square
// root 143 and a division 156; the integer pipe is some sixty times cheaper.  Newton's
// iterations in fixed point, from the FP32 approximations (22 bits, then 44, then 61),
// leave a result to 2 units of 2^-62; a double takes 10 fewer bits, so its rounding is
// certain unless the cut bits lie within 8 units of a tie.  Those 1.6% of values, and
// operands or results that are not normal, take the instruction sequence: the same
// bits always.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pimc {

// 2^62 / d for d = M / 2^64 in [1/2, 1); f24: the 23 bits of d's double below the leading one
__device__ __forceinline__ unsigned long long fixed_reciprocal(unsigned long long M,
                                                               unsigned f24) {
  const unsigned rb = __float_as_uint(__fdividef(1.0f, __uint_as_float(0x3f000000u | f24)));
  const unsigned x0 = ((rb & 0x7fffffu) | 0x800000u) << ((rb >> 23) - 120u);  // 2^30 / d
  const unsigned long long t =
      (unsigned long long)(unsigned)(M >> 32) * x0 + (((unsigned long long)(unsigned)M * x0) >> 32);
  const int e0 = (int)((long long)((1ull << 62) - t) >> 10);
  const unsigned long long x1 = ((unsigned long long)x0 << 32) +
                                (unsigned long long)(((long long)(int)(x0 >> 1) * e0) >> 19);
  const int e1 = (int)((1ull << 62) - __umul64hi(M, x1));
  return x1 + (unsigned long long)(((long long)(int)(unsigned)(x1 >> 33) * e1) >> 29);
}

// 1 / a
static __device__ __noinline__ double reciprocal_call(double a) { return __drcp_rn(a); }
__device__ __forceinline__ double reciprocal(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b, e = (hi >> 20) & 0x7ffu;
  const unsigned long long x =
      fixed_reciprocal((1ull << 63) | (b << 11), ((hi & 0xfffffu) << 3) | (lo >> 29)) + 512ull;
  // (a power of two would carry past the format)
  if ((((hi & 0xfffffu) | lo) == 0u) || e - 2u > 2042u || ((unsigned)x & 1023u) - 8u > 1008u)
    return reciprocal_call(a);
  return __longlong_as_double(
      (long long)((((unsigned long long)(2045u - e) << 52) + (x >> 10) - (1ull << 52)) |
                  (b & (1ull << 63))));
}

// a / b
static __device__ __noinline__ double divide_call(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double divide(double a, double b) {
  const unsigned long long A = (unsigned long long)__double_as_longlong(a);
  const unsigned long long B = (unsigned long long)__double_as_longlong(b);
  const unsigned ea = (unsigned)(A >> 52) & 0x7ffu, eb = (unsigned)(B >> 52) & 0x7ffu;
  unsigned long long q =
      __umul64hi((1ull << 63) | (A << 11),
                 fixed_reciprocal((1ull << 63) | (B << 11), (unsigned)(B >> 29) & 0x7fffffu));
  int e = (int)ea - (int)eb + 1023;
  if (!(q >> 62)) {
    q <<= 1;
    e -= 1;
  }
  q += 512ull;
  if (ea - 1u > 2045u || eb - 1u > 2045u || (unsigned)(e - 1) > 2044u ||
      ((unsigned)q & 1023u) - 8u > 1008u)
    return divide_call(a, b);
  return __longlong_as_double((long long)((((unsigned long long)e << 52) + (q >> 10) - (1ull << 52)) |
                                          ((A ^ B) & (1ull << 63))));
}

// sqrt(a): a = 4^k d with d in [1, 4), s = d y with the FP32 reciprocal root y, then
// s += (d - s^2) y / 2 twice
static __device__ __noinline__ double square_root_call(double a) { return sqrt(a); }
__device__ __forceinline__ double square_root(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const bool even = (hi >> 20) & 1u;  // (of the exponent; the bias is odd)
  const unsigned long long d = ((b & 0xfffffffffffffull) | (1ull << 52)) << (even ? 10 : 11);
  const unsigned yb = __float_as_uint(rsqrtf(__uint_as_float(
      (even ? 0x3f800000u : 0x40000000u) | ((hi & 0xfffffu) << 3) | (lo >> 29))));
  const unsigned y = ((yb & 0x7fffffu) | 0x800000u) << ((yb >> 23) - 119u);  // 2^31 / sqrt(d)
  const int y2 = (int)(y >> 1);
  const unsigned long long s6 = ((unsigned long long)(unsigned)(d >> 32) * y) >> 30;
  const unsigned s0 = s6 > 0xffffffffull ? 0xffffffffu : (unsigned)s6;
  const long long e0 = (long long)(d - (unsigned long long)s0 * s0);
  const unsigned long long s1 = ((unsigned long long)s0 << 31) +
                                (unsigned long long)(((long long)(int)(e0 >> 14) * y2) >> 17);
  const unsigned long long plo = s1 * s1, dlo = d << 62;
  const unsigned long long ehi = (d >> 2) - __umul64hi(s1, s1) - (dlo < plo);
  const int e1 = (int)((ehi << 10) | ((dlo - plo) >> 54));
  const unsigned long long s2 = s1 + (unsigned long long)(((long long)e1 * y2) >> 39) + 512ull;
  // (zero, subnormal, infinite, NaN and negative values)
  if (hi - 0x00100000u >= 0x7fe00000u || ((unsigned)s2 & 1023u) - 8u > 1008u)
    return square_root_call(a);
  return __longlong_as_double((long long)(((unsigned long long)((hi + (1023u << 20)) >> 21) << 52) +
                                          (s2 >> 10) - (1ull << 52)));
}

// 2^k, -1023 < k < 1024 (a conversion takes 16 clocks of the FP64 pipe)
__device__ __forceinline__ double pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }

// An integer of at most 53 bits times 2^k, exactly (results normal or 0)
__device__ __forceinline__ double scaled_integer(unsigned long long m, int k, bool negative = false) {
  const int z = __clzll((long long)m);
  const unsigned long long v = ((unsigned long long)(1023 + 63 - z + k) << 52) | ((m << z << 1) >> 12);
  return m ? __longlong_as_double((long long)(v | ((unsigned long long)negative << 63))) : 0.0;
}

}  // namespace pimc
