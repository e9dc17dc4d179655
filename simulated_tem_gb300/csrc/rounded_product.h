// The product of two FP64 numbers, rounded to nearest (ties to even), in integer arithmetic: for sums
// of products whose products have to be rounded by themselves, where the FP64 unit is the bottleneck.
// The factors are taken apart once per tile (pixel_factor, weight_factor); the product is four
// 32 x 32 -> 64-bit multiply-adds, one conditional shift and the rounding.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define RP_HD __host__ __device__ __forceinline__
#else
#define RP_HD inline
#endif

namespace stem {

struct RoundedFactor {
  uint32_t lo, hi;  // significand: 53 bits with the leading one, for a weight shifted left by 11 bits
  uint32_t e;       // sign at bit 31 and biased exponent at bit 20, for a weight less 1024
};

// ok: a normal number between 2^-700 and 2^700 in magnitude, or zero (significand 0, whose product is
// meaningless and to be left out).
RP_HD RoundedFactor pixel_factor(uint64_t bits, bool& ok) {
  const uint32_t e = (uint32_t)(bits >> 52) & 0x7FF;
  const bool zero = (bits << 1) == 0;
  ok = zero || (e >= 1023 - 700 && e <= 1023 + 700);
  RoundedFactor r;
  r.lo = (uint32_t)bits;
  r.hi = zero ? 0 : ((uint32_t)(bits >> 32) & 0xFFFFF) | 0x100000;
  r.e = (uint32_t)(bits >> 32) & 0xFFF00000;
  return r;
}

// ok: a positive normal number between 2^-200 and 2^200.
RP_HD RoundedFactor weight_factor(uint64_t bits, bool& ok) {
  const uint32_t e = (uint32_t)(bits >> 52);
  ok = e >= 1023 - 200 && e <= 1023 + 200;
  const uint64_t m = ((bits & ((1ULL << 52) - 1)) | (1ULL << 52)) << 11;
  RoundedFactor r;
  r.lo = (uint32_t)m;
  r.hi = (uint32_t)(m >> 32);
  r.e = (e - 1024) << 20;
  return r;
}

// The bits of f k rounded.  With both factors in their ranges the result is a normal number.
RP_HD uint64_t rounded_product(const RoundedFactor& f, const RoundedFactor& k) {
  // hi:lo = f k 2^-64 as 53 bits and 64 bits of fraction; hi in [2^51, 2^53)
  const uint64_t t0 = (uint64_t)f.lo * k.lo;
  const uint64_t t1 = (uint64_t)f.hi * k.lo + (uint32_t)(t0 >> 32);
  const uint64_t t2 = (uint64_t)f.lo * k.hi + (uint32_t)t1;
  const uint64_t hi = (uint64_t)f.hi * k.hi + (uint32_t)(t1 >> 32) + (uint32_t)(t2 >> 32);
  uint32_t h1 = (uint32_t)(hi >> 32), h0 = (uint32_t)hi, l1 = (uint32_t)t2;
  l1 |= (uint32_t)t0 != 0 ? 1u : 0u;  // what lies below only says whether there is anything
  const uint32_t exponent = f.e + k.e + (h1 & 0x100000);
  if (!(h1 & 0x100000)) {  // below 2^52: one bit more
    h1 = (h1 << 1) | (h0 >> 31);
    h0 = (h0 << 1) | (l1 >> 31);
    l1 <<= 1;
  }
  // half an ulp and more (or exactly half and odd) rounds up; a carry out of the significand belongs to
  // the exponent
  const uint32_t up = l1 > 0x80000000u - (h0 & 1) ? 1u : 0u;
  return (((uint64_t)(h1 + exponent) << 32) | h0) + up;
}

}  // namespace stem
