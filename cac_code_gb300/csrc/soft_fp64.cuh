// FP64 sums of products by the integer units.
//
// The FP64 unit of sm_103a takes a warp instruction every 16 cycles of an SM, the
// integer pipes four a cycle: a product and a sum rounded as the FP64 unit rounds them
// (IEEE, to nearest even) cost 64 issue slots each there and about 35 each here.  The
// passes that the FP64 unit bounds give it the part of a pair that is left and form the
// interpolated positions and densities with dot8, at the same time.  Results are the
// FP64 unit's bit for bit (but for the sign of a zero) as long as every operand is zero
// or has an exponent of at most DOT_RANGE either way, so that nothing over- or
// underflows: dot_ready tells.
//
// Also compiled for the host, by the test that compares it with the host's FP64.
#pragma once
#include <stdint.h>
#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace cacg {
namespace soft {

constexpr int DOT_RANGE = 200;

// (-1)^sign m 2^(e - 1075), m = hi:lo below 2^53 (0 or normal); sign: 0 or ~0
struct Op {
  uint32_t lo, hi;
  int e, sign;
};

__host__ __device__ __forceinline__ Op op_of(uint32_t hi, uint32_t lo) {
  Op o;
  o.e = (int) (hi >> 20) & 0x7FF;
  o.hi = o.e ? (hi & 0xFFFFFu) | 0x100000u : 0u;
  o.lo = o.e ? lo : 0u;
  o.sign = (int) hi >> 31;
  return o;
}

// zero, or an exponent within DOT_RANGE
__host__ __device__ __forceinline__ bool dot_ready(uint32_t hi, uint32_t lo) {
  const int e = (int) (hi >> 20) & 0x7FF;
  return ((hi << 1) | lo) == 0u || (e >= 1023 - DOT_RANGE && e <= 1023 + DOT_RANGE);
}

__host__ __device__ __forceinline__ int clz64(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long) x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

// a signed 64-bit mantissa with at least 7 zero bits below the 53: |m| in
// [2^59, 2^61] or 0; the value is m 2^(e - 1083)
struct Acc {
  int64_t m;
  int e;
};

// RN(a b).  The product of the mantissas, 104 to 106 bits in 32-bit limbs, less its 50
// low bits (whether any is set: the lowest bit kept), is 2 or 3 bits too long.
__host__ __device__ __forceinline__ Acc mul(const Op &a, const Op &b) {
  const uint64_t p0 = (uint64_t) a.lo * b.lo;
  uint64_t mid = (uint64_t) a.lo * b.hi + (p0 >> 32);
  mid += (uint64_t) a.hi * b.lo;
  const uint64_t top = (uint64_t) a.hi * b.hi + (mid >> 32);
  const uint32_t ml = (uint32_t) mid;
  const uint32_t lost = (ml & 0x3FFFFu) | (uint32_t) p0;
  uint64_t w = (top << 14) | (ml >> 18);
  w |= lost < 1u ? lost : 1u;
  // rounded at bit 3 or 2 (to even: by half less one, plus the last bit kept)
  const bool c = (uint32_t) (w >> 32) >> 23 != 0u;
  const uint32_t odd = c ? (uint32_t) w >> 3 : (uint32_t) w >> 2;
  w += (odd & 1u) + (c ? 3u : 1u);
  w &= c ? ~(uint64_t) 7 : ~(uint64_t) 3;
  const int64_t m = (int64_t) (w << 5);
  const int64_t sign = a.sign ^ b.sign;
  Acc r;
  r.m = (m ^ sign) - sign;
  r.e = a.e + b.e - 1022;
  return r;
}

// RN(a + b).  The smaller in exponent is shifted to the other's with what is lost
// jammed into its lowest bit; rounding a two's complement number to the nearest even
// multiple is the same for both signs.
__host__ __device__ __forceinline__ Acc add(const Acc &a, const Acc &b) {
  int d = a.e - b.e;
  const bool less = d < 0;
  const int64_t big = less ? b.m : a.m, small = less ? a.m : b.m;
  const int e = less ? b.e : a.e;
  d = less ? -d : d;
  d = d < 63 ? d : 63;
  int64_t s = small >> d;
  s |= (int64_t) ((uint64_t) s << d) != small ? 1 : 0;
  const int64_t r = big + s;
  int n = clz64((uint64_t) (r ^ (r >> 63))) - 2;
  n = n > 0 ? n : 0;
  int64_t t = (int64_t) ((uint64_t) r << n);
  t += 255 + (int) (((uint32_t) t >> 9) & 1u);
  t &= ~(int64_t) 511;
  Acc q;
  q.m = t >> 1;
  q.e = n == 62 ? 0 : e - n + 1;  // (62: a zero, below every product)
  return q;
}

// a sum as a factor, an operand as a term
__host__ __device__ __forceinline__ Op op_of(const Acc &a) {
  const int64_t s = a.m >> 63;
  const uint64_t m = (uint64_t) ((a.m ^ s) - s) >> 8;  // at most 2^53
  return Op{(uint32_t) m, (uint32_t) (m >> 32), a.e, (int) s};
}
__host__ __device__ __forceinline__ Acc acc_of(const Op &o) {
  const int64_t m = (int64_t) (((uint64_t) o.hi << 32 | o.lo) << 8), s = o.sign;
  return Acc{(m ^ s) - s, o.e};
}

// the IEEE bits of a sum (of two terms or more)
__host__ __device__ __forceinline__ uint64_t bits(const Acc &a) {
  const int64_t s = a.m >> 63;
  const uint64_t m = (uint64_t) ((a.m ^ s) - s) >> 8;  // 2^52 to 2^53
  const uint64_t r = ((uint64_t) (uint32_t) (a.e - 1) << 52) + m;
  return m ? r | ((uint64_t) s << 63) : 0u;
}

}  // namespace soft
}  // namespace cacg
