// Fixed-point arithmetic on the integer pipes, for the points of a
// composition through map forms.
//
// GB300 runs one warp FP64 instruction in the time of 64 issue slots of a
// scheduler, so a product of two 60-bit fixed-point numbers (three 32 x 32 ->
// 64 bit multiply-adds) costs a small fraction of an FP64 multiply-add, and
// points and forms of a map are O(1) with absolute accuracy all that matters:
// 2^-58 steps carry them more exactly than FP64's 2^-53 roundings.
//
// A number is an int64 in units of 2^-58 or, to be multiplied, two limbs
// h 2^-29 + l 2^-59 with |l| < 2^30.  A product of limbs is h h' (units
// 2^-58) plus h l' + l h' (2^-88); l l' (below 2^-58) is dropped.
#pragma once
#include <cuda_runtime.h>

#include "ff.cuh"

namespace cmm {
namespace dev {

constexpr double kFxUnit = 3.469446951953614e-18;   // 2^-58

struct Limbs {
  int h, l;
};

// X (units of 2^-58), |X| < 4 in value
__device__ __forceinline__ Limbs fx_limbs(long long X) {
  return Limbs{(int)(X >> 29), (int)(((unsigned)X << 1) & 0x3fffffffu)};
}

// The running sums of products: hi in units of 2^-58, lo in 2^-88.  Within
// |lo| < 2^63 for up to 12 cross products of |h| < 2^30 and |l| < 2^30 whose
// h are not all at their bound (|point|^2 < 1.4, |form entry| < 2).
struct FxSum {
  long long hi, lo;
  __device__ __forceinline__ void add(Limbs a, Limbs b) {
    hi += (long long)a.h * b.h;
    lo += (long long)a.h * b.l;
    lo += (long long)a.l * b.h;
  }
  __device__ __forceinline__ long long value() const { return hi + (lo >> 30); }
};

// v / 2^(eb - 1022), at most 1 in magnitude where eb is the largest biased
// exponent met, as limbs (2^-59 steps, toward zero), from the double's bits;
// where v is larger (its exponent above eb) or not finite the sign bit of
// `bad` is set and the limbs are meaningless.
__device__ __forceinline__ Limbs fx_scaled(double v, int eb, int& bad) {
  const int hi = __double2hiint(v);
  const unsigned lo = (unsigned)__double2loint(v);
  const int e = eb + 1 - (int)(((unsigned)hi << 1) >> 21);   // right shift of the 53-bit significand << 7
  bad |= e;
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  unsigned long long T = ((((unsigned long long)mh) << 32) | lo) << 7;
  asm("shr.u64 %0, %1, %2;" : "=l"(T) : "l"(T), "r"(e));   // 0 from a shift of 64 on
  const int sg = (hi >> 31) | 1;
  return Limbs{(int)(T >> 30) * sg, (int)((unsigned)T & 0x3fffffffu) * sg};
}

// A form entry |q| < 2 as limbs.
__device__ __forceinline__ Limbs fx_entry(double q, int& bad) { return fx_scaled(q, 1022, bad); }

// Biased exponent of a double.
__device__ __forceinline__ int fx_exponent(double v) { return (int)(((unsigned)__double2hiint(v) << 1) >> 21); }

// X 2^(eb - 1022 - 58) as a double (truncated toward zero, 59 <= eb < 2000),
// from the bits: the conversion and the scaling would take the FP64 pipe.
__device__ __forceinline__ double fx_to_double(long long X, int eb) {
  unsigned long long M = X < 0 ? (unsigned long long)-X : (unsigned long long)X;
  const int n = __clzll(M);
  if (n == 64) return 0.0;
  M <<= n;   // leading bit at 63: value 2^(63 - n)
  const unsigned hi = ((unsigned)(M >> 43) & 0xfffffu) | ((unsigned)(eb - 1080 + 1023 + 63 - n) << 20);
  return __hiloint2double((int)(hi | (X < 0 ? 0x80000000u : 0u)), (int)(unsigned)(M >> 11));
}

// x, |x| < 16, in units of 2^-58 (toward zero)
__device__ __forceinline__ long long fx_of(double x) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int e = 1028 - (int)(((unsigned)hi << 1) >> 21);   // right shift of the 53-bit significand << 11
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  unsigned long long T = ((((unsigned long long)mh) << 32) | lo) << 11;
  asm("shr.u64 %0, %1, %2;" : "=l"(T) : "l"(T), "r"(e));
  return hi < 0 ? -(long long)T : (long long)T;
}

// X as a float: its high word, rounded (within 2^-25 of |x| <= 1)
__device__ __forceinline__ float fx_f32(long long X) { return __fmul_rn((float)(int)(X >> 32), 1.4901161193847656e-08f); }

}  // namespace dev
}  // namespace cmm
