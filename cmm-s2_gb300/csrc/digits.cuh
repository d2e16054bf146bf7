// 9-bit digits of 53-bit integers in bf16, and 64-bit sums back to FP64
// (sht_digits.cu describes the scheme).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cmm {
namespace dig {

constexpr int kDigits = 6;
constexpr int kLevels = 7;

__host__ __device__ __forceinline__ int groups16(int n) { return (n + 15) / 16; }

// x 2^(1075 - e) rounded to nearest, e the biased exponent of the scale's
// binade (>= 1; that of x or more): |result| < 2^53.  x = 1 may have e = 1022:
// 2^53, whose digits are (256, 0, ...).
__device__ __forceinline__ long long to_fixed(double x, int e) {
  const long long b = __double_as_longlong(x);
  int ex = (int)((b >> 52) & 2047);
  long long v = b & 0xfffffffffffffLL;
  if (ex)
    v |= 0x10000000000000LL;
  else
    ex = 1;
  const int sh = e - ex;
  if (sh > 54) return 0;
  if (sh > 0) v = (v + (1LL << (sh - 1))) >> sh;
  if (sh < 0) v <<= 1;
  return b < 0 ? -v : v;
}

// The six digits of eight entries as bf16 vectors, highest first.  With 256
// added to the lower five, a digit is a field of 9 bits; its float comes from
// the bits of 2^23 + field, and is exact in bf16 (8 significant bits).
__device__ __forceinline__ void digits8(const long long* v, uint4* out) {
  uint32_t w[kDigits][4];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long r = v[q] + 256LL * (1 + (1LL << 9) + (1LL << 18) + (1LL << 27) + (1LL << 36));
#pragma unroll
    for (int i = 0; i < kDigits; ++i) {
      float f;
      if (i == 0) {   // -256 .. 256
        f = __uint_as_float(0x4B000000u | ((uint32_t)(r >> 45) + 256u)) - 8388864.f;
      } else {
        const uint32_t x = (uint32_t)((unsigned long long)r >> (9 * (kDigits - 1 - i))) & 511u;
        f = __uint_as_float(0x4B000000u | x) - 8388864.f;
      }
      const uint32_t u = __float_as_uint(f);
      if (q & 1)
        w[i][q >> 1] = __byte_perm(w[i][q >> 1], u, 0x7632);   // high halves of both
      else
        w[i][q >> 1] = u;
    }
  }
#pragma unroll
  for (int i = 0; i < kDigits; ++i) out[i] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// a b + c
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// v 2^p to nearest without the FP64 pipe.
static __device__ __noinline__ double fixed_wide(long long v, int p) { return ldexp((double)v, p); }
__device__ __forceinline__ double fixed_to_double(long long v, int p) {
  if (v == 0) return 0.0;
  const unsigned long long mag = v < 0 ? -(unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)mag), e = 63 - lz + p + 1023;
  if ((unsigned)(e - 1) >= 2045u) return fixed_wide(v, p);
  unsigned long long n = mag << lz;                       // top bit set
  const unsigned rem = (unsigned)n & 0x7ffu;
  n >>= 11;                                               // 53 bits; a carry below raises the exponent
  n += rem > 0x400u || (rem == 0x400u && (n & 1));
  n += (unsigned long long)(e - 1) << 52;
  return __longlong_as_double((long long)(n | (v < 0 ? 0x8000000000000000ULL : 0ULL)));
}

}  // namespace dig
}  // namespace cmm
