// FP64 velocity synthesis on the tensor cores (tcgen05, sm_103a) by exact
// integer digits.
//
// The Legendre synthesis of one order m is a product
//   S_even/odd[t][n] = sum_{l - m even/odd} Pbar_lm(theta_t) A[l][n]
// over ring pairs t and 12 real columns n (six complex fields).  GB300 has 2
// FP64 multiply-adds per SM and cycle, so FP64 arithmetic takes 12 L^3 / 4 of
// them (1.03 ms at L = 512) where the table's bytes need 60 us.  Instead every
// row of Pbar (over l) and every column of A gets the power of two above its
// largest entry as its scale, and each entry becomes the integer x 2^53 / scale,
// rounded (entries of the largest one's binade exactly, the others to half an
// ulp of it: the size of one FP64 rounding of the sum), cut into six signed
// digits of 9 bits: integers of at most 256, exact in bf16.  Products of digits
// i and j belong to level i + j; the levels' sums over 64 degrees are integers
// accumulated exactly in FP32 in tensor memory (levels 0 to 3 stay within 4 x
// 64 x 2^16 = 2^24; the lower levels' bound is larger only for digits that are
// all extreme, and they then round at 2^-52 of the scales' product), and are
// added up as 64-bit integers.  Levels 7 and up (2^-61 of the scales' product)
// are left out.  The scheme is known as Ozaki splitting.  Measured: 1032 -> 98 us
// at L = 512, 167 -> 31 at L = 256, 59 -> 13 at L = 128, results to the same
// error against 64 bits.
//
// Layouts: both operands as K-major core-matrix images without swizzle in
// groups of 16 degrees of one parity.  The table (12 bytes per entry) of (m,
// row block): [even groups, odd groups][6 digits][2 halves of 8 degrees][8-row
// groups][8 rows][8 degrees]; the data of m: [groups][2 halves][14 8-column
// groups][8][8], column 16 j + n for digit j, so that digit i of the table times
// the first columns is one MMA that lands at column 16 i: level i + j.  Column
// block 6 is zero: it clears level 6.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "cmm_internal.h"
#include "device_common.cuh"
#include "digits.cuh"
#include "sht_fields.cuh"
#include "tc.cuh"

namespace cmm {

using namespace dig;
using namespace sht;
using namespace tc;

namespace {

constexpr int kRows = 128;              // ring pairs per work item (MMA M)
constexpr int kCols = 12;               // real columns (16 with padding)
constexpr int kChunkGroups = 4;         // groups of 16 degrees per chunk
constexpr int kRowGroupBytes = kDigits * 2 * 128;          // one 8-row group of one degree group
constexpr int kAGroup = 2 * 14 * 128;                      // one degree group of the data
constexpr int kPStage = kChunkGroups * kRowGroupBytes * (kRows / 8);
constexpr int kStage = kPStage + kChunkGroups * kAGroup;   // 110 KiB
constexpr int kStages = 2;
constexpr int kAccCols = 16 * kLevels;  // 112 of 128 TMEM columns per accumulator
constexpr uint32_t kTmemCols = 256;
constexpr int kNonFinite = 1 << 20;     // column scale of a column with an infinity or NaN

struct DigGeometry {
  int L, rows, nblk;      // ring pairs t = 1 .. rows, in nblk blocks
  const int* gbase;       // (L+1) prefix sums of the degree groups per m
};

// ----------------------------------------------------------- tables, data
// Block (row block, m): the digit table of its rows from the FP64 table
// tab[m][l - m][t], one thread per row; scales in pexp[m][t - 1].
__global__ void __launch_bounds__(kRows) build_digits_kernel(DigGeometry g, const double* __restrict__ tab,
                                                             unsigned char* __restrict__ out,
                                                             int* __restrict__ pexp) {
  const int blk = blockIdx.x, m = blockIdx.y, row = threadIdx.x, L = g.L;
  const int npair = L / 2 + 1, t = 1 + blk * kRows + row, n = L - m;
  const int rg = min(kRows / 8, (g.rows - blk * kRows + 7) / 8), rgt = (g.rows + 7) / 8;
  if (row >= 8 * rg) return;
  const bool real = t <= g.rows;
  const double* P = tab + tab_off(m, L, npair) + t;
  int e = 1;
  if (real)
    for (int k = 0; k < n; ++k) e = max(e, (__double2hiint(P[(int64_t)k * npair]) >> 20) & 2047);
  const int ke = groups16((n + 1) / 2), ko = groups16(n / 2);
  unsigned char* base = out + (int64_t)g.gbase[m] * kRowGroupBytes * rgt +
                        (int64_t)(ke + ko) * kRowGroupBytes * (kRows / 8) * blk + (row >> 3) * 128 + (row & 7) * 16;
  const int gb = kRowGroupBytes * rg;   // bytes of one degree group of this block
  for (int q = 0; q < 2 * (ke + ko); ++q) {
    const int grp = q >> 1, half = q & 1, par = grp >= ke;
    const int k0 = 16 * (par ? grp - ke : grp) + 8 * half;
    long long v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = par + 2 * (k0 + u);
      v[u] = real && k < n ? to_fixed(P[(int64_t)k * npair], e) : 0;
    }
    uint4 d[kDigits];
    digits8(v, d);
    unsigned char* o = base + (int64_t)grp * gb + half * rg * 128;
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4*)(o + i * 2 * rg * 128) = d[i];
  }
  if (real) pexp[(int64_t)m * g.rows + t - 1] = e;
}

// c[k][l] = sqrt(max(l(l+1) - k(k-1), 0)) / 2, k = 0 .. L+1, and in row L+2
// -1 / (l(l+1)) (0 at l = 0).
__global__ void ladder_table_kernel(int L, double* __restrict__ c) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (l >= L) return;
  const double ll = (double)l * (double)(l + 1), q = (double)k;
  c[(int64_t)k * L + l] =
      k < L + 2 ? 0.5 * sqrt(fmax(ll - q * (q - 1.0), 0.0)) : (l == 0 ? 0.0 : -1.0 / ll);
}

// Per call: the six coefficient fields of one order m (velocity_fields_at), in
// shared memory, their column scales and digits (FP64-bound: 27 us at L = 512
// where the fields alone took 38).  Also what the contraction
// leaves out: the spectra of the two poles (zero but for m = 0), and the stream
// function where it is asked for.  The ladder factors come from a table: their
// square roots and the division were two thirds of the FP64 work.
constexpr int kFieldThreads = 384;        // 256: 5 us more at L = 512, 128: 10
constexpr int kFieldStride = kCols + 1;   // doubles per degree (no bank conflicts)

__global__ void __launch_bounds__(kFieldThreads) velocity_digits_kernel(
    DigGeometry g, const double2* __restrict__ a, int lap, double2* __restrict__ psi_out,
    const double* __restrict__ c, const double* __restrict__ tab, unsigned char* __restrict__ tiles,
    int* __restrict__ aexp, double2* __restrict__ S) {
  extern __shared__ double fld[];   // [l - m][kFieldStride]
  __shared__ int emax[kCols];
  __shared__ double pole[2][kCols];
  const int m = blockIdx.x, L = g.L, n = L - m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kCols) emax[tid] = 1;
  if (psi_out)
    for (int l = tid; l < m; l += kFieldThreads) psi_out[(int64_t)m * L + l] = make_double2(0.0, 0.0);
  __syncthreads();
  int e[kCols];
#pragma unroll
  for (int k = 0; k < kCols; ++k) e[k] = 0;
  for (int i = tid; i < n; i += kFieldThreads) {
    const int l = m + i;
    const double d = lap ? c[(int64_t)(L + 2) * L + l] : 1.0;
    double cc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int q = m - 1 + k;   // q(q-1) is symmetric: order -1 as order 2
      cc[k] = c[(int64_t)(q < 0 ? 2 : q) * L + l];
    }
    double2 f[kVelLegendre];
    velocity_fields_at(a, L, l, m, d, cc, f);
#pragma unroll
    for (int k = 0; k < kVelLegendre; ++k) {
      fld[i * kFieldStride + 2 * k] = f[k].x;
      fld[i * kFieldStride + 2 * k + 1] = f[k].y;
      e[2 * k] = max(e[2 * k], (__double2hiint(f[k].x) >> 20) & 2047);
      e[2 * k + 1] = max(e[2 * k + 1], (__double2hiint(f[k].y) >> 20) & 2047);
    }
    if (psi_out) psi_out[(int64_t)m * L + l] = f[0];
  }
#pragma unroll
  for (int k = 0; k < kCols; ++k) {
    e[k] = __reduce_max_sync(0xffffffffu, e[k]);
    if (lane == 0) atomicMax(&emax[k], e[k]);
  }
  __syncthreads();
  if (tid < kCols) aexp[m * kCols + tid] = emax[tid] == 2047 ? kNonFinite : emax[tid];
  const int ke = groups16((n + 1) / 2), ko = groups16(n / 2);
  unsigned char* base = tiles + (int64_t)g.gbase[m] * kAGroup;
  for (int u = tid; u < 2 * (ke + ko) * kCols; u += kFieldThreads) {
    const int col = u % kCols, q = u / kCols, grp = q >> 1, half = q & 1, par = grp >= ke;
    const int k0 = 16 * (par ? grp - ke : grp) + 8 * half, ec = emax[col];
    long long v[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int k = par + 2 * (k0 + w);
      v[w] = k < n && ec < 2047 ? to_fixed(fld[k * kFieldStride + col], ec) : 0;
    }
    uint4 d[kDigits];
    digits8(v, d);
    unsigned char* o = base + (int64_t)grp * kAGroup + half * (kAGroup / 2) + (col >> 3) * 128 + (col & 7) * 16;
#pragma unroll
    for (int j = 0; j < kDigits; ++j) *(uint4*)(o + 2 * j * 128) = d[j];
  }
  // the poles
  if (m > 0) {
    if (tid < 2 * kVelSpectra) {
      const int64_t row = L + 1, t = tid & 1 ? L : 0;
      S[(int64_t)(tid >> 1) * row * row + t * row + m] = make_double2(0.0, 0.0);
    }
    return;
  }
  const int npair = L / 2 + 1;
  for (int col = warp; col < kCols; col += kFieldThreads / 32) {
    double v = 0.0;   // a lane's degrees have its parity
    for (int l = lane; l < L; l += 32) v += tab[(int64_t)l * npair] * fld[l * kFieldStride + col];
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const double odd = __shfl_down_sync(0xffffffffu, v, 1);
    if (lane == 0) {
      pole[0][col] = v + odd;
      pole[1][col] = v - odd;
    }
  }
  __syncthreads();
  if (tid < 2 * kVelLegendre) {
    const int f = tid >> 1, o = tid & 1;
    store_velocity_spectra(S, L, f, o ? L : 0, 0, make_double2(pole[o][2 * f], pole[o][2 * f + 1]));
  }
}

// ------------------------------------------------------------- synthesis
// Persistent, one block per SM, over the work items (m, row block) in order
// of decreasing length, dealt in alternating direction so that each block's
// share is about the same.  Three roles: warp 4 streams the chunks (up to 64
// degrees of one parity: 96 KiB of table, 14 KiB of data) into two stages by
// bulk copies, warp 5 issues a chunk's MMAs (six per 16 degrees) into one of
// two accumulators, and warps 0-3, a ring pair per lane, add the levels into
// 64-bit integers and write an item's spectra at its end.  Bounded by the
// table's bytes; copies of one stage are always in flight while the other is
// multiplied.  Every wait is bounded; a timeout in one role stops all.
struct DigCursor {
  int round, m, blk, ke, ko, nce, nch, c;
};

__device__ __forceinline__ bool dig_item(DigCursor& u, int nitems, const DigGeometry& g) {
  const int G = gridDim.x, b = blockIdx.x;
  const int item = u.round * G + ((u.round & 1) ? G - 1 - b : b);
  if (item >= nitems) return false;
  u.m = item / g.nblk;
  u.blk = item % g.nblk;
  const int n = g.L - u.m;
  u.ke = groups16((n + 1) / 2);
  u.ko = groups16(n / 2);
  u.nce = (u.ke + kChunkGroups - 1) / kChunkGroups;
  u.nch = u.nce + (u.ko + kChunkGroups - 1) / kChunkGroups;
  u.c = 0;
  return true;
}

__device__ __forceinline__ bool dig_next(DigCursor& u, int nitems, const DigGeometry& g) {
  if (++u.c < u.nch) return true;
  ++u.round;
  return dig_item(u, nitems, g);
}

// First group of the cursor's chunk in its item, and the number of groups.
__device__ __forceinline__ int chunk_groups(const DigCursor& u, int* first) {
  const bool odd = u.c >= u.nce;
  const int g0 = kChunkGroups * (odd ? u.c - u.nce : u.c);
  *first = (odd ? u.ke : 0) + g0;
  return min(kChunkGroups, (odd ? u.ko : u.ke) - g0);
}

__device__ __forceinline__ int row_groups(const DigGeometry& g, int blk) {
  return min(kRows / 8, (g.rows - blk * kRows + 7) / 8);
}

// v 2^p (v zero or normal)
__device__ __noinline__ double scale_wide(double v, int p) { return ldexp(v, p); }
__device__ __forceinline__ double scale2(double v, int p) {
  const int h = __double2hiint(v), e = (h >> 20) & 2047;
  if (e == 0) return v;
  if ((unsigned)(e + p - 1) >= 2046u) return scale_wide(v, p);
  return __hiloint2double(h + p * (1 << 20), __double2loint(v));
}

constexpr int kSynThreads = 192;

__global__ void __launch_bounds__(kSynThreads, 1) synth_digits_kernel(DigGeometry g, int nitems,
                                                                      const unsigned char* __restrict__ ptab,
                                                                      const int* __restrict__ pexp,
                                                                      const unsigned char* __restrict__ tiles,
                                                                      const int* __restrict__ aexp,
                                                                      double2* __restrict__ S,
                                                                      int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];   // kStages stages of kStage bytes
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_s;
  __shared__ int drain_fail_s;
  const int L = g.L;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int b = 0; b < kStages; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    abort_s = 0;
    drain_fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_s)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  DigCursor u;
  u.round = 0;
  if (warp == 4 && lane == 0) {
    const int rgt = (g.rows + 7) / 8;
    long long j = 0;
    bool ok = dig_item(u, nitems, g);
    while (ok && !abort_s) {
      const int st = (int)(j % kStages);
      if (j >= kStages && !wait_or_abort(&empty[st], (uint32_t)((j / kStages - 1) & 1), &abort_s)) break;
      int first;
      const int ng = chunk_groups(u, &first), gb = kRowGroupBytes * row_groups(g, u.blk);
      const int64_t base = g.gbase[u.m];
      const unsigned char* sp = ptab + base * kRowGroupBytes * rgt +
                                (int64_t)(u.ke + u.ko) * kRowGroupBytes * (kRows / 8) * u.blk + (int64_t)first * gb;
      unsigned char* d = smem + st * kStage;
      mbar_expect_tx(&full[st], (uint32_t)(ng * (gb + kAGroup)));
      bulk_g2s(d, sp, (uint32_t)(ng * gb), &full[st]);
      bulk_g2s(d + kPStage, tiles + (base + first) * kAGroup, (uint32_t)(ng * kAGroup), &full[st]);
      ++j;
      ok = dig_next(u, nitems, g);
    }
    // copies still in flight land before the block exits (bounded)
    if (abort_s) {
      bool drained = true;
      for (long long k = (j > kStages ? j - kStages : 0); k < j; ++k)
        drained &= mbar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1));
      if (!drained) drain_fail_s = 1;
    }
  } else if (warp == 5 && lane == 0) {
    const uint32_t s0 = smem_u32(smem);
    long long j = 0;
    bool committed = false;
    bool ok = dig_item(u, nitems, g);
    while (ok && !abort_s) {
      const int b = (int)(j & 1), st = (int)(j % kStages);
      if (j >= 2 && !wait_or_abort(&acc_empty[b], (uint32_t)(((j >> 1) - 1) & 1), &abort_s)) break;
      if (!wait_or_abort(&full[st], (uint32_t)((j / kStages) & 1), &abort_s)) break;
      tc_fence_after();
      int first;
      const int ng = chunk_groups(u, &first), rg = row_groups(g, u.blk);
      for (int q = 0; q < ng; ++q) {
        const uint32_t pa = s0 + st * kStage + q * kRowGroupBytes * rg;
        const uint64_t db = smem_desc(s0 + st * kStage + kPStage + q * kAGroup, kAGroup / 2, 128u);
        // rows past the block's last 8-row group read what lies behind it in
        // the stage; their results are not used
        for (int i = 0; i < kDigits; ++i)
          mma_bf16(tmem + b * 128 + 16 * i, smem_desc(pa + i * 2 * rg * 128, (uint32_t)rg * 128u, 128u), db,
                   mma_idesc(kAccCols - 16 * i), (q > 0 || i > 0) ? 1u : 0u);
      }
      mma_commit(&empty[st]);
      mma_commit(&acc_full[b]);
      committed = true;
      ++j;
      ok = dig_next(u, nitems, g);
    }
    // products in flight complete before the tensor memory is released (bounded)
    if (abort_s && committed) {
      const long long jl = j - 1;
      if (!mbar_wait(&empty[jl % kStages], (uint32_t)((jl / kStages) & 1))) drain_fail_s = 1;
    }
  } else if (warp < 4) {
    long long E[kCols], acc[kCols];   // units of 2^-52 of the scales' product
    float El[kCols], accl[kCols];     // the lower levels, in the same unit
#pragma unroll
    for (int k = 0; k < kCols; ++k) {
      E[k] = acc[k] = 0;
      El[k] = accl[k] = 0.f;
    }
    long long j = 0;
    bool have = dig_item(u, nitems, g);
    while (have) {
      const int b = (int)(j & 1);
      if (!wait_or_abort(&acc_full[b], (uint32_t)((j >> 1) & 1), &abort_s)) break;
      tc_fence_after();
      const bool rows_here = 32 * warp < 8 * row_groups(g, u.blk);   // uniform for the warp
      if (rows_here) {
        const uint32_t buf = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)b * 128;
        long long h[kCols];
#pragma unroll
        for (int s = 0; s < kLevels; ++s) {
          float v[16];
          tmem_ld16(buf + 16 * s, v);
#pragma unroll
          for (int k = 0; k < kCols; ++k) {
            if (s == 0)
              h[k] = __float2int_rn(v[k]);
            else if (s <= 4)
              h[k] = h[k] * 512 + __float2int_rn(v[k]);
            else
              accl[k] = fmaf(v[k], s == 5 ? 1.f / 512.f : 1.f / 262144.f, accl[k]);
          }
        }
#pragma unroll
        for (int k = 0; k < kCols; ++k) acc[k] += h[k];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
      if (u.c == u.nce - 1) {   // the even degrees are complete
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
          E[k] = acc[k];
          El[k] = accl[k];
          acc[k] = 0;
          accl[k] = 0.f;
        }
      }
      if (u.c == u.nch - 1) {   // the work item's last chunk: its spectra
        const int t = 1 + u.blk * kRows + 32 * warp + lane;
        if (t <= g.rows) {
          const int pe = pexp[(int64_t)u.m * g.rows + t - 1] - 2096;
          // value = (hi + lo) 2^54 2^(pe + ae - 2150), (hi + lo) 2^54 the
          // integers' products, the scales' exponents biased
          int ae_[kCols];   // all loads before the stores
#pragma unroll
          for (int k = 0; k < kCols; ++k) ae_[k] = aexp[u.m * kCols + k];
#pragma unroll
          for (int f = 0; f < kVelLegendre; ++f) {
            double v[2][2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int k = 2 * f + r, ae = ae_[k];
              v[0][r] = scale2((double)(E[k] + acc[k]) + (double)(El[k] + accl[k]), pe + ae);
              v[1][r] = scale2((double)(E[k] - acc[k]) + (double)(El[k] - accl[k]), pe + ae);
              if (ae == kNonFinite) v[0][r] = v[1][r] = __longlong_as_double(0x7ff8000000000000LL);
            }
            store_velocity_spectra(S, L, f, t, u.m, make_double2(v[0][0], v[0][1]));
            if (L - t != t) store_velocity_spectra(S, L, f, L - t, u.m, make_double2(v[1][0], v[1][1]));
          }
        }
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
          E[k] = acc[k] = 0;
          El[k] = accl[k] = 0.f;
        }
      }
      ++j;
      have = dig_next(u, nitems, g);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) {   // beside the status, a NaN on a ring: the velocity is seen to be unusable
    atomicOr(status, drain_fail_s ? CMM_FLAG_TIMEOUT | CMM_FLAG_DRAIN_TIMEOUT : CMM_FLAG_TIMEOUT);
    S[L + 1] = make_double2(__longlong_as_double(0x7ff8000000000000LL), 0.0);
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                 : "memory");
}

int check(const char* what) {
  note_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CMM_OK : cuda_fail(e, what);
}

}  // namespace

// Host side ---------------------------------------------------------------
struct DigitTables {
  int L = 0, sms = 1;
  DeviceBuffer gbase, digits, pexp, ladder;
  DigGeometry geometry() const {
    const int rows = L / 2;
    return DigGeometry{L, rows, (rows + kRows - 1) / kRows, (const int*)gbase.p};
  }
};

static int total_groups(int L) {
  int n = 0;
  for (int m = 0; m < L; ++m) n += groups16((L - m + 1) / 2) + groups16((L - m) / 2);
  return n;
}

int digit_tables_build(int L, const double* tab, std::shared_ptr<DigitTables>* out, cudaStream_t s) {
  auto t = std::make_shared<DigitTables>();
  t->L = L;
  const int rows = L / 2, rgt = (rows + 7) / 8;
  std::vector<int> gb(L + 1, 0);
  for (int m = 0; m < L; ++m) gb[m + 1] = gb[m] + groups16((L - m + 1) / 2) + groups16((L - m) / 2);
  int rc, dev = 0;
  if ((rc = t->gbase.upload(gb.data(), gb.size() * sizeof(int))) ||
      (rc = t->digits.alloc((size_t)gb[L] * kRowGroupBytes * rgt)) ||
      (rc = t->pexp.alloc((size_t)L * rows * sizeof(int))) ||
      (rc = t->ladder.alloc((size_t)(L + 3) * L * sizeof(double))))
    return rc;
  cudaError_t e = cudaStreamSynchronize(0);   // the upload, before s reads it
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(synth_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kStage);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(velocity_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kDigitMaxL * kFieldStride * (int)sizeof(double));
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&t->sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "digit_tables_build");
  const DigGeometry g = t->geometry();
  build_digits_kernel<<<dim3(g.nblk, L), kRows, 0, s>>>(g, tab, (unsigned char*)t->digits.p, (int*)t->pexp.p);
  if ((rc = check("build_digits_kernel"))) return rc;
  ladder_table_kernel<<<dim3((L + 127) / 128, L + 3), 128, 0, s>>>(L, (double*)t->ladder.p);
  if ((rc = check("ladder_table_kernel"))) return rc;
  *out = std::move(t);
  return CMM_OK;
}

int digit_workspace(int L, DeviceBuffer* tiles, DeviceBuffer* aexp) {
  int rc;
  if ((rc = aexp->alloc((size_t)L * kCols * sizeof(int))) || (rc = tiles->alloc((size_t)total_groups(L) * kAGroup)))
    return rc;
  // the padding columns and the zero block are never written; complete before
  // the caller's stream, which may not wait for this one, uses the tiles
  cudaError_t e = cudaMemset(tiles->p, 0, tiles->bytes);
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e == cudaSuccess) return CMM_OK;
  tiles->release();
  return cuda_fail(e, "cudaMemset(digit tiles)");
}

int digit_velocity(const DigitTables& t, const double* tab, const double2* a, bool lap, double2* psi_out,
                   void* tiles, void* aexp, double2* S, int* status, cudaStream_t s) {
  const DigGeometry g = t.geometry();
  const int L = t.L, nitems = L * g.nblk;
  velocity_digits_kernel<<<L, kFieldThreads, (size_t)L * kFieldStride * sizeof(double), s>>>(
      g, a, lap, psi_out, (const double*)t.ladder.p, tab, (unsigned char*)tiles, (int*)aexp, S);
  int rc = check("velocity_digits_kernel");
  if (rc) return rc;
  synth_digits_kernel<<<std::min(nitems, t.sms), kSynThreads, kStages * kStage, s>>>(
      g, nitems, (const unsigned char*)t.digits.p, (const int*)t.pexp.p, (const unsigned char*)tiles,
      (const int*)aexp, S, status);
  return check("synth_digits_kernel");
}

}  // namespace cmm
