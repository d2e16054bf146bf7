// FP64 velocity synthesis on the tensor cores (tcgen05, sm_103a) by exact
// integer digits.
//
// The Legendre synthesis of one order m is a product
//   S_even/odd[t][n] = sum_{l - m even/odd} Pbar_lm(theta_t) A[l][n]
// over ring pairs t and 12 real columns n (six complex fields).  GB300 has 2
// FP64 multiply-adds per SM and cycle, so FP64 arithmetic takes 12 L^3 / 4 of
// them (1.03 ms at L = 512) where the table's bytes need 60 us.  Instead, in
// each group of 16 degrees of one parity, every row of Pbar (over l) and every
// column of A gets the power of two above its largest entry as its scale, and
// each entry becomes the integer x 2^53 / scale, rounded (entries of the largest
// one's binade exactly, the others to half an ulp of it), cut into six signed
// digits of 9 bits: integers of at most 256, exact in bf16.  Products of digits
// i and j belong to level i + j; the levels' sums over a group are integers,
// accumulated exactly in FP32 in tensor memory (at most 6 x 16 x 2^16 < 2^24),
// and make one 64-bit integer.  Levels 7 and up (2^-61 of the scales' product)
// are left out.  The groups' integers are added in 64 bits at the largest scale
// met.  The scheme is known as Ozaki splitting.  The scales follow the decay of
// a smooth field's coefficients and the growth of Pbar towards high degrees near
// the poles within 32 degrees.  Against exact sums (60 draws per case): a ring's
// spectrum over all orders errs by 0.7 to 7e-16 of its size (FP64 0.5 to 10e-16;
// coefficients e^(-l/3) to e^(-l/40), polar to equatorial rings of L = 256).  A
// single order far below the others on its ring, as sin^m is next to the poles,
// loses more of its own value: e^(-l/8) at L = 512, first five rings, 5e-15 on
// average at order 2 and 4e-15 at 20 (FP64 8e-16 and 9e-16), e^(-l/40) 6e-16 at 1 and
// 9e-16 at 20 (FP64 10e-16 and 8e-16); with a scale per 64 degrees 4e-14 and 2e-10,
// with one for all degrees 4e-13 and 2e-2 (e^(-l/8)).
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
constexpr int kMaxGroups = 2 * (kDigitMaxL / 32);          // degree groups of one order
constexpr int kAccs = 4;                // accumulators, of one degree group each
constexpr int kScaleBytes = kChunkGroups * (2 * kRows + 4 * kCols);   // a chunk's scales: rows' shorts, columns' ints
constexpr int kScales = 4;              // chunks of them
constexpr int kSmemBytes = kStages * kStage + kScales * kScaleBytes;
constexpr int kAccCols = 16 * kLevels;  // 112 of 128 TMEM columns per accumulator
constexpr uint32_t kTmemCols = 128 * kAccs;
constexpr int kNonFinite = 1 << 20;     // column scale of a group with an infinity or NaN

struct DigGeometry {
  int L, rows, nblk;      // ring pairs t = 1 .. rows, in nblk blocks
  const int* gbase;       // (L+1) prefix sums of the degree groups per m
};

// ----------------------------------------------------------- tables, data
// Block (row block, degree group, m): the digit table of its rows and degrees
// from the FP64 table tab[m][l - m][t], one thread per row; the rows' scales in
// pexp, laid out as the table: [m][row block][group][row].
__global__ void __launch_bounds__(kRows) build_digits_kernel(DigGeometry g, const double* __restrict__ tab,
                                                             unsigned char* __restrict__ out,
                                                             short* __restrict__ pexp) {
  const int blk = blockIdx.x, grp = blockIdx.y, m = blockIdx.z, row = threadIdx.x, L = g.L;
  const int npair = L / 2 + 1, t = 1 + blk * kRows + row, n = L - m;
  const int rg = min(kRows / 8, (g.rows - blk * kRows + 7) / 8), rgt = (g.rows + 7) / 8;
  const int ke = groups16((n + 1) / 2), ko = groups16(n / 2), par = grp >= ke;
  if (grp >= ke + ko || row >= 8 * rg) return;
  const bool real = t <= g.rows;
  const double* P = tab + tab_off(m, L, npair) + t;
  const int k0 = par + 32 * (par ? grp - ke : grp);
  double x[16];
  int e = 1;
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    x[u] = real && k0 + 2 * u < n ? P[(int64_t)(k0 + 2 * u) * npair] : 0.0;
    e = max(e, (__double2hiint(x[u]) >> 20) & 2047);
  }
  unsigned char* o = out + (int64_t)g.gbase[m] * kRowGroupBytes * rgt +
                     (int64_t)(ke + ko) * kRowGroupBytes * (kRows / 8) * blk + (int64_t)grp * kRowGroupBytes * rg +
                     (row >> 3) * 128 + (row & 7) * 16;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    long long v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = to_fixed(x[8 * half + u], e);
    uint4 d[kDigits];
    digits8(v, d);
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4*)(o + (2 * i + half) * rg * 128) = d[i];
  }
  pexp[(int64_t)g.gbase[m] * 8 * rgt + (int64_t)(ke + ko) * kRows * blk + grp * 8 * rg + row] = (short)e;
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
  __shared__ int emax[kMaxGroups][kCols];
  __shared__ double pole[2][kCols];
  const int m = blockIdx.x, L = g.L, n = L - m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ke = groups16((n + 1) / 2), ko = groups16(n / 2);
  if (psi_out)
    for (int l = tid; l < m; l += kFieldThreads) psi_out[(int64_t)m * L + l] = make_double2(0.0, 0.0);
  for (int i0 = 32 * warp; i0 < n; i0 += kFieldThreads) {   // a warp's degrees: one group of either parity
    const int i = i0 + lane, l = m + i;
    double2 f[kVelLegendre];
#pragma unroll
    for (int k = 0; k < kVelLegendre; ++k) f[k] = make_double2(0.0, 0.0);
    if (i < n) {
      const double d = lap ? c[(int64_t)(L + 2) * L + l] : 1.0;
      double cc[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = m - 1 + k;   // q(q-1) is symmetric: order -1 as order 2
        cc[k] = c[(int64_t)(q < 0 ? 2 : q) * L + l];
      }
      velocity_fields_at(a, L, l, m, d, cc, f);
      if (psi_out) psi_out[(int64_t)m * L + l] = f[0];
#pragma unroll
      for (int k = 0; k < kVelLegendre; ++k) {
        fld[i * kFieldStride + 2 * k] = f[k].x;
        fld[i * kFieldStride + 2 * k + 1] = f[k].y;
      }
    }
    const int grp = (lane & 1 ? ke : 0) + i0 / 32;
#pragma unroll
    for (int k = 0; k < kCols; ++k) {
      const int e = max(1, (__double2hiint(k & 1 ? f[k >> 1].y : f[k >> 1].x) >> 20) & 2047);
      const int ev = __reduce_max_sync(0xffffffffu, lane & 1 ? 0 : e), od = __reduce_max_sync(0xffffffffu, lane & 1 ? e : 0);
      if (lane < 2 && grp < ke + ko) emax[grp][k] = lane ? od : ev;
    }
  }
  __syncthreads();
  for (int k = tid; k < (ke + ko) * kCols; k += kFieldThreads)
    aexp[g.gbase[m] * kCols + k] = emax[0][k] == 2047 ? kNonFinite : emax[0][k];
  unsigned char* base = tiles + (int64_t)g.gbase[m] * kAGroup;
  for (int u = tid; u < 2 * (ke + ko) * kCols; u += kFieldThreads) {
    const int col = u % kCols, q = u / kCols, grp = q >> 1, half = q & 1, par = grp >= ke;
    const int k0 = 16 * (par ? grp - ke : grp) + 8 * half, ec = emax[grp][col];
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
// share is about the same.  Three roles: warp 12 streams the chunks (up to 64
// degrees of one parity: 96 KiB of table, 14 KiB of data) into two stages by
// bulk copies, warp 13 issues six MMAs per group of 16 degrees into one of four
// accumulators, and warps 0-11, a ring pair and four columns per lane, add the
// groups' levels to 64-bit integers and write an item's spectra at its end.  Bounded by the
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

constexpr int kAddWarps = 12, kAddCols = kCols / 3;
constexpr int kSynThreads = 32 * (kAddWarps + 2);

__global__ void __launch_bounds__(kSynThreads, 1) synth_digits_kernel(DigGeometry g, int nitems,
                                                                      const unsigned char* __restrict__ ptab,
                                                                      const short* __restrict__ pexp,
                                                                      const unsigned char* __restrict__ tiles,
                                                                      const int* __restrict__ aexp,
                                                                      double2* __restrict__ S,
                                                                      int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];   // the stages, then the chunks' scales
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[kAccs], acc_empty[kAccs];
  __shared__ __align__(8) uint64_t sc_full[kScales], sc_empty[kScales];
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
    for (int b = 0; b < kScales; ++b) {
      mbar_init(&sc_full[b], 1);
      mbar_init(&sc_empty[b], kAddWarps);
    }
    for (int b = 0; b < kAccs; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kAddWarps);
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
  if (warp == kAddWarps && lane == 0) {
    const int rgt = (g.rows + 7) / 8;
    long long j = 0;
    bool ok = dig_item(u, nitems, g);
    while (ok && !abort_s) {
      const int st = (int)(j % kStages);
      if (j >= kStages && !wait_or_abort(&empty[st], (uint32_t)((j / kStages - 1) & 1), &abort_s)) break;
      const int sc = (int)(j % kScales);
      if (j >= kScales && !wait_or_abort(&sc_empty[sc], (uint32_t)((j / kScales - 1) & 1), &abort_s)) break;
      int first;
      const int ng = chunk_groups(u, &first), gb = kRowGroupBytes * row_groups(g, u.blk);
      const int64_t base = g.gbase[u.m];
      const unsigned char* sp = ptab + base * kRowGroupBytes * rgt +
                                (int64_t)(u.ke + u.ko) * kRowGroupBytes * (kRows / 8) * u.blk + (int64_t)first * gb;
      unsigned char* d = smem + st * kStage;
      mbar_expect_tx(&full[st], (uint32_t)(ng * (gb + kAGroup)));
      bulk_g2s(d, sp, (uint32_t)(ng * gb), &full[st]);
      bulk_g2s(d + kPStage, tiles + (base + first) * kAGroup, (uint32_t)(ng * kAGroup), &full[st]);
      unsigned char* e = smem + kStages * kStage + sc * kScaleBytes;
      const int rows = 8 * row_groups(g, u.blk);
      mbar_expect_tx(&sc_full[sc], (uint32_t)(ng * (2 * rows + 4 * kCols)));
      bulk_g2s(e, aexp + (base + first) * kCols, (uint32_t)(4 * ng * kCols), &sc_full[sc]);
      bulk_g2s(e + 4 * kChunkGroups * kCols, pexp + base * 8 * rgt + (int64_t)(u.ke + u.ko) * kRows * u.blk + first * rows,
               (uint32_t)(2 * ng * rows), &sc_full[sc]);
      ++j;
      ok = dig_next(u, nitems, g);
    }
    // copies still in flight land before the block exits (bounded)
    if (abort_s) {
      bool drained = true;
      for (long long k = (j > kStages ? j - kStages : 0); k < j; ++k)
        drained &= mbar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1));
      for (long long k = (j > kScales ? j - kScales : 0); k < j; ++k)
        drained &= mbar_wait(&sc_full[k % kScales], (uint32_t)((k / kScales) & 1));
      if (!drained) drain_fail_s = 1;
    }
  } else if (warp == kAddWarps + 1 && lane == 0) {
    const uint32_t s0 = smem_u32(smem);
    long long j = 0, k = 0;   // chunks, groups
    bool ok = dig_item(u, nitems, g), stop = false;
    while (ok && !stop && !abort_s) {
      const int st = (int)(j % kStages);
      if (!wait_or_abort(&full[st], (uint32_t)((j / kStages) & 1), &abort_s)) break;
      int first;
      const int ng = chunk_groups(u, &first), rg = row_groups(g, u.blk);
      for (int q = 0; q < ng; ++q, ++k) {
        const int b = (int)(k % kAccs);
        if (k >= kAccs && !wait_or_abort(&acc_empty[b], (uint32_t)((k / kAccs - 1) & 1), &abort_s)) {
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t pa = s0 + st * kStage + q * kRowGroupBytes * rg;
        const uint64_t db = smem_desc(s0 + st * kStage + kPStage + q * kAGroup, kAGroup / 2, 128u);
        // rows past the block's last 8-row group read what lies behind it in
        // the stage; their results are not used
        for (int i = 0; i < kDigits; ++i)
          mma_bf16(tmem + b * 128 + 16 * i, smem_desc(pa + i * 2 * rg * 128, (uint32_t)rg * 128u, 128u), db,
                   mma_idesc(kAccCols - 16 * i), i > 0 ? 1u : 0u);
        mma_commit(&acc_full[b]);
      }
      if (stop) break;
      mma_commit(&empty[st]);
      ++j;
      ok = dig_next(u, nitems, g);
    }
    // products in flight complete before the tensor memory is released (bounded)
    if (abort_s && k > 0 && !mbar_wait(&acc_full[(k - 1) % kAccs], (uint32_t)(((k - 1) / kAccs) & 1))) drain_fail_s = 1;
  } else if (warp < kAddWarps) {
    constexpr int N = kAddCols;
    const int quad = warp & 3, col0 = N * (warp >> 2);
    const uint32_t lanes = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)col0;
    // sums in units of 2^53 2^(ex - 2150) (below 2^62: 32 groups of 2^57), ex the
    // largest of the groups' exponents so far; the even degrees' beside
    long long acc[N], E[N];
    int ex[N], Ex[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      acc[n] = 0;
      ex[n] = 0;
    }
    // a level's sum as an integer, |x| <= 2^22: the bits of 1.5 2^23 + x, less
    // those of 1.5 2^23 (taken off the group's products at once)
    constexpr long long kBits = 0x4B400000LL;
    auto bits = [](float x) { return __float_as_int(__fadd_rn(x, 12582912.f)); };
    // Two groups of a chunk at a time (one where a parity has an odd number), the
    // next ones' first levels on their way from tensor memory while these are
    // added: one by one, the waits and the bookkeeping took as long as the sums.
    // Rows past the last ring: never stored.
    float v[N * kLevels];
    auto start = [&](unsigned k, bool two) {
      const unsigned last = k + two;
      if (!warp_wait(&acc_full[last % kAccs], (last / kAccs) & 1, &abort_s)) return false;
      tc_fence_after();
      tmem_start7x4(lanes + k % kAccs * 128, 16, v);
      return true;
    };
    auto products = [&](long long* h) {   // in units of 2^53
      const float* x = v;
      tmem_wait7x4(v);
#pragma unroll
      for (int n = 0; n < N; ++n) {
        h[n] = mad_wide(bits(x[n]), 1 << 27, -kBits * ((1 << 27) + (1 << 18) + 512 + 1));   // 512^3; 512 and 2 to come
        h[n] = mad_wide(bits(x[N + n]), 1 << 18, h[n]);
        h[n] = mad_wide(bits(x[2 * N + n]), 512, h[n]);
        h[n] = mad_wide(bits(x[3 * N + n]), 1, h[n]);
        h[n] = mad_wide(__float2int_rn(x[4 * N + n]), 2, h[n] * 1024);
        h[n] = mad_wide(__float2int_rn(fmaf(x[6 * N + n], 2.f / 262144.f, x[5 * N + n] * (2.f / 512.f))), 1, h[n]);
      }
    };
    int i = 0, q = 0;   // group of the item, of the chunk
    unsigned j = 0;     // chunks
    bool have = dig_item(u, nitems, g);
    bool two = u.ke > 1;
    have = have && start(0, two);
    int rows = have ? 8 * row_groups(g, u.blk) : 0;
#pragma unroll 1
    for (unsigned k = 0; have;) {   // groups
      long long h[2][N];
      products(h[0]);
      if (two) {
        tmem_start7x4(lanes + (k + 1) % kAccs * 128, 16, v);
        products(h[1]);
      } else {
#pragma unroll
        for (int n = 0; n < N; ++n) h[1][n] = 0;
      }
      tc_fence_before();
      __syncwarp();
      if (lane <= two)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[(k + lane) % kAccs])) : "memory");
      // the groups' scales, exponents biased
      const unsigned sc = j % kScales;
      if (q == 0 && !warp_wait(&sc_full[sc], (j / kScales) & 1, &abort_s)) break;
      const unsigned char* scales = smem + kStages * kStage + sc * kScaleBytes;
      const short* pes = (const short*)(scales + 4 * kChunkGroups * kCols) + q * rows + min(32 * quad + lane, rows - 1);
      const int4* aes = (const int4*)(scales + 4 * (q * kCols + col0));
      int e[2][N];
      {
        const int pe = pes[0];
        const int4 a = aes[0];
        e[0][0] = pe + a.x, e[0][1] = pe + a.y, e[0][2] = pe + a.z, e[0][3] = pe + a.w;
      }
      if (two) {
        const int pe = pes[rows];
        const int4 a = aes[kCols / 4];
        e[1][0] = pe + a.x, e[1][1] = pe + a.y, e[1][2] = pe + a.z, e[1][3] = pe + a.w;
      } else {
#pragma unroll
        for (int n = 0; n < N; ++n) e[1][n] = 0;
      }
      i += 1 + two;
      q += 1 + two;
      k += 1 + two;
      const bool even_end = i == u.ke, item_end = i == u.ke + u.ko;
      const bool chunk_end = even_end || item_end || q == kChunkGroups;
      const int m = u.m, t = 1 + u.blk * kRows + 32 * quad + lane;
      if (chunk_end) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sc_empty[sc])) : "memory");
        ++j;
        q = 0;
      }
      if (item_end) {
        ++u.round;
        have = dig_item(u, nitems, g);
        rows = 8 * row_groups(g, u.blk);
        i = 0;
      }
      two = (i < u.ke ? u.ke : u.ke + u.ko) - i > 1;
      have = have && start(k, two);
      // at the largest of the scales, rounded
      bool up = false;
#pragma unroll
      for (int n = 0; n < N; ++n) up = up || max(e[0][n], e[1][n]) > ex[n];
      if (__any_sync(0xffffffffu, up)) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
          const int to = max(ex[n], max(e[0][n], e[1][n])), d = min(to - ex[n], 62);
          acc[n] = (acc[n] + ((1LL << d) >> 1)) >> d;
          ex[n] = to;
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int n = 0; n < N; ++n) {
          const int d = min(ex[n] - e[w][n], 62);
          acc[n] += (h[w][n] + ((1LL << d) >> 1)) >> d;
        }
      if (even_end) {   // the even degrees are complete
#pragma unroll
        for (int n = 0; n < N; ++n) {
          E[n] = acc[n];
          Ex[n] = ex[n];
          acc[n] = 0;
          ex[n] = 0;
        }
      }
      if (item_end) {   // the item's spectra
#pragma unroll
        for (int f = 0; f < N / 2; ++f) {
          double z[2][2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int n = 2 * f + r;
            // an integer unit is 2^53 2^(pe - 1075) 2^(ae - 1075)
            const double ev = fixed_to_double(E[n], Ex[n] - 2097), od = fixed_to_double(acc[n], ex[n] - 2097);
            z[0][r] = ev + od;
            z[1][r] = ev - od;
            if (max(Ex[n], ex[n]) >= kNonFinite) z[0][r] = z[1][r] = __longlong_as_double(0x7ff8000000000000LL);
            acc[n] = 0;
            ex[n] = 0;
          }
          const int fld = f + col0 / 2;
          if (t <= g.rows) store_velocity_spectra(S, L, fld, t, m, make_double2(z[0][0], z[0][1]));
          if (t <= g.rows && L - t != t) store_velocity_spectra(S, L, fld, L - t, m, make_double2(z[1][0], z[1][1]));
        }
      }
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
  int* gbase = nullptr;
  unsigned char* digits = nullptr;
  short* pexp = nullptr;
  double* ladder = nullptr;
  DigGeometry geometry() const {
    const int rows = L / 2;
    return DigGeometry{L, rows, (rows + kRows - 1) / kRows, gbase};
  }
};

static int total_groups(int L) {
  int n = 0;
  for (int m = 0; m < L; ++m) n += groups16((L - m + 1) / 2) + groups16((L - m) / 2);
  return n;
}

static size_t aligned(size_t n) { return (n + 255) / 256 * 256; }
static size_t digits_bytes(int L) { return aligned((size_t)total_groups(L) * kRowGroupBytes * ((L / 2 + 7) / 8)); }
static size_t pexp_bytes(int L) { return aligned((size_t)total_groups(L) * 8 * ((L / 2 + 7) / 8) * sizeof(short)); }
static size_t ladder_bytes(int L) { return aligned((size_t)(L + 3) * L * sizeof(double)); }

size_t digit_tables_bytes(int L) {
  return digits_bytes(L) + pexp_bytes(L) + ladder_bytes(L) + (L + 1) * sizeof(int);
}

int digit_tables_build(int L, const double* tab, void* mem, std::shared_ptr<DigitTables>* out, cudaStream_t s) {
  auto t = std::make_shared<DigitTables>();
  t->L = L;
  t->digits = (unsigned char*)mem;
  t->pexp = (short*)(t->digits + digits_bytes(L));
  t->ladder = (double*)((unsigned char*)t->pexp + pexp_bytes(L));
  t->gbase = (int*)((unsigned char*)t->ladder + ladder_bytes(L));
  std::vector<int> gb(L + 1, 0);
  for (int m = 0; m < L; ++m) gb[m + 1] = gb[m] + groups16((L - m + 1) / 2) + groups16((L - m) / 2);
  int rc, dev = 0;
  // from pageable memory: staged before the call returns
  cudaError_t e = cudaMemcpyAsync(t->gbase, gb.data(), gb.size() * sizeof(int), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(synth_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(velocity_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kDigitMaxL * kFieldStride * (int)sizeof(double));
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&t->sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "digit_tables_build");
  const DigGeometry g = t->geometry();
  build_digits_kernel<<<dim3(g.nblk, gb[1], L), kRows, 0, s>>>(g, tab, t->digits, t->pexp);
  if ((rc = check("build_digits_kernel"))) return rc;
  ladder_table_kernel<<<dim3((L + 127) / 128, L + 3), 128, 0, s>>>(L, t->ladder);
  if ((rc = check("ladder_table_kernel"))) return rc;
  *out = std::move(t);
  return CMM_OK;
}

// Workspace of a plan: the data tiles, whose padding columns and zero block are
// never written and have to be zero, then the column scales.
static size_t tile_bytes(int L) { return aligned((size_t)total_groups(L) * kAGroup); }
size_t digit_work_bytes(int L) { return tile_bytes(L) + aligned((size_t)total_groups(L) * kCols * sizeof(int)); }
int digit_work_clear(int L, void* work, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(work, 0, tile_bytes(L), s);
  return e == cudaSuccess ? CMM_OK : cuda_fail(e, "cudaMemsetAsync(digit tiles)");
}

int digit_velocity(const DigitTables& t, const double* tab, const double2* a, bool lap, double2* psi_out, void* work,
                   double2* S, int* status, cudaStream_t s) {
  const DigGeometry g = t.geometry();
  const int L = t.L, nitems = L * g.nblk;
  unsigned char* tiles = (unsigned char*)work;
  int* aexp = (int*)(tiles + tile_bytes(L));
  velocity_digits_kernel<<<L, kFieldThreads, (size_t)L * kFieldStride * sizeof(double), s>>>(g, a, lap, psi_out, t.ladder,
                                                                                            tab, tiles, aexp, S);
  int rc = check("velocity_digits_kernel");
  if (rc) return rc;
  synth_digits_kernel<<<std::min(nitems, t.sms), kSynThreads, kSmemBytes, s>>>(g, nitems, t.digits, t.pexp, tiles, aexp, S,
                                                                              status);
  return check("synth_digits_kernel");
}

}  // namespace cmm
