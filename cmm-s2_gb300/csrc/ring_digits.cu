// Inverse ring transforms of the FP64 velocity (complex to real, length 2L) by
// exact digits on the tensor cores (tcgen05, sm_103a; sht_digits.cu describes
// the scheme).
//
// x[p] = Re S_0 + 2 sum_{m<L} (Re S_m cos(pi m p / L) - Im S_m sin(pi m p / L)).
// FP64-bound as a fast transform (339 us for 9 x 513 rings at L = 512, where
// the bytes need 11; this: 34 us of digits and 96 of products; L = 256: 73 -> 12
// + 27).  The four sums over even and odd m
//   Ce, Co = sum 2 Re S_m cos,   Se, So = sum 2 Im S_m sin
// at p = 1 .. L/2 give x at p, 2L-p, L-p and L+p:
//   Ce + Co -+ (Se + So),  Ce - Co +- (Se - So),
// L^2 multiply-adds per ring.  The table is the digits of cos and sin (scale 1);
// a ring's data has one scale per 64 orders of one parity (the accumulation
// chunk), so that the digits' half-ulp truncation follows a spectrum's decay;
// the chunks' integer sums are shifted to the ring's largest scale and added as
// 64-bit integers.
// x[0] and x[L] are plain sums, made with the digits.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <memory>

#include "cmm_internal.h"
#include "device_common.cuh"
#include "digits.cuh"
#include "tc.cuh"

namespace cmm {

using namespace dig;
using namespace tc;

namespace {

constexpr int kRows = 128;              // rings per work item (MMA M)
constexpr int kChunk = 4;               // groups of 16 orders per accumulation chunk
constexpr int kMaxChunks = kDigitMaxL / 2 / 64;   // chunks of one parity
constexpr int kAGroup = kDigits * 2 * 128 * (kRows / 8);   // bytes of one group of the data
constexpr int kStages = 4;              // of one group each
constexpr int kNonFinite = 2047;

// Bytes of one group of the table for a tile of NT columns (and its zero block).
__host__ __device__ constexpr int b_group(int NT) { return 2 * kLevels * NT / 8 * 128; }
__host__ __device__ constexpr int stage_bytes(int NT) { return kAGroup + b_group(NT); }

struct RingGeometry {
  int L, rows;            // rings (all fields)
  int ke, ko;             // groups of the even and odd orders
  int ntile;              // column tiles of NT
  __host__ __device__ int groups() const { return 2 * (ke + ko); }
  __host__ __device__ int count(int type) const { return type & 1 ? ko : ke; }
  // first group of type 0..3 = (cos, even), (cos, odd), (sin, even), (sin, odd)
  __host__ __device__ int first(int type) const { return (type >> 1) * (ke + ko) + (type & 1) * ke; }
};

// Table: [tile][group][half of 8 orders][8-column groups][8 columns][8 orders],
// column j NT + c for digit j of p = 1 + NT tile + c; zero for p > L/2.
template <int NT>
__global__ void ring_table_kernel(RingGeometry g, unsigned char* __restrict__ out) {
  const int tile = blockIdx.y, grp = blockIdx.x, L = g.L;
  const int c = threadIdx.x % NT, half = threadIdx.x / NT;   // 2 NT threads
  int type = 0;
  while (type < 3 && grp >= g.first(type + 1)) ++type;
  const int k0 = 16 * (grp - g.first(type)) + 8 * half, p = 1 + NT * tile + c;
  long long v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int m = (type & 1) + 2 * (k0 + u);
    v[u] = 0;
    if (m < L && p <= L / 2) {
      const int r = (int)(((long long)m * p) % (2 * L));
      const double a = (double)r / (double)L;
      v[u] = to_fixed(type < 2 ? cospi(a) : sinpi(a), 1022);
    }
  }
  uint4 d[kDigits];
  digits8(v, d);
  unsigned char* o = out + ((int64_t)tile * g.groups() + grp) * b_group(NT) + half * (b_group(NT) / 2);
#pragma unroll
  for (int j = 0; j < kDigits; ++j) {
    const int n = j * NT + c;
    *(uint4*)(o + (n >> 3) * 128 + (n & 7) * 16) = d[j];
  }
}

// Per call, 8 rings per block: the data digits [128-ring block][group][6
// digits][2 halves][16 8-ring groups][8][8 orders], the chunks' scales and the
// samples x[0], x[L].  S: (rows, L+1) spectra, m = L unused.
constexpr int kDataThreads = 256;

__global__ void __launch_bounds__(kDataThreads) ring_digits_kernel(RingGeometry g, const double2* __restrict__ S,
                                                                   unsigned char* __restrict__ out,
                                                                   int* __restrict__ rexp,
                                                                   unsigned char* __restrict__ shift,
                                                                   double* __restrict__ x) {
  extern __shared__ double2 sm[];   // [8][L + 1 (odd count of 16 bytes: no bank conflicts)]
  __shared__ int ce[8][2][kMaxChunks];
  const int L = g.L, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int stride = (L + 1) | 1;
  const int row0 = blockIdx.x * 8;
  {
    const int r = row0 + warp;
    const bool real = r < g.rows;
    double s = 0.0;
    int emax = 1;
    for (int c = 0; 128 * c < L; ++c) {
      int e = 1;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = 128 * c + 32 * q + lane;
        double2 v = make_double2(0.0, 0.0);
        if (real && m < L) {
          v = S[(int64_t)r * (L + 1) + m];
          if (m == 0) v = make_double2(0.5 * v.x, 0.0);
          sm[warp * stride + m] = v;
        } else if (m < L) {
          sm[warp * stride + m] = v;
        }
        s += v.x;
        e = max(e, max((__double2hiint(v.x) >> 20) & 2047, (__double2hiint(v.y) >> 20) & 2047));
      }
#pragma unroll
      for (int o = 2; o < 32; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));   // by parity of m
      if (lane < 2) ce[warp][lane][c] = e;
      emax = max(emax, e);
    }
#pragma unroll
    for (int o = 2; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 1));
    const double odd = __shfl_xor_sync(0xffffffffu, s, 1);
    if (real && lane < 2) {   // lane 0: even sum in s; lane 1: odd sum in s
      if (lane == 0) {
        rexp[r] = emax;
        x[(int64_t)r * 2 * L] = 2.0 * (s + odd);
        x[(int64_t)r * 2 * L + L] = 2.0 * (s - odd);
      }
      for (int c = 0; 128 * c < L; ++c)
        shift[(int64_t)r * 2 * kMaxChunks + lane * kMaxChunks + c] = (unsigned char)min(emax - ce[warp][lane][c], 255);
    }
  }
  __syncthreads();
  const int row = tid & 7, G = g.groups();
  const int64_t r = row0 + row;
  unsigned char* base = out + (r / kRows) * G * (int64_t)kAGroup + ((r % kRows) >> 3) * 128 + row * 16;
  for (int u = tid >> 3; u < 2 * G; u += kDataThreads / 8) {
    const int half = u & 1, grp = u >> 1;
    int type = 0;
    while (type < 3 && grp >= g.first(type + 1)) ++type;
    const int k0 = 16 * (grp - g.first(type)) + 8 * half, par = type & 1;
    const int e = ce[row][par][k0 >> 6];
    long long v[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int m = par + 2 * (k0 + w);
      v[w] = 0;
      if (m < L && e < kNonFinite) {
        const double2 z = sm[row * stride + m];
        v[w] = to_fixed(type < 2 ? z.x : z.y, e);
      }
    }
    uint4 d[kDigits];
    digits8(v, d);
    unsigned char* o = base + (int64_t)grp * kAGroup + half * (kRows / 8) * 128;
#pragma unroll
    for (int i = 0; i < kDigits; ++i) *(uint4*)(o + i * 2 * (kRows / 8) * 128) = d[i];
  }
}

// Persistent over the items (block of 128 rings, tile of NT columns).  Warp 8
// streams groups of 16 orders into four stages, warp 9 issues the MMAs (N = NT
// (7 - i) for data digit i: level i + j at column NT (i + j); the zero block
// clears level 6) into one of two accumulators per chunk of 64 orders, and
// warps 0-7, with NT / 2 columns and 32 rings each, shift and add the chunks'
// sums (integer multiply-adds) and write the samples through shared memory,
// NT / 2 neighbours at a time.  At L = 512 a chunk's MMAs take 1800 cycles, its
// sums 2000, an item's samples 15000.
constexpr int kDrainWarps = 8;
constexpr int kRingThreads = 32 * (kDrainWarps + 2);

template <int NT>
struct RingShape {
  static constexpr int kCols = NT / 2;                      // columns of one adding warp
  static constexpr int kAccStride = NT == 32 ? 256 : 128;   // TMEM columns per accumulator (7 NT used)
  static constexpr int kOutStride = kCols + 1;
  static constexpr int kKept = 2;                           // types kept in shared memory until the end
  static constexpr int kWarpBytes = 32 * 8 * (kOutStride + kKept * kCols);
  static constexpr int kSmem = kStages * stage_bytes(NT) + kDrainWarps * kWarpBytes;
};

struct RingCursor {
  int item, type, c;   // work item, type of sum, chunk of the type
};

__device__ __forceinline__ int chunks(int groups) { return (groups + kChunk - 1) / kChunk; }

__device__ __forceinline__ bool ring_next(RingCursor& u, int nitems, const RingGeometry& g) {
  if (++u.c < chunks(g.count(u.type))) return true;
  u.c = 0;
  if (++u.type < 4) return true;
  u.type = 0;
  u.item += gridDim.x;
  return u.item < nitems;
}

template <int NT>
__global__ void __launch_bounds__(kRingThreads, 1)
    ring_synthesis_digits_kernel(RingGeometry g, int nitems, int xbit, const unsigned char* __restrict__ data,
                                 const int* __restrict__ rexp, const unsigned char* __restrict__ shift,
                                 const unsigned char* __restrict__ table, double* __restrict__ x,
                                 int* __restrict__ status) {
  using Sh = RingShape<NT>;
  constexpr int kDrain = kDrainWarps;
  constexpr uint32_t kTmemCols = 2 * Sh::kAccStride;
  constexpr int kStage = stage_bytes(NT);
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_s;
  __shared__ int drain_fail_s;
  const int L = g.L, G = g.groups();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int b = 0; b < kStages; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kDrain);
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
  RingCursor u;
  u.item = blockIdx.x;
  u.type = u.c = 0;
  bool have = u.item < nitems;
  if (warp == kDrain && lane == 0) {
    long long j = 0;   // stages
    bool stop = false;
    while (have && !abort_s && !stop) {
      const int rb = u.item / g.ntile, tile = u.item % g.ntile;
      const int n = min(kChunk, g.count(u.type) - kChunk * u.c), g0 = g.first(u.type) + kChunk * u.c;
      for (int q = 0; q < n; ++q) {
        const int st = (int)(j % kStages);
        if (j >= kStages && !wait_or_abort(&empty[st], (uint32_t)((j / kStages - 1) & 1), &abort_s)) {
          stop = true;
          break;
        }
        unsigned char* d = smem + st * kStage;
        mbar_expect_tx(&full[st], (uint32_t)kStage);
        bulk_g2s(d, data + ((int64_t)rb * G + g0 + q) * kAGroup, (uint32_t)kAGroup, &full[st]);
        bulk_g2s(d + kAGroup, table + ((int64_t)tile * G + g0 + q) * b_group(NT), (uint32_t)b_group(NT), &full[st]);
        ++j;
      }
      have = ring_next(u, nitems, g);
    }
    if (abort_s) {   // copies still in flight land before the block exits (bounded)
      bool drained = true;
      for (long long k = (j > kStages ? j - kStages : 0); k < j; ++k)
        drained &= mbar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1));
      if (!drained) drain_fail_s = 1;
    }
  } else if (warp == kDrain + 1 && lane == 0) {
    const uint32_t s0 = smem_u32(smem);
    long long j = 0, k = 0;   // stages, chunks
    bool stop = false;
    while (have && !abort_s && !stop) {
      const int b = (int)(k & 1);
      if (k >= 2 && !wait_or_abort(&acc_empty[b], (uint32_t)(((k >> 1) - 1) & 1), &abort_s)) break;
      const int n = min(kChunk, g.count(u.type) - kChunk * u.c);
      for (int q = 0; q < n; ++q) {
        const int st = (int)(j % kStages);
        if (!wait_or_abort(&full[st], (uint32_t)((j / kStages) & 1), &abort_s)) {
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t pa = s0 + st * kStage;
        const uint64_t db = smem_desc(pa + kAGroup, b_group(NT) / 2, 128u);
#pragma unroll
        for (int i = 0; i < kDigits; ++i)
          mma_bf16(tmem + b * Sh::kAccStride + NT * i,
                   smem_desc(pa + i * 2 * (kRows / 8) * 128, (kRows / 8) * 128u, 128u), db,
                   mma_idesc(NT * (kLevels - i)), (q > 0 || i > 0) ? 1u : 0u);
        mma_commit(&empty[st]);
        ++j;
      }
      if (stop) break;
      mma_commit(&acc_full[b]);
      ++k;
      have = ring_next(u, nitems, g);
    }
    // products in flight complete before the tensor memory is released (bounded)
    if (abort_s && j > 0) {
      const long long jl = j - 1;
      if (!mbar_wait(&empty[jl % kStages], (uint32_t)((jl / kStages) & 1))) drain_fail_s = 1;
    }
  } else if (warp < kDrain) {
    constexpr int C = Sh::kCols;
    const int q = warp & 3, col0 = C * (warp >> 2);
    double* out = (double*)(smem + kStages * kStage + warp * Sh::kWarpBytes);   // [32][kOutStride]
    long long* kept = (long long*)(out + 32 * Sh::kOutStride) + lane;           // [type][C][32]: Ce, Co
    const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)col0;
    long long a[C], se[C];   // the type's sums in units of 2^-(52 + xbit) of the ring's scale; Se
    const int m0 = 1 << (6 + xbit), m1 = 1 << (27 + xbit), m2 = 1 << (18 + xbit), m3 = 512 << xbit, m4 = 1 << xbit;
    const float f5 = (float)m4 / 512.f, f6 = (float)m4 / 262144.f;
    long long k = 0;
    while (have) {
      const int rb = u.item / g.ntile, tile = u.item % g.ntile, r = rb * kRows + 32 * q + lane;
      bool ok = true;
#pragma unroll 1
      for (int type = 0; type < 4; ++type) {   // Ce, Co, Se, So
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (type == 1 || type == 2) kept[((type - 1) * C + c) * 32] = a[c];
          if (type == 3) se[c] = a[c];
          a[c] = 0;
        }
        const int n = chunks(g.count(type));
#pragma unroll 1
        for (int ch = 0; ch < n; ++ch) {
          const int sh = r < g.rows ? shift[(int64_t)r * 2 * kMaxChunks + (type & 1) * kMaxChunks + ch] : 0;
          const int b = (int)(k & 1);
          if (!warp_wait(&acc_full[b], (uint32_t)((k >> 1) & 1), &abort_s)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t buf = lanes + (uint32_t)(b * Sh::kAccStride);
          long long h[C];
          float lo[C];
          constexpr int kPer = 32 / C;   // levels per load
#pragma unroll
          for (int s0 = 0; s0 < kLevels; s0 += kPer) {
            float v[32];
            if (C == 16)
              tmem_ld2x16(buf + NT * s0, buf + NT * min(s0 + 1, kLevels - 1), v);
            else
              tmem_ld4x8(buf + NT * s0, buf + NT * (s0 + 1), buf + NT * (s0 + 2), buf + NT * min(s0 + 3, kLevels - 1), v);
#pragma unroll
            for (int w = 0; w < kPer; ++w) {
              const int s = s0 + w;
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const float x = v[w * C + c];
                if (s == 0)
                  h[c] = mad_wide(__float2int_rn(x) * m0, 1 << 30, 0);
                else if (s <= 4)
                  h[c] = mad_wide(__float2int_rn(x), s == 1 ? m1 : (s == 2 ? m2 : (s == 3 ? m3 : m4)), h[c]);
                else if (s == 5)
                  lo[c] = x * f5;
                else if (s == 6)
                  h[c] += __float2int_rn(fmaf(x, f6, lo[c]));
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
          ++k;
          if (sh < 63) {
            const long long round = sh > 0 ? 1LL << (sh - 1) : 0;
#pragma unroll
            for (int c = 0; c < C; ++c) a[c] += (h[c] + round) >> sh;
          }
        }
        if (!ok) break;
      }
      if (!ok) break;
      const int e = r < g.rows ? rexp[r] : 1, p0 = 1 + NT * tile + col0;
      const int scale = e - 1073 - xbit;   // x = (sums) 2^scale
#pragma unroll 1
      for (int im = 0; im < 4; ++im) {   // p, 2L - p, L - p, L + p
        const bool far = im >= 2, plus = im == 1 || im == 2;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const long long ce = kept[c * 32], co = kept[(C + c) * 32];
          const long long cs = far ? ce - co : ce + co, sn = far ? se[c] - a[c] : se[c] + a[c];
          double v = fixed_to_double(plus ? cs + sn : cs - sn, scale);
          if (e == kNonFinite) v = __longlong_as_double(0x7ff8000000000000LL);
          out[lane * Sh::kOutStride + c] = v;
        }
        __syncwarp();
        const int c = lane % C, p = p0 + c;
        const int at = im == 0 ? p : (im == 1 ? 2 * L - p : (im == 2 ? L - p : L + p));
        if (p <= L / 2 && (!far || 2 * p != L)) {
#pragma unroll
          for (int w = 0; w < C; ++w) {
            const int row = (32 / C) * w + lane / C, rr = rb * kRows + 32 * q + row;
            if (rr < g.rows) x[(int64_t)rr * 2 * L + at] = out[row * Sh::kOutStride + c];
          }
        }
        __syncwarp();
      }
      u.item += gridDim.x;
      have = u.item < nitems;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) {   // beside the status, a NaN: the velocity is seen to be unusable
    atomicOr(status, drain_fail_s ? CMM_FLAG_TIMEOUT | CMM_FLAG_DRAIN_TIMEOUT : CMM_FLAG_TIMEOUT);
    x[2 * L] = __longlong_as_double(0x7ff8000000000000LL);
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

RingGeometry geometry(int L, int rows, int nt) {
  return RingGeometry{L, rows, groups16((L + 1) / 2), groups16(L / 2), (L / 2 + nt - 1) / nt};
}

}  // namespace

// Host side ---------------------------------------------------------------
struct RingTables {
  int L = 0, sms = 1, nt = 32;
  const unsigned char* table = nullptr;
};

// Columns per tile: 32 (the data is read half as often) where that gives every
// SM an item, else 16 (twice the items).
static int ring_tile(int L, int fields, int sms) {
  const int64_t blocks = ((int64_t)fields * (L + 1) + kRows - 1) / kRows;
  return blocks * ((L / 2 + 31) / 32) >= sms ? 32 : 16;
}

static int table_bytes(const RingGeometry& g, int nt) { return g.ntile * g.groups() * b_group(nt); }

size_t ring_tables_bytes(int L, int fields) {   // of either tile
  return std::max(table_bytes(geometry(L, fields * (L + 1), 16), 16), table_bytes(geometry(L, fields * (L + 1), 32), 32));
}

template <int NT>
static int ring_tables_nt(const RingGeometry& g, unsigned char* table, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(table, 0, table_bytes(g, NT), s);   // the zero block
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ring_synthesis_digits_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             RingShape<NT>::kSmem);
  if (e != cudaSuccess) return cuda_fail(e, "ring_tables_build");
  ring_table_kernel<NT><<<dim3(g.groups(), g.ntile), 2 * NT, 0, s>>>(g, table);
  return check("ring_table_kernel");
}

int ring_tables_build(int L, int fields, void* mem, std::shared_ptr<RingTables>* out, cudaStream_t s) {
  auto t = std::make_shared<RingTables>();
  t->L = L;
  t->table = (unsigned char*)mem;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&t->sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ring_digits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             8 * (kDigitMaxL + 1) * (int)sizeof(double2));
  if (e != cudaSuccess) return cuda_fail(e, "ring_tables_build");
  t->nt = ring_tile(L, fields, t->sms);
  const RingGeometry g = geometry(L, fields * (L + 1), t->nt);
  const int rc = t->nt == 32 ? ring_tables_nt<32>(g, (unsigned char*)mem, s) : ring_tables_nt<16>(g, (unsigned char*)mem, s);
  if (rc) return rc;
  *out = std::move(t);
  return CMM_OK;
}

// Workspace of a plan: the data digits, then rexp, then shift.  The rows past
// the last ring of its block are never written and have to be finite.
static size_t work_layout(int L, int fields, size_t* rexp_at, size_t* shift_at) {
  const size_t rows = (size_t)fields * (L + 1), blocks = (rows + kRows - 1) / kRows;
  const RingGeometry g = geometry(L, (int)rows, 32);
  *rexp_at = blocks * g.groups() * kAGroup;
  *shift_at = *rexp_at + rows * sizeof(int);
  return *shift_at + rows * 2 * kMaxChunks;
}

size_t ring_work_bytes(int L, int fields) {
  size_t a, b;
  return (work_layout(L, fields, &a, &b) + 255) / 256 * 256;
}

int ring_work_clear(int L, int fields, void* work, cudaStream_t s) {
  size_t a, b;
  work_layout(L, fields, &a, &b);
  const size_t block = (size_t)geometry(L, fields * (L + 1), 32).groups() * kAGroup;   // the last one
  const cudaError_t e = cudaMemsetAsync((unsigned char*)work + a - block, 0, block, s);
  return e == cudaSuccess ? CMM_OK : cuda_fail(e, "cudaMemsetAsync(ring data)");
}

int ring_inverse(const RingTables& t, int fields, const double2* S, void* data, double* x, int* status, cudaStream_t s) {
  const int L = t.L, rows = fields * (L + 1);
  const RingGeometry g = geometry(L, rows, t.nt);
  size_t ra, sa;
  work_layout(L, fields, &ra, &sa);
  unsigned char* d = (unsigned char*)data;
  int* rexp = (int*)(d + ra);
  unsigned char* shift = d + sa;
  ring_digits_kernel<<<(rows + 7) / 8, kDataThreads, 8 * (size_t)((L + 1) | 1) * sizeof(double2), s>>>(g, S, d, rexp,
                                                                                                     shift, x);
  int rc = check("ring_digits_kernel");
  if (rc) return rc;
  const int nitems = (rows + kRows - 1) / kRows * g.ntile, grid = std::min(nitems, t.sms);
  // the sums stay below sqrt(2) L in units of the scale, and 64-bit: one bit
  // more than 52 up to L = 721
  const int xbit = 1.42 * L * 9007199254740992.0 < 9.2e18 ? 1 : 0;
  if (t.nt == 32)
    ring_synthesis_digits_kernel<32><<<grid, kRingThreads, RingShape<32>::kSmem, s>>>(
        g, nitems, xbit, d, rexp, shift, t.table, x, status);
  else
    ring_synthesis_digits_kernel<16><<<grid, kRingThreads, RingShape<16>::kSmem, s>>>(
        g, nitems, xbit, d, rexp, shift, t.table, x, status);
  return check("ring_synthesis_digits_kernel");
}

}  // namespace cmm
