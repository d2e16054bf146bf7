// The analysis weights' contraction over the odd fine rings by exact digits on
// the tensor cores (tcgen05, sm_103a; sht_digits.cu describes the scheme):
// W[m][t][i] = sum_jj Pbar_(m+i)m(odd ring jj) Kp[v][jj][t] + we_t
// Pbar_(m+i)m(ring t).  Set-up work of a table, L^4 / 16 multiply-adds.  Kp
// depends on the parities v of m and i alone, so that the rows (m, i) of a class
// v follow each other, order after order, in blocks of 128; tiles of 32
// columns, chunks of 32 jj, each with a scale per row and per column; the
// chunks' integers are added at the largest scale met.  (Pbar is largest next
// to the poles and Kp next to jj = t: with one scale for all jj the weights of
// low orders erred 2 to 3 times as much as by FP64 sums, so 0.5 to 0.7 times:
// emulated, L = 256 and 512.)  Towards the poles Pbar falls off exponentially:
// a block leaves out the leading chunks in which all its rows are below 1e-30.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>

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

constexpr int kRows = 128, kNT = 32, kChunk = 2, kStages = 4;
constexpr int kAGroup = kDigits * 2 * 128 * (kRows / 8);   // 16 jj of a row block
constexpr int kBGroup = 2 * kLevels * kNT / 8 * 128;       // 16 jj of a column tile, zero block last
constexpr int kStage = kAGroup + kBGroup;
constexpr int kAccStride = 256;                            // TMEM columns per accumulator (7 x 32 used)
constexpr uint32_t kTmemCols = 512;
constexpr int kAddWarps = 16, kThreads = 32 * (kAddWarps + 2), kCols = kNT / (kAddWarps / 4);
constexpr int kBatch = 288;                                // most row blocks whose digits exist at a time
constexpr int kMaxChunks = kDigitMaxL / 2 / (16 * kChunk);
constexpr int kTiny = 1023 - 100;                          // biased exponent of about 1e-30

__host__ __device__ __forceinline__ int chunks_of(int G) { return (G + kChunk - 1) / kChunk; }

// The classes v = 2 (m odd) + (i odd): order m = 2 k + (v >> 1) has N - k rows,
// i = (v & 1), (v & 1) + 2, ...
struct WGeometry {
  int L, first[5];   // first row block of each class, and the total
  __host__ __device__ int N(int v) const { return (L - (v >> 1) - (v & 1) + 1) / 2; }
  __host__ __device__ int rows(int v) const { return N(v) * (N(v) + 1) / 2; }
  __device__ __forceinline__ int cls(int b) const { return (b >= first[1]) + (b >= first[2]) + (b >= first[3]); }
  // row r of class v
  __device__ __forceinline__ void row(int v, int r, int& m, int& i) const {
    const int n = N(v);
    const float h = n + 0.5f;
    int k = min(n - 1, (int)(h - sqrtf(fmaxf(h * h - 2.f * r, 0.f))));
    auto start = [&](int q) { return q * n - q * (q - 1) / 2; };
    while (k > 0 && start(k) > r) --k;
    while (start(k + 1) <= r) ++k;
    m = 2 * k + (v >> 1);
    i = 2 * (r - start(k)) + (v & 1);
  }
};

// Block (tile, v): the column scales, cexp[chunk][v][t], and digits of
// Kp[v][jj][t], t of the tile, with the zero block.  Also clears the blocks'
// first chunks (nlead of them) and *fail.
__global__ void __launch_bounds__(256) w_table_kernel(int npo, int npair, int G, const double* __restrict__ Kp,
                                                      unsigned char* __restrict__ out, int* __restrict__ cexp,
                                                      int* __restrict__ lead, int nlead, int* __restrict__ fail) {
  for (int k = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + threadIdx.x; k < nlead; k += 256 * gridDim.x * gridDim.y)
    lead[k] = 1 << 30;
  if (blockIdx.x + blockIdx.y + threadIdx.x == 0) *fail = 0;
  __shared__ int emax[kMaxChunks][kNT];
  const int tile = blockIdx.x, v = blockIdx.y, c = threadIdx.x % kNT, t = tile * kNT + c, ntile = gridDim.x;
  const double* K = Kp + (int64_t)v * npo * npair + t;
  const int nch = chunks_of(G);
  for (int ch = threadIdx.x / kNT; ch < nch; ch += 256 / kNT) {
    int e = 1;
    if (t < npair)
      for (int k = 16 * kChunk * ch; k < min(npo, 16 * kChunk * (ch + 1)); ++k)
        e = max(e, (__double2hiint(K[(int64_t)k * npair]) >> 20) & 2047);
    emax[ch][c] = cexp[(ch * 4 + v) * ntile * kNT + t] = e;
  }
  __syncthreads();
  unsigned char* base = out + ((int64_t)v * ntile + tile) * G * kBGroup + (c >> 3) * 128 + (c & 7) * 16;
  for (int q = threadIdx.x / kNT; q < 2 * G; q += 256 / kNT) {
    const int e = emax[q / (2 * kChunk)][c];
    long long x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = 8 * q + u;
      x[u] = t < npair && k < npo ? to_fixed(K[(int64_t)k * npair], e) : 0;
    }
    uint4 d[kDigits];
    digits8(x, d);
    unsigned char* o = base + (int64_t)(q >> 1) * kBGroup + (q & 1) * (kBGroup / 2);
#pragma unroll
    for (int j = 0; j < kDigits; ++j) *(uint4*)(o + j * (kNT / 8) * 128) = d[j];
    *(uint4*)(o + kDigits * (kNT / 8) * 128) = make_uint4(0, 0, 0, 0);
  }
}

// Eight rows per block (of row block b0 + blockIdx.x / 16): scales, rexp[block]
// [chunk][row], digits of po[m][i][jj] and the row block's first chunk.
__global__ void __launch_bounds__(256) w_rows_kernel(WGeometry g, int npo, int G, int b0, const double* __restrict__ po,
                                                     unsigned char* __restrict__ out, int* __restrict__ rexp,
                                                     int* __restrict__ first) {
  extern __shared__ double sm[];   // [8][stride]
  __shared__ int es[kMaxChunks][8];
  const int b = blockIdx.x >> 4, rg = blockIdx.x & 15, stride = 16 * G + 2, nch = chunks_of(G);
  const int v = g.cls(b0 + b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  {
    const int r = (b0 + b - g.first[v]) * kRows + rg * 8 + warp;
    const bool real = r < g.rows(v);
    int m = 0, i = 0;
    if (real) g.row(v, r, m, i);
    const double* P = po + tab_off(m, g.L, npo) + (int64_t)i * npo;
    static_assert(16 * kChunk == 32, "a chunk is a warp's lanes");
    int lead = nch - 1;
    for (int ch = 0; ch < nch; ++ch) {
      const int k = 32 * ch + lane;
      const double x = real && k < npo ? P[k] : 0.0;
      if (k < 16 * G) sm[warp * stride + k] = x;
      const int e = __reduce_max_sync(0xffffffffu, max(1, (__double2hiint(x) >> 20) & 2047));
      if (e >= kTiny) lead = min(lead, ch);
      if (lane == 0) es[ch][warp] = rexp[((int64_t)b * nch + ch) * kRows + rg * 8 + warp] = e;
    }
    if (real && lane == 0) atomicMin(first + b, lead);
  }
  __syncthreads();
  const int row = threadIdx.x & 7;
  unsigned char* base = out + (int64_t)b * G * kAGroup + rg * 128 + row * 16;
  for (int q = threadIdx.x >> 3; q < 2 * G; q += 32) {
    const int e = es[q / (2 * kChunk)][row];
    long long x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = to_fixed(sm[row * stride + 8 * q + u], e);
    uint4 d[kDigits];
    digits8(x, d);
    unsigned char* o = base + (int64_t)(q >> 1) * kAGroup + (q & 1) * (kRows / 8) * 128;
#pragma unroll
    for (int j = 0; j < kDigits; ++j) *(uint4*)(o + j * 2 * (kRows / 8) * 128) = d[j];
  }
}

// Persistent over the items (row block, column tile); roles as in
// ring_synthesis_digits_kernel, one sum per output.
__global__ void __launch_bounds__(kThreads, 1) w_product_kernel(WGeometry g, int npo, int G, int ntile, int nitems,
                                                                int b0, const int* __restrict__ lead,
                                                                const unsigned char* __restrict__ rows,
                                                                const int* __restrict__ rexp,
                                                                const unsigned char* __restrict__ table,
                                                                const int* __restrict__ cexp,
                                                                const double* __restrict__ ps,
                                                                const double* __restrict__ w, double pi_L,
                                                                double* __restrict__ W, int* __restrict__ fail) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, L = g.L, npair = L / 2 + 1;
  const int nch = chunks_of(G);
  if (tid == 0) {
    for (int b = 0; b < kStages; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kAddWarps);
    }
    abort_s = 0;
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
  if (warp == kAddWarps && lane == 0) {
    long long j = 0;   // groups
    for (int item = blockIdx.x; item < nitems && !abort_s; item += gridDim.x) {
      const int b = item / ntile, tile = item % ntile, v = g.cls(b0 + b);
      const unsigned char* A = rows + (int64_t)b * G * kAGroup;
      const unsigned char* B = table + ((int64_t)v * ntile + tile) * G * kBGroup;
      for (int q = kChunk * lead[b]; q < G; ++q, ++j) {
        const int st = (int)(j % kStages);
        if (j >= kStages && !wait_or_abort(&empty[st], (uint32_t)((j / kStages - 1) & 1), &abort_s)) break;
        unsigned char* d = smem + st * kStage;
        mbar_expect_tx(&full[st], (uint32_t)kStage);
        bulk_g2s(d, A + (int64_t)q * kAGroup, (uint32_t)kAGroup, &full[st]);
        bulk_g2s(d + kAGroup, B + (int64_t)q * kBGroup, (uint32_t)kBGroup, &full[st]);
      }
    }
    // copies still in flight land before the block exits (bounded)
    if (abort_s)
      for (long long k = (j > kStages ? j - kStages : 0); k < j; ++k)
        mbar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1));
  } else if (warp == kAddWarps + 1 && lane == 0) {
    const uint32_t s0 = smem_u32(smem);
    long long j = 0, k = 0;   // groups, chunks
    for (int item = blockIdx.x; item < nitems && !abort_s; item += gridDim.x)
      for (int q = kChunk * lead[item / ntile]; q < G; ++q, ++j) {
        const int b = (int)(k & 1), st = (int)(j % kStages), in_chunk = q % kChunk;
        if (in_chunk == 0 && k >= 2 && !wait_or_abort(&acc_empty[b], (uint32_t)(((k >> 1) - 1) & 1), &abort_s)) break;
        if (!wait_or_abort(&full[st], (uint32_t)((j / kStages) & 1), &abort_s)) break;
        tc_fence_after();
        const uint32_t pa = s0 + st * kStage;
        const uint64_t db = smem_desc(pa + kAGroup, kBGroup / 2, 128u);
#pragma unroll
        for (int i = 0; i < kDigits; ++i)
          mma_bf16(tmem + b * kAccStride + kNT * i, smem_desc(pa + i * 2 * (kRows / 8) * 128, (kRows / 8) * 128u, 128u),
                   db, mma_idesc(kNT * (kLevels - i)), (in_chunk > 0 || i > 0) ? 1u : 0u);
        mma_commit(&empty[st]);
        if (in_chunk == kChunk - 1 || q == G - 1) {
          mma_commit(&acc_full[b]);
          ++k;
        }
      }
    // products in flight complete before the tensor memory is released (bounded)
    if (abort_s && j > 0) mbar_wait(&empty[(j - 1) % kStages], (uint32_t)(((j - 1) / kStages) & 1));
  } else if (warp < kAddWarps) {
    const int q = warp & 3, col0 = kCols * (warp >> 2);
    const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)col0;
    long long k = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
      const int b = item / ntile, tile = item % ntile, v = g.cls(b0 + b);
      const int r = 32 * q + lane, rc = (b0 + b - g.first[v]) * kRows + r;   // row of the block, of the class
      long long a[kCols];   // in units of 2^53 2^(ex - 2150), below 2^62: 16 chunks of 2^58
      int ex[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        a[c] = 0;
        ex[c] = 0;
      }
#pragma unroll 1
      for (int ch = lead[b]; ch < nch; ++ch, ++k) {
        const int buf = (int)(k & 1);
        const int re = rexp[((int64_t)b * nch + ch) * kRows + r];
        int ce[kCols];
#pragma unroll
        for (int c = 0; c < kCols; c += 4) *(int4*)(ce + c) = *(const int4*)(cexp + ((ch * 4 + v) * ntile + tile) * kNT + col0 + c);
        if (!warp_wait(&acc_full[buf], (uint32_t)((k >> 1) & 1), &abort_s)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t at = lanes + (uint32_t)(buf * kAccStride);
        long long h[kCols];   // the chunk's products in units of 2^53
        float x[32];
        tmem_ld4x8(at, at + kNT, at + 2 * kNT, at + 3 * kNT, x);
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          h[c] = mad_wide(__float2int_rn(x[c]), 1 << 27, 0);   // 512^3; 512 and 2 to come
          h[c] = mad_wide(__float2int_rn(x[8 + c]), 1 << 18, h[c]);
          h[c] = mad_wide(__float2int_rn(x[16 + c]), 512, h[c]) + __float2int_rn(x[24 + c]);
        }
        tmem_ld4x8(at + 4 * kNT, at + 5 * kNT, at + 6 * kNT, at + 6 * kNT, x);
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          h[c] = mad_wide(__float2int_rn(x[c]), 2, h[c] * 1024) +
                 __float2int_rn(fmaf(x[16 + c], 2.f / 262144.f, x[8 + c] * (2.f / 512.f)));
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[buf])) : "memory");
        // at the larger of the two scales, rounded
        bool up = false;
#pragma unroll
        for (int c = 0; c < kCols; ++c) up = up || re + ce[c] > ex[c];
        if (__any_sync(0xffffffffu, up)) {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            const int d = min(max(re + ce[c] - ex[c], 0), 62);
            a[c] = (a[c] + ((1LL << d) >> 1)) >> d;
            ex[c] = max(ex[c], re + ce[c]);
          }
        }
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int d = min(ex[c] - re - ce[c], 62);
          a[c] += (h[c] + ((1LL << d) >> 1)) >> d;
        }
      }
      if (!ok || rc >= g.rows(v)) continue;
      int m, i;
      g.row(v, rc, m, i);
      const int64_t off = tab_off(m, L, npair);
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int t = tile * kNT + col0 + c;
        if (t < npair)
          W[off + (int64_t)t * (L - m) + i] =
              fixed_to_double(a[c], ex[c] - 2097) + pi_L * w[2 * t] * ps[off + (int64_t)i * npair + t];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) atomicExch(fail, 1);
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

static WGeometry w_geometry(int L) {
  WGeometry g{L, {0}};
  for (int v = 0; v < 4; ++v) g.first[v + 1] = g.first[v] + (g.rows(v) + kRows - 1) / kRows;
  return g;
}

// Scratch: the row digits of a batch, the table, the scales, the first chunks.
struct WScratch {
  size_t rows, table, rexp, cexp, first, total;
  WScratch(const WGeometry& g, int G, int ntile) {
    const size_t nb = std::min(kBatch, g.first[4]);
    auto next = [&](size_t n) {
      const size_t at = total;
      total += (n + 255) / 256 * 256;
      return at;
    };
    total = 0;
    rows = next(nb * G * kAGroup);
    table = next((size_t)4 * ntile * G * kBGroup);
    rexp = next(nb * chunks_of(G) * kRows * sizeof(int));
    cexp = next((size_t)4 * chunks_of(G) * ntile * kNT * sizeof(int));
    first = next((size_t)g.first[4] * sizeof(int));
  }
};

size_t digit_weights_bytes(int L) {
  return WScratch(w_geometry(L), groups16((L + 1) / 2), (L / 2 + kNT) / kNT).total;
}

int digit_weights(int L, const double* po, const double* ps, const double* Kp, const double* w, double* W,
                  void* scratch, int* fail, cudaStream_t s) {
  const int npo = (L + 1) / 2, npair = L / 2 + 1, G = groups16(npo), ntile = (npair + kNT - 1) / kNT;
  const WGeometry g = w_geometry(L);
  const WScratch at(g, G, ntile);
  unsigned char* mem = (unsigned char*)scratch;
  int *rexp = (int*)(mem + at.rexp), *cexp = (int*)(mem + at.cexp), *first = (int*)(mem + at.first);
  int dev = 0, sms = 1, rc;
  cudaError_t e =
      cudaFuncSetAttribute(w_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kStage);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "digit_weights");
  w_table_kernel<<<dim3(ntile, 4), 256, 0, s>>>(npo, npair, G, Kp, mem + at.table, cexp, first, g.first[4], fail);
  if ((rc = check("w_table_kernel"))) return rc;
  const int nbatch = (g.first[4] + kBatch - 1) / kBatch, batch = (g.first[4] + nbatch - 1) / nbatch;
  for (int b = 0; b < g.first[4]; b += batch) {
    const int n = std::min(batch, g.first[4] - b), nitems = n * ntile;
    w_rows_kernel<<<n * 16, 256, (size_t)8 * (16 * G + 2) * sizeof(double), s>>>(g, npo, G, b, po, mem + at.rows, rexp,
                                                                                first + b);
    if ((rc = check("w_rows_kernel"))) return rc;
    w_product_kernel<<<std::min(nitems, sms), kThreads, kStages * kStage, s>>>(
        g, npo, G, ntile, nitems, b, first + b, mem + at.rows, rexp, mem + at.table, cexp, ps, w, 3.141592653589793 / L, W,
        fail);
    if ((rc = check("w_product_kernel"))) return rc;
  }
  return CMM_OK;
}

}  // namespace cmm
