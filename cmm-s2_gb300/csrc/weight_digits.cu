// The analysis weights' contraction over the odd fine rings (sht.cu,
// build_w_kernel) by exact digits on the tensor cores (tcgen05, sm_103a;
// sht_digits.cu describes the scheme): W[m][t][i] = sum_jj Pbar_(m+i)m(odd ring
// jj) Kp[v][jj][t] + we_t Pbar_(m+i)m(ring t).  Set-up work of a table, L^4 / 16
// multiply-adds: FP64-bound (about 10 of the 15 ms that a table took at L =
// 512).  Rows of one order and parity in blocks of 128, tiles of 32 columns,
// chunks of 32 jj, each with a scale per row (m, i) and per column (v, t); the
// chunks' integers are added at the largest scale met.  (Pbar is largest next
// to the poles and Kp next to jj = t: with one scale for all jj the weights of
// low orders erred 2 to 3 times as much as by FP64 sums, so 0.5 to 0.7 times:
// emulated, L = 256 and 512.)
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
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

constexpr int kRows = 128, kNT = 32, kChunk = 2, kStages = 4;
constexpr int kAGroup = kDigits * 2 * 128 * (kRows / 8);   // 16 jj of a row block
constexpr int kBGroup = 2 * kLevels * kNT / 8 * 128;       // 16 jj of a column tile, zero block last
constexpr int kStage = kAGroup + kBGroup;
constexpr int kAccStride = 256;                            // TMEM columns per accumulator (7 x 32 used)
constexpr uint32_t kTmemCols = 512;
constexpr int kAddWarps = 8, kThreads = 32 * (kAddWarps + 2), kCols = kNT / 2;
constexpr int kBatch = 64;                                 // orders whose row digits exist at a time

constexpr int kMaxChunks = kDigitMaxL / 2 / (16 * kChunk);

struct WBlock {
  int m, par, rb;
};

__host__ __device__ __forceinline__ int chunks_of(int G) { return (G + kChunk - 1) / kChunk; }

// Block (tile, v): the column scales, cexp[chunk][v][t], and digits of
// Kp[v][jj][t], t of the tile.
__global__ void __launch_bounds__(256) w_table_kernel(int npo, int npair, int G, const double* __restrict__ Kp,
                                                      unsigned char* __restrict__ out, int* __restrict__ cexp) {
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
  }
}

// Eight rows per block (of row block blockIdx.x / 16): scales, rexp[block][chunk]
// [row], and digits of po[m][i][jj], i = 2 r + par.
__global__ void __launch_bounds__(256) w_rows_kernel(int L, int npo, int G, const WBlock* __restrict__ blocks,
                                                     const double* __restrict__ po, unsigned char* __restrict__ out,
                                                     int* __restrict__ rexp) {
  extern __shared__ double sm[];   // [8][stride]
  __shared__ int es[kMaxChunks][8];
  const int b = blockIdx.x >> 4, rg = blockIdx.x & 15, stride = 16 * G + 2;
  const WBlock w = blocks[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  {
    const int i = 2 * (w.rb * kRows + rg * 8 + warp) + w.par;
    const bool real = i < L - w.m;
    const double* P = po + tab_off(w.m, L, npo) + (int64_t)i * npo;
    static_assert(16 * kChunk == 32, "a chunk is a warp's lanes");
    const int nch = chunks_of(G);
    for (int ch = 0; ch < nch; ++ch) {
      const int k = 32 * ch + lane;
      const double x = real && k < npo ? P[k] : 0.0;
      if (k < 16 * G) sm[warp * stride + k] = x;
      const int e = __reduce_max_sync(0xffffffffu, max(1, (__double2hiint(x) >> 20) & 2047));
      if (lane == 0) es[ch][warp] = rexp[((int64_t)b * nch + ch) * kRows + rg * 8 + warp] = e;
    }
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
__global__ void __launch_bounds__(kThreads, 1) w_product_kernel(int L, int npo, int G, int ntile, int nitems,
                                                                const WBlock* __restrict__ blocks,
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
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, npair = L / 2 + 1;
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
      const int b = item / ntile, tile = item % ntile, v = 2 * (blocks[b].m & 1) + blocks[b].par;
      const unsigned char* A = rows + (int64_t)b * G * kAGroup;
      const unsigned char* B = table + ((int64_t)v * ntile + tile) * G * kBGroup;
      for (int q = 0; q < G; ++q, ++j) {
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
      for (int q = 0; q < G; ++q, ++j) {
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
      const int b = item / ntile, tile = item % ntile;
      const WBlock wb = blocks[b];
      const int r = 32 * q + lane, i = 2 * (wb.rb * kRows + r) + wb.par, nl = L - wb.m;
      const int v = 2 * (wb.m & 1) + wb.par;
      long long a[kCols];   // in units of 2^53 2^(ex - 2150), below 2^62: 16 chunks of 2^58
      int ex[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        a[c] = 0;
        ex[c] = 0;
      }
#pragma unroll 1
      for (int ch = 0; ch < nch; ++ch, ++k) {
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
        float lo[kCols];
#pragma unroll
        for (int s0 = 0; s0 < kLevels; s0 += 2) {
          float x[32];
          tmem_ld2x16(at + kNT * s0, at + kNT * min(s0 + 1, kLevels - 1), x);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int s = s0 + u;
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
              const float y = x[u * 16 + c];
              if (s <= 3)
                h[c] = mad_wide(__float2int_rn(y), s == 0 ? 1 << 27 : (s == 1 ? 1 << 18 : (s == 2 ? 512 : 1)), s ? h[c] : 0);
              else if (s == 4)
                h[c] = mad_wide(__float2int_rn(y), 2, h[c] * 1024);
              else if (s == 5)
                lo[c] = y * (2.f / 512.f);
              else if (s == 6)
                h[c] += __float2int_rn(fmaf(y, 2.f / 262144.f, lo[c]));
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[buf])) : "memory");
#pragma unroll
        for (int c = 0; c < kCols; ++c) {   // at the larger of the two scales, rounded
          const int e = re + ce[c], up = min(max(e - ex[c], 0), 62), dn = min(max(ex[c] - e, 0), 62);
          a[c] = ((a[c] + ((1LL << up) >> 1)) >> up) + ((h[c] + ((1LL << dn) >> 1)) >> dn);
          ex[c] = max(ex[c], e);
        }
      }
      if (!ok || i >= nl) continue;
      const int64_t off = tab_off(wb.m, L, npair);
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int t = tile * kNT + col0 + c;
        if (t < npair)
          W[off + (int64_t)t * nl + i] =
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

int digit_weights(int L, const double* po, const double* ps, const double* Kp, const double* w, double* W,
                  cudaStream_t s) {
  const int npo = (L + 1) / 2, npair = L / 2 + 1, G = groups16(npo), ntile = (npair + kNT - 1) / kNT;
  std::vector<WBlock> blocks;
  std::vector<int> first;   // of each batch of orders
  size_t most = 0;
  for (int m = 0; m < L; ++m) {
    if (m % kBatch == 0) first.push_back((int)blocks.size());
    for (int par = 0; par < 2; ++par)
      for (int rb = 0; 2 * rb * kRows + par < L - m; ++rb) blocks.push_back(WBlock{m, par, rb});
  }
  first.push_back((int)blocks.size());
  for (size_t b = 0; b + 1 < first.size(); ++b) most = std::max(most, (size_t)(first[b + 1] - first[b]));
  DeviceBuffer db, rows, rexp, table, cexp, fail;
  int rc, dev = 0, sms = 1, failed = 0;
  if ((rc = db.upload(blocks.data(), blocks.size() * sizeof(WBlock))) ||
      (rc = rows.alloc(most * G * kAGroup)) || (rc = rexp.alloc(most * chunks_of(G) * kRows * sizeof(int))) ||
      (rc = table.alloc((size_t)4 * ntile * G * kBGroup)) ||
      (rc = cexp.alloc((size_t)4 * chunks_of(G) * ntile * kNT * sizeof(int))) ||
      (rc = fail.upload(&failed, sizeof(int))))
    return rc;
  cudaError_t e = cudaStreamSynchronize(0);   // the uploads, before s reads them
  if (e == cudaSuccess) e = cudaMemsetAsync(table.p, 0, table.bytes, s);   // the zero blocks
  const size_t row_smem = (size_t)8 * (16 * G + 2) * sizeof(double);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(w_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kStage);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_fail(e, "digit_weights");
  w_table_kernel<<<dim3(ntile, 4), 256, 0, s>>>(npo, npair, G, Kp, (unsigned char*)table.p, (int*)cexp.p);
  if ((rc = check("w_table_kernel"))) return rc;
  for (size_t b = 0; b + 1 < first.size(); ++b) {
    const int n = first[b + 1] - first[b], nitems = n * ntile;
    const WBlock* bl = (const WBlock*)db.p + first[b];
    w_rows_kernel<<<n * 16, 256, row_smem, s>>>(L, npo, G, bl, po, (unsigned char*)rows.p, (int*)rexp.p);
    if ((rc = check("w_rows_kernel"))) return rc;
    w_product_kernel<<<std::min(nitems, sms), kThreads, kStages * kStage, s>>>(
        L, npo, G, ntile, nitems, bl, (const unsigned char*)rows.p, (const int*)rexp.p,
        (const unsigned char*)table.p, (const int*)cexp.p, ps, w, 3.141592653589793 / L, W,
        (int*)fail.p);
    if ((rc = check("w_product_kernel"))) return rc;
  }
  e = cudaMemcpyAsync(&failed, fail.p, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "w_product_kernel");
  if (failed) {
    set_last_error("analysis weights: a bounded wait inside the kernel ran out");
    return CMM_ERR_TIMEOUT;
  }
  return CMM_OK;
}

}  // namespace cmm
