// Point location, Powell-Sabin assembly, map evaluation and composition
// kernels for the icosahedral mesh (sm_103a).
//
// Location: a query descends the icosahedral refinement hierarchy.  At each
// node three great-circle tests (the planes through the edge midpoints)
// choose one of the four children.  Tests run in FP32 against unit normals
// and are redone in FP64 only when |n.q| < kFilter, inside which the FP32
// sign is not guaranteed (|q| = |n| = 1: the FP32 dot is within ~6e-7 of
// the exact dot of the FP64 inputs).  The FP64 decision equals the
// reference's Qhull choice except for queries within rounding distance of
// an edge, where either neighbour contains the query.
//
// Evaluation: with bcc = Minv q (precomputed inverse vertex matrix per
// triangle) the Powell-Sabin sub-triangle is picked by argmin/argmax of the
// bcc with numpy's first-index tie rule (cmm_s2/core/spherical_spline.py:
// 691-697); the sub-triangle barycentrics follow in closed form from the
// triangle's, since its corners are v_hi, (v_hi+v_mid)/|v_hi+v_mid| and
// (v1+v2+v3)/|v1+v2+v3|:
//     gV = b_hi - b_mid,  gE = |v_hi+v_mid| (b_mid - b_lo),  gC = |v1+v2+v3| b_lo
// which is the same linear map the reference obtains from four 3x3
// determinants (new_vpoints + bary_coords, :668-689).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "cmm_internal.h"
#include "dd.cuh"
#include "device_common.cuh"
#include "ff.cuh"
#include "fixed.cuh"

namespace cmm {

using namespace dev;

namespace {

constexpr int kBlock = 256;
// The composition through coefficient records normalises the point every
// kNormEvery submaps (a power of two); queries whose FP32 squared norm is
// outside [1/4, 4] are normalised first, so the unnormalised chain stays far
// from overflow.
constexpr int kNormEvery = 8;
// default register budgets of the compositions through records, as resident
// 256-thread blocks per SM; the autotuner may set others
constexpr int kComposeJacBlocks = 4;
constexpr int kComposeBlocks = 4;
constexpr int64_t kBlockWave = (int64_t)kBlock * kNumSMs;   // queries of one block per SM
constexpr int64_t kL2Bytes = 129LL << 20;
// Submaps listed in the kernel parameters of the usual calls (768 bytes);
// longer lists take the 24 KB form, whose upload alone costs microseconds.
constexpr int kShortList = 32;

// Submap lists: by value in the kernel parameters (host calls), or a
// device table whose length comes from a device-driven step's state.
// Each submap has its coefficient record and, optionally, its map-form
// record (form(s) != NULL: evaluated as quadratic forms).
// A submap with a form record may also have the low floats of its
// float-float split (the Jacobian pushes then load them instead of
// extracting them from the doubles on the integer pipe).
template <int N>
struct SubmapPtrs {
  const double* p[N];
  const double* f[N];
  const float* g[N];
  int S;
  __device__ __forceinline__ int count() const { return S; }
  __device__ __forceinline__ const double* at(int s, int) const { return p[s]; }
  __device__ __forceinline__ const double* form(int s, int) const { return f[s]; }
  __device__ __forceinline__ const float* form_ff(int s, int) const { return g[s]; }
};
struct DevSubmaps {
  const double* const* tab;
  const double* const* ftab;   // forms of the stack slots, or NULL
  const BveState* st;
  const double* last;
  __device__ __forceinline__ int count() const { return st->nc + 1; }
  __device__ __forceinline__ const double* at(int s, int S) const { return s < S - 1 ? tab[s] : last; }
  __device__ __forceinline__ const double* form(int s, int S) const {
    return ftab && s < S - 1 ? ftab[s] : nullptr;
  }
  __device__ __forceinline__ const float* form_ff(int, int) const { return nullptr; }
};

// Orthonormal tangent basis (t1, t2) at the unit point p, in float-float
// from the FP64 point (the Jacobian's tangent pushes run in float-float on
// the FP32 pipe).
__device__ __forceinline__ void tangent_basis_ff(const double* p, ff* t1, ff* t2) {
  const ff p0 = ff_of(p[0]), p1 = ff_of(p[1]), p2 = ff_of(p[2]);
  const bool polar = !(fabsf(p2.h) < 0.9f);
  // t1 = e x p normalised, e = z (or x near the poles): (p1, -p0, 0) or (0, p2, -p1)
  const ff a = polar ? p2 : p1, b = polar ? ff_neg(p1) : ff_neg(p0);
  const ff r = ff_rsqrt(ff_dot2(a, a, b, b));
  const ff ua = ff_mul(a, r), ub = ff_mul(b, r);
  const ff z{0.f, 0.f};
  t1[0] = polar ? z : ua;
  t1[1] = polar ? ua : ub;
  t1[2] = polar ? ub : z;
  // t2 = p x t1
  t2[0] = ff_sub(ff_mul(p1, t1[2]), ff_mul(p2, t1[1]));
  t2[1] = ff_sub(ff_mul(p2, t1[0]), ff_mul(p0, t1[2]));
  t2[2] = ff_sub(ff_mul(p0, t1[1]), ff_mul(p1, t1[0]));
}

__device__ __forceinline__ ff pick_ff(const ff* b, int i) { return i == 0 ? b[0] : (i == 1 ? b[1] : b[2]); }

// Twelve float-float values of one thread in shared memory, value-major
// (value k at s[2k * stride], s[(2k + 1) * stride]: conflict-free): the two
// tangent pushes (0..5) and their barycentric directions (6..11).
struct Pushes {
  float* s;
  int stride;
  __device__ __forceinline__ ff get(int k) const { return ff{s[2 * k * stride], s[(2 * k + 1) * stride]}; }
  __device__ __forceinline__ void set(int k, ff v) {
    s[2 * k * stride] = v.h;
    s[(2 * k + 1) * stride] = v.l;
  }
};

// 2^m as a double, from its bit pattern
__device__ __forceinline__ double pow2(int m) { return __longlong_as_double((long long)(1023 + m) << 52); }

__global__ void __launch_bounds__(kBlock) locate_kernel(MeshView m, const double* __restrict__ q,
                                                        int64_t n, int32_t* __restrict__ tri,
                                                        double* __restrict__ bcc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double x = q[3 * i], y = q[3 * i + 1], z = q[3 * i + 2];
    if (!finite3(x, y, z)) {
      flag(m, CMM_FLAG_NONFINITE);
      tri[i] = -1;
      if (bcc) bcc[3 * i] = bcc[3 * i + 1] = bcc[3 * i + 2] = nan("");
      continue;
    }
    int t = locate_row(m, x, y, z);
    tri[i] = t;
    if (bcc) {
      Bcc b = bcc_of(m.tri_loc + (int64_t)t * kLocStride, x, y, z);
      bcc[3 * i] = b.b0;
      bcc[3 * i + 1] = b.b1;
      bcc[3 * i + 2] = b.b2;
      if (fmin(b.b0, fmin(b.b1, b.b2)) < -1e-10) flag(m, CMM_FLAG_LOCATE);
    }
  }
}

// The 19 ordinates of each component from the jets of a triangle's three
// vertices (assemble_coefficients, cmm_s2/core/spherical_spline.py:300-337)
// using the per-triangle factors (factor-major, coalesced loads).  Three
// threads per triangle: first one per corner (its value and its three
// ordinates, for all components), then one per component (the inner ordinates
// from the corners').  The block's records are staged in shared memory (rows
// padded to stride+1 doubles against bank conflicts) and written out as one
// contiguous, coalesced range, record padding included (zeros).  FP64-bound
// (153 per triangle); one thread per triangle held 166 registers and left
// four warps per SM at level 5 (17 us; level 6: 38 us).
constexpr int kAsmTri = 64;   // triangles per block

template <int NC>
__global__ void __launch_bounds__(3 * kAsmTri) assemble_kernel(MeshView m, const double* __restrict__ jets,
                                                               double* __restrict__ coeffs,
                                                               const BveState* __restrict__ st) {
  if (st) coeffs = st->vel[0];
  constexpr int kStride = NC == 3 ? kCoeffStride3 : kCoeffStride1;
  constexpr int kRow = kStride + 1;
  __shared__ double rec[kAsmTri * kRow];
  const int t0 = blockIdx.x * kAsmTri;
  const int nblk = min(kAsmTri, m.nt - t0);
  const int tl = threadIdx.x % kAsmTri, part = threadIdx.x / kAsmTri, t = t0 + tl;   // part: corner, then component
  double* out = rec + tl * kRow;
  const int nv = m.nv, nt = m.nt;
  const double* A = m.tri_asm + t;   // factor j at A[j * nt]
  if (tl < nblk) {
    const int4 tv = m.tri_v[t];
    const int v = part == 0 ? tv.x : (part == 1 ? tv.y : tv.z);
    double a[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[i][j] = __ldg(A + (int64_t)(4 * (3 * part + i) + j) * nt);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const double f = __ldg(jets + (int64_t)(k * 4) * nv + v);
      // d_j f_k = jets[j][1+k] (three components), jets[1+j] (scalar)
      const int g0 = NC == 3 ? 1 + k : 1, dg = NC == 3 ? 4 : 1;
      const double gx = __ldg(jets + (int64_t)g0 * nv + v), gy = __ldg(jets + (int64_t)(g0 + dg) * nv + v),
                   gz = __ldg(jets + (int64_t)(g0 + 2 * dg) * nv + v);
      out[NC * part + k] = f;
#pragma unroll
      for (int i = 0; i < 3; ++i)
        out[NC * (3 + 3 * part + i) + k] = a[i][0] * gx + a[i][1] * gy + a[i][2] * gz - a[i][3] * f;
    }
    for (int j = 19 * NC + part; j < kStride; j += 3) out[j] = 0.0;
  }
  __syncthreads();
  if (tl < nblk && part < NC) {
    double e[9], c[12];
#pragma unroll
    for (int j = 0; j < 9; ++j) e[j] = __ldg(A + (int64_t)(36 + j) * nt);
#pragma unroll
    for (int o = 3; o < 12; ++o) c[o] = out[NC * o + part];
    out[NC * 12 + part] = e[0] * c[3] + e[1] * c[8];
    out[NC * 13 + part] = e[2] * c[6] + e[3] * c[11];
    out[NC * 14 + part] = e[5] * c[9] + e[4] * c[5];
    out[NC * 15 + part] = e[0] * c[4] + e[1] * c[7];
    out[NC * 16 + part] = e[2] * c[7] + e[3] * c[10];
    out[NC * 17 + part] = e[4] * c[4] + e[5] * c[10];
    out[NC * 18 + part] = e[6] * c[4] + e[7] * c[7] + e[8] * c[10];
  }
  __syncthreads();
  double* dst = coeffs + (int64_t)t0 * kStride;
  for (int i = threadIdx.x; i < nblk * kStride; i += 3 * kAsmTri) dst[i] = rec[(i / kStride) * kRow + i % kStride];
}

// FP32 velocity records (velmesh with rec32, ncomp = 3): the same
// ordinates from FP32 jets and the FP32 factor table, in FP32.  J: the
// jets' storage type (double jets are rounded to float here; float jets
// are the split form's FP32 jets, the same values without conversions).
template <typename J>
__global__ void __launch_bounds__(kAsmTri) assemble_f32_kernel(MeshView m, const J* __restrict__ jets,
                                                               float* __restrict__ coeffs,
                                                               const BveState* __restrict__ st) {
  if (st) coeffs = (float*)st->vel[0];
  constexpr int kStride = kCoeffStride3;
  constexpr int kRow = kStride + 1;
  __shared__ float rec[kAsmTri * kRow];
  const int t0 = blockIdx.x * kAsmTri;
  const int nblk = min(kAsmTri, m.nt - t0);
  const int tl = threadIdx.x, t = t0 + tl;
  float* out = rec + tl * kRow;
  if (tl < nblk) {
    const int nv = m.nv, nt = m.nt;
    const int4 tv = m.tri_v[t];
    const int vid[3] = {tv.x, tv.y, tv.z};
    const float* A = m.tri_asm_f + t;
    const int corner[9] = {0, 0, 0, 1, 1, 1, 2, 2, 2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float f[3], c[19];
#pragma unroll
      for (int v = 0; v < 3; ++v) f[v] = (float)__ldg(jets + (int64_t)(k * 4) * nv + vid[v]);
      c[0] = f[0];
      c[1] = f[1];
      c[2] = f[2];
#pragma unroll
      for (int o = 0; o < 9; ++o) {
        const int v = vid[corner[o]];
        const float gx = (float)__ldg(jets + (int64_t)(0 * 4 + 1 + k) * nv + v);
        const float gy = (float)__ldg(jets + (int64_t)(1 * 4 + 1 + k) * nv + v);
        const float gz = (float)__ldg(jets + (int64_t)(2 * 4 + 1 + k) * nv + v);
        c[3 + o] = __ldg(A + (int64_t)(4 * o) * nt) * gx + __ldg(A + (int64_t)(4 * o + 1) * nt) * gy +
                   __ldg(A + (int64_t)(4 * o + 2) * nt) * gz - __ldg(A + (int64_t)(4 * o + 3) * nt) * f[corner[o]];
      }
      float e[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) e[j] = __ldg(A + (int64_t)(36 + j) * nt);
      c[12] = e[0] * c[3] + e[1] * c[8];
      c[13] = e[2] * c[6] + e[3] * c[11];
      c[14] = e[5] * c[9] + e[4] * c[5];
      c[15] = e[0] * c[4] + e[1] * c[7];
      c[16] = e[2] * c[7] + e[3] * c[10];
      c[17] = e[4] * c[4] + e[5] * c[10];
      c[18] = e[6] * c[4] + e[7] * c[7] + e[8] * c[10];
#pragma unroll
      for (int o = 0; o < 19; ++o) out[3 * o + k] = c[o];
    }
#pragma unroll
    for (int j = 57; j < kStride; ++j) out[j] = 0.f;
  }
  __syncthreads();
  float* dst = coeffs + (int64_t)t0 * kStride;
  for (int i = tl; i < nblk * kStride; i += kAsmTri) dst[i] = rec[(i / kStride) * kRow + i % kStride];
}

// Map forms: one thread per (triangle, sub-triangle).  The sub-triangle
// barycentrics are gamma = T p with rows T_V = R_hi - R_mid,
// T_E = |v_hi + v_mid| (R_mid - R_lo), T_C = |v1 + v2 + v3| R_lo (R the
// inverse vertex rows of the location record), so the patch
// P_c = gamma^T M_c gamma (M_c the symmetric matrix of the sub-triangle's
// six ordinates) is the homogeneous quadratic form p^T Q_c p with
// Q_c = T^T M_c T.  Q is O(1) while T is O(1/h), so its entries cancel
// terms ~1/h^2 times larger: T, M_c T and Q_c are formed in double-double
// and rounded once.  The result is the exact quadratic form of the patch
// the record's rows R define, and p^T Q p then evaluates in FP64 without
// cancellation (~2e-16 against the Bernstein sum's ~1e-14 from R p).
__device__ __forceinline__ void assemble_form(const MeshView& m, const double* __restrict__ coeffs,
                                              double* __restrict__ forms, int64_t idx) {
  const int t = (int)(idx / 6), sub = (int)(idx % 6);
  const int lo = kSubLo[sub], hi = kSubHi[sub], mid = 3 - lo - hi;
  const double* L = m.tri_loc + (int64_t)t * kLocStride;
  const double ne = edge_norm(L, hi, mid), n4 = __ldg(L + 9);
  dd T[3][3];   // rows V, E, C
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double rh = __ldg(L + 3 * hi + j), rm = __ldg(L + 3 * mid + j), rl = __ldg(L + 3 * lo + j);
    T[0][j] = dd_two_sum(rh, -rm);
    T[1][j] = dd_mul_d(dd_two_sum(rm, -rl), ne);
    T[2][j] = dd_two_prod(n4, rl);
  }
  const int* id = kSplitOrd[lo][hi];   // V^2, E^2, C^2, VE, EC, VC
  const double* rec = coeffs + (int64_t)t * kCoeffStride3;
  double* out = forms + (int64_t)t * kFormStride + 18 * sub;
  // M_c = [[V2, VE, VC], [VE, E2, EC], [VC, EC, C2]] of each component
  double M[3][6];   // per component: the pairs (VV, EE, CC, VE, EC, VC)
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 6; ++k) M[c][k] = __ldg(rec + 3 * id[k] + c);
  // Q_c[i][j] = sum over role pairs a <= b of M_c,ab P_ab[i][j] with
  // P_aa = T_a,i T_a,j and P_ab = T_a,i T_b,j + T_b,i T_a,j (a < b):
  // symmetric in (i, j) by construction, so the stored 2 Q_ij is exact
  const int pa[6] = {0, 1, 2, 0, 1, 0}, pb[6] = {0, 1, 2, 1, 2, 2};   // VV, EE, CC, VE, EC, VC
  const int ei[6] = {0, 1, 2, 0, 0, 1}, ej[6] = {0, 1, 2, 1, 2, 2};   // xx, yy, zz, xy, xz, yz
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    const int i = ei[e], j = ej[e];
    dd P[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int a = pa[k], b = pb[k];
      P[k] = a == b ? dd_mul(T[a][i], T[a][j]) : dd_add_fast(dd_mul(T[a][i], T[b][j]), dd_mul(T[b][i], T[a][j]));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double q = dd_dot_d(P, M[c]);
      out[6 * c + e] = i == j ? q : 2.0 * q;
    }
  }
  if (sub == 0)
    for (int k = 108; k < kFormStride; ++k) forms[(int64_t)t * kFormStride + k] = 0.0;
}

__global__ void __launch_bounds__(128) assemble_forms_kernel(MeshView m, const double* __restrict__ coeffs,
                                                             double* __restrict__ forms) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx < 6LL * m.nt) assemble_form(m, coeffs, forms, idx);
}

// The device-driven step's remap: the forms of the stack slot the current
// map has just been copied to (st->count + 1 in the remap schedule), a
// no-op on the other steps.
__global__ void __launch_bounds__(128) remap_forms_kernel(MeshView m, const BveState* __restrict__ st, int n_maps,
                                                          int Nt, const double* const* __restrict__ table,
                                                          double* const* __restrict__ ftable) {
  const int c = st->count + 1;
  const int slot = c == Nt ? (Nt - 1) / n_maps : (c < Nt && c % n_maps == 0 ? c / n_maps - 1 : -1);
  if (slot < 0) return;
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx < 6LL * m.nt) assemble_form(m, table[slot], ftable[slot], idx);
}

// Low floats of the form records' float-float split: one thread per
// (triangle, sub-triangle, component), the low floats of ff_of of the six
// entries of Q, the cross terms halved (exact), written as three float2
// (padding floats zeroed).
__global__ void __launch_bounds__(128) forms_ff_kernel(int nt, const double* __restrict__ forms,
                                                       float* __restrict__ out) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= 18LL * nt) return;
  const int t = (int)(idx / 18), sc = (int)(idx % 18);   // sc = 3 sub + c
  const double* q = forms + (int64_t)t * kFormStride + 6 * sc;
  float2* o = reinterpret_cast<float2*>(out + (int64_t)t * kFormFFStride + 6 * sc);
  o[0] = make_float2(ff_of(q[0]).l, ff_of(q[1]).l);
  o[1] = make_float2(ff_of(q[2]).l, __fmul_rn(0.5f, ff_of(q[3]).l));
  o[2] = make_float2(__fmul_rn(0.5f, ff_of(q[4]).l), __fmul_rn(0.5f, ff_of(q[5]).l));
  if (sc == 0)
    for (int k = 108; k < kFormFFStride; ++k) out[(int64_t)t * kFormFFStride + k] = 0.f;
}

__global__ void to_f32_kernel(const double* __restrict__ a, int64_t n, float* __restrict__ b) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

// One submap from its coefficient record at p, in triangle t: the
// un-normalised image P and, with JAC, the two pushes (half derivatives).
template <bool JAC>
__device__ __forceinline__ void record_eval(const MeshView& m, const double* __restrict__ recs, int t,
                                            const double* p, Pushes w, double* P) {
  double Lr[13];
  load_loc(m, t, Lr);
  const Bcc b = bcc_of(Lr, p[0], p[1], p[2]);
  const Split sp = split_of(b);
  const Gam g = gamma_of(Lr, b, sp);
  const double* rec = recs + (int64_t)t * kCoeffStride3;
  if (JAC) {
            // The patch is the quadratic form P_c = gamma^T M_c gamma of the
            // symmetric ordinate matrix M_c; its half gradient M_c gamma (FP64)
            // gives the value with three more operations per component and
            // serves the two tangent pushes: half derivatives along the
            // barycentric directions dgamma = T Minv w, formed in float-float
            // from the FP64 location record.
            // the pushes' sub-triangle barycentric directions, ff values 6..11
            // of the thread's shared-memory slots
            {
              ff d1[3], d2[3];
              // the inverse vertex rows re-read (L1) rather than held in
              // registers from the value path
              const double* Lp = m.tri_loc + (int64_t)t * kLocStride;
    #pragma unroll
              for (int r = 0; r < 3; ++r) {
                const ff m0 = ff_of(__ldg(Lp + 3 * r)), m1 = ff_of(__ldg(Lp + 3 * r + 1)),
                         m2 = ff_of(__ldg(Lp + 3 * r + 2));
                d1[r] = ff_dot3(m0, w.get(0), m1, w.get(1), m2, w.get(2));
                d2[r] = ff_dot3(m0, w.get(3), m1, w.get(4), m2, w.get(5));
              }
              const ff en = ff_of(edge_norm(Lr, sp.hi, sp.mid)), ec = ff_of(Lr[9]);
              const ff l1 = pick_ff(d1, sp.lo), m1 = pick_ff(d1, sp.mid), h1 = pick_ff(d1, sp.hi);
              const ff l2 = pick_ff(d2, sp.lo), m2 = pick_ff(d2, sp.mid), h2 = pick_ff(d2, sp.hi);
              w.set(6, ff_sub(h1, m1));
              w.set(7, ff_mul(en, ff_sub(m1, l1)));
              w.set(8, ff_mul(ec, l1));
              w.set(9, ff_sub(h2, m2));
              w.set(10, ff_mul(en, ff_sub(m2, l2)));
              w.set(11, ff_mul(ec, l2));
            }
            const int* id = kSplitOrd[sp.lo][sp.hi];
    #pragma unroll
            for (int c = 0; c < 3; ++c) {
              double o[6];
    #pragma unroll
              for (int k = 0; k < 6; ++k) o[k] = __ldg(rec + 3 * id[k] + c);
              const double pV = g.V * o[0] + g.E * o[3] + g.C * o[5];
              const double pE = g.E * o[1] + g.V * o[3] + g.C * o[4];
              const double pC = g.C * o[2] + g.E * o[4] + g.V * o[5];
              P[c] = g.V * pV + g.E * pE + g.C * pC;
              const ff fV = ff_of(pV), fE = ff_of(pE), fC = ff_of(pC);
              w.set(c, ff_dot3(fV, w.get(6), fE, w.get(7), fC, w.get(8)));
              w.set(3 + c, ff_dot3(fV, w.get(9), fE, w.get(10), fC, w.get(11)));
            }
  } else {
    Ords<3> o;
    load_ords<3>(rec, sp, o);
    sbb<3>(o, g, P);
  }
}

// A composition's submaps: coefficient records only, some with map forms, all
// forms with their low floats.  (Apart: the form code beside the records' cost
// the Jacobians through records 4 %.)
constexpr int kNoForms = 0, kForms = 1, kFormsFF = 2;

// A form's value in FP64: P_c = p^T Q_c p.
__device__ __forceinline__ void form_value(const double* __restrict__ q, const double* p, double* P) {
  const double2* qf = reinterpret_cast<const double2*>(q);
  const double xx = p[0] * p[0], yy = p[1] * p[1], zz = p[2] * p[2];
  const double xy = p[0] * p[1], xz = p[0] * p[2], yz = p[1] * p[2];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double2 q01 = __ldg(qf + 3 * c), q23 = __ldg(qf + 3 * c + 1), q45 = __ldg(qf + 3 * c + 2);
    P[c] = q01.x * xx + q01.y * yy + q23.x * zz + q23.y * xy + q45.x * xz + q45.y * yz;
  }
}

// One submap from its map form: P_c = p^T Q_c p of the sub-triangle's
// quadratic form (24 FP64 operations for the three components) and the
// pushes' half derivatives (Q_c p) . w in float-float.  q: the form's 18
// doubles; g (FF): the low floats of their split, else converted here to the
// same pairs.  ROLL: one component at a time; unrolled, the three copies
// overflow the instruction cache (a quarter of the issue slots lost), but a
// lone warp's three components overlap.  Same operations either way.
template <bool FF, bool ROLL>
__device__ __forceinline__ void form_push(const double* __restrict__ q, const float* __restrict__ g, const double* p,
                                          Pushes w, double* P) {
  const double2* qf = reinterpret_cast<const double2*>(q);
  const float2* qg = reinterpret_cast<const float2*>(g);
  const double xx = p[0] * p[0], yy = p[1] * p[1], zz = p[2] * p[2];
  const double xy = p[0] * p[1], xz = p[0] * p[2], yz = p[1] * p[2];
  const ff u0 = ff_of(p[0]), u1 = ff_of(p[1]), u2 = ff_of(p[2]);
  const ff a0 = w.get(0), a1 = w.get(1), a2 = w.get(2), c0 = w.get(3), c1 = w.get(4), c2 = w.get(5);
#pragma unroll ROLL ? 1 : 3
  for (int c = 0; c < 3; ++c) {
    const double2 q01 = __ldg(qf + 3 * c), q23 = __ldg(qf + 3 * c + 1), q45 = __ldg(qf + 3 * c + 2);
    const double v = q01.x * xx + q01.y * yy + q23.x * zz + q23.y * xy + q45.x * xz + q45.y * yz;
    ff Q00, Q11, Q22, Q01, Q02, Q12;
    if (FF) {   // the stored low floats; the high floats from the doubles' bits
      const float2 ga = __ldg(qg + 3 * c), gb = __ldg(qg + 3 * c + 1), gc = __ldg(qg + 3 * c + 2);
      Q00 = ff{ff_hi(q01.x), ga.x};
      Q11 = ff{ff_hi(q01.y), ga.y};
      Q22 = ff{ff_hi(q23.x), gb.x};
      Q01 = ff{__fmul_rn(0.5f, ff_hi(q23.y)), gb.y};
      Q02 = ff{__fmul_rn(0.5f, ff_hi(q45.x)), gc.x};
      Q12 = ff{__fmul_rn(0.5f, ff_hi(q45.y)), gc.y};
    } else {
      Q00 = ff_of(q01.x);
      Q11 = ff_of(q01.y);
      Q22 = ff_of(q23.x);
      const ff h01 = ff_of(q23.y), h02 = ff_of(q45.x), h12 = ff_of(q45.y);
      Q01 = ff{__fmul_rn(0.5f, h01.h), __fmul_rn(0.5f, h01.l)};
      Q02 = ff{__fmul_rn(0.5f, h02.h), __fmul_rn(0.5f, h02.l)};
      Q12 = ff{__fmul_rn(0.5f, h12.h), __fmul_rn(0.5f, h12.l)};
    }
    const ff g0 = ff_dot3(Q00, u0, Q01, u1, Q02, u2);
    const ff g1 = ff_dot3(Q01, u0, Q11, u1, Q12, u2);
    const ff g2 = ff_dot3(Q02, u0, Q12, u1, Q22, u2);
    w.set(c, ff_dot3(g0, a0, g1, a1, g2, a2));
    w.set(3 + c, ff_dot3(g0, c0, g1, c1, g2, c2));
    P[0] = c == 0 ? v : P[0];
    P[1] = c == 1 ? v : P[1];
    P[2] = c == 2 ? v : P[2];
  }
}

// The pushes brought to the normalised point p: their components along p
// removed, scaled by sc.
__device__ __forceinline__ void project_pushes(const double* p, double scale, Pushes w) {
  const ff sc = ff_of(scale);
  const ff u0 = ff_of(p[0]), u1 = ff_of(p[1]), u2 = ff_of(p[2]);
  const ff d1 = ff_dot3(u0, w.get(0), u1, w.get(1), u2, w.get(2));
  const ff d2 = ff_dot3(u0, w.get(3), u1, w.get(4), u2, w.get(5));
  const ff u[3] = {u0, u1, u2};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w.set(c, ff_mul(ff_sub(w.get(c), ff_mul(u[c], d1)), sc));
    w.set(3 + c, ff_mul(ff_sub(w.get(3 + c), ff_mul(u[c], d2)), sc));
  }
}

// A query's point, normalised first where its FP32 squared norm is outside
// [1/4, 4]; false where it is not finite.
__device__ __forceinline__ bool load_query(const double* __restrict__ q, int64_t i, double* p) {
  p[0] = q[3 * i];
  p[1] = q[3 * i + 1];
  p[2] = q[3 * i + 2];
  const float f0 = to_f32_trunc(p[0]), f1 = to_f32_trunc(p[1]), f2 = to_f32_trunc(p[2]);
  const float n2 = f0 * f0 + f1 * f1 + f2 * f2;
  if (!(n2 > 0.25f && n2 < 4.f)) {   // also NaN / inf
    const double inv = rsqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    p[0] *= inv;
    p[1] *= inv;
    p[2] *= inv;
  }
  return finite3(p[0], p[1], p[2]);
}

// The outputs of a query without a finite image: NaN points and Jacobians,
// ids -1 from submap s (the first not evaluated) on.
template <bool JAC>
__device__ __forceinline__ void store_nan(const MeshView& m, int64_t i, int64_t n, int s, int S,
                                          double* __restrict__ out, int32_t* __restrict__ tri,
                                          int32_t* __restrict__ tri_all, double* __restrict__ jac) {
  flag(m, CMM_FLAG_NONFINITE);
  out[3 * i] = out[3 * i + 1] = out[3 * i + 2] = nan("");
  if (tri && s == S - 1) tri[i] = -1;
  if (tri_all)
    for (; s >= 0; --s) tri_all[(int64_t)s * n + i] = -1;
  if (JAC)
    for (int k = 0; k < 9; ++k) jac[9 * i + k] = nan("");
}

// The Jacobian from the pushes and the tangent basis at the query (formed
// again from q: cheaper than keeping it in registers across the submaps).
__device__ __forceinline__ void store_jacobian(const double* __restrict__ q, int64_t i, Pushes w,
                                               double* __restrict__ jac) {
  const double q0[3] = {q[3 * i], q[3 * i + 1], q[3 * i + 2]};
  ff t1[3], t2[3];
  tangent_basis_ff(q0, t1, t2);
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b2 = 0; b2 < 3; ++b2)
      jac[9 * i + 3 * a + b2] = ff_to_double(ff_dot2(w.get(a), t1[b2], w.get(3 + a), t2[b2]));
}

// Composition in FP64 with the Jacobian's pushes in float-float: through
// coefficient records, through map forms with JAC, and through lists of both
// with many records.  (The fixed-point
// evaluation of compose_forms_kernel does not pay with Jacobians: the pushes
// fill the issue slots that it takes; 2.63 against 2.42 ms per 2^22 queries.)
// perm (nullable): process the queries in this order (grouped by coarse
// cell, cmm_query_order) so that neighbouring threads gather neighbouring
// records; every query's own arithmetic and output slot are unchanged.
// MINB: resident 256-thread blocks per SM the register allocation must
// allow (the register budget; cmm_mesh_set_variant).
template <bool JAC, class Src, int MINB, int FORMS = kNoForms, bool ROLL = false>
__global__ void __launch_bounds__(kBlock, MINB) compose_kernel(MeshView m, Src cp,
                                                         const double* __restrict__ q, int64_t n,
                                                         double* __restrict__ out,
                                                         int32_t* __restrict__ tri,
                                                         int32_t* __restrict__ tri_all,
                                                         double* __restrict__ jac,
                                                         const int32_t* __restrict__ perm) {
  // Jacobian: two tangent vectors pushed through the chain in float-float
  // on the FP32 pipe (points, location predicates, barycentrics and patch
  // values stay FP64).  They live in shared memory, [value][thread], not in
  // registers: with them the loop exceeds the register budget of four
  // resident blocks and spills to local memory, whose traffic thrashes the
  // L1 that the gathers need.
  __shared__ float push_smem[JAC ? 24 * kBlock : 1];
  const int S = cp.count();
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm ? (int64_t)__ldg(perm + j) : j;
    if ((uint64_t)i >= (uint64_t)n) {   // a bad permutation entry
      flag(m, CMM_FLAG_INDEX);
      continue;
    }
    double p[3];
    if (!load_query(q, i, p)) {
      store_nan<JAC>(m, i, n, S - 1, S, out, tri, tri_all, jac);
      continue;
    }
    Pushes w{push_smem + threadIdx.x, (int)blockDim.x};
    int since = 0;   // submaps pushed since the last normalisation
    if (JAC) {   // pushed from the tangent basis at q
      ff t1[3], t2[3];
      tangent_basis_ff(p, t1, t2);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        w.set(c, t1[c]);
        w.set(3 + c, t2[c]);
      }
    }
    for (int s = S - 1; s >= 0; --s) {
      double P[3];
      const double* fr = FORMS != kNoForms ? cp.form(s, S) : nullptr;
      const PointD pt{p[0], p[1], p[2]};
      const float fx = to_f32_trunc(p[0]), fy = to_f32_trunc(p[1]), fz = to_f32_trunc(p[2]);
      Split sp;
      const int t = fr ? locate_split(m, pt, fx, fy, fz, &sp) : locate_row_f(m, pt, fx, fy, fz);
      if (s == S - 1 && tri) tri[i] = t;
      if (tri_all) tri_all[(int64_t)s * n + i] = t;
      if (fr) {
        const int sub = 18 * kSubIndex[sp.lo][sp.hi];
        constexpr bool FF = FORMS == kFormsFF;
        fr += (int64_t)t * kFormStride + sub;
        if (JAC)
          form_push<FF, ROLL>(fr, FF ? cp.form_ff(s, S) + (int64_t)t * kFormFFStride + sub : nullptr, p, w, P);
        else
          form_value(fr, p, P);
      } else {
        record_eval<JAC>(m, cp.at(s, S), t, p, w, P);
      }
      ++since;
      // Location, barycentrics and sub-triangle choice are invariant under
      // p -> lambda p (lambda > 0) and the patch is homogeneous of degree 2,
      // so the projection onto the sphere can wait: normalising every
      // kNormEvery-th submap (and the result) keeps |p| within ~1e-3 of 1
      // for queries on the sphere (|P| = 1 + O(h^3) per submap, the
      // deviation at most doubled per submap) and saves the FP64 square
      // root and scaling.  The tangent pushes then carry exactly the factor
      // |p| / 2^(submaps since the last normalisation) against the
      // normalised chain, and their components along p stay along p
      // (DP(p)[p] = 2 P); both are removed where the point is normalised.
      if ((s & (kNormEvery - 1)) != 0) {
        p[0] = P[0];
        p[1] = P[1];
        p[2] = P[2];
        continue;
      }
      const double inv_n = rsqrt(P[0] * P[0] + P[1] * P[1] + P[2] * P[2]);
      p[0] = P[0] * inv_n;
      p[1] = P[1] * inv_n;
      p[2] = P[2] * inv_n;
      if (JAC) {
        project_pushes(p, inv_n * pow2(since), w);
        since = 0;
      }
    }
    if (!finite3(p[0], p[1], p[2])) flag(m, CMM_FLAG_NONFINITE);
    out[3 * i] = p[0];
    out[3 * i + 1] = p[1];
    out[3 * i + 2] = p[2];
    if (JAC) store_jacobian(q, i, w, jac);
  }
}

// The point of the fixed-point composition as a location's argument: FP64
// values on demand.
struct PointX {
  const long long* X;
  __device__ __forceinline__ PointD fp64() const {
    return PointD{(double)X[0] * kFxUnit, (double)X[1] * kFxUnit, (double)X[2] * kFxUnit};
  }
};

// Points-only composition through map forms (submaps without one through
// their coefficient records).  The point is kept in fixed point (fixed.cuh)
// and every form P_c = p^T Q_c p evaluated on the integer pipes: in FP64 its
// 24 operations per map bound the kernel on GB300 (89 % of the FP64 pipe, 25
// FP64 instructions per evaluation; now ~5 beside ~960 others).  Errors are
// below FP64's roundings: entries to 2^-59, sums to ~2^-57.  A form with an
// entry of 2 or more (a map stretching by more than about 2) goes through
// FP64; a point outside (0.5, 1.4) in squared norm is normalised first.

// The form's nine double2 (in global memory, or GATHER in shared) at X -> X;
// false, with X unchanged, where an entry is out of range.
template <bool GATHER>
__device__ __forceinline__ bool form_fixed(const double2* form, long long* X) {
  double2 Q[9];   // own: all in flight together where the registers hold them
  if (!GATHER) {
#pragma unroll
    for (int k = 0; k < 9; ++k) Q[k] = __ldg(form + k);
  }
  const Limbs x = fx_limbs(X[0]), y = fx_limbs(X[1]), z = fx_limbs(X[2]);
  auto prod = [](Limbs a, Limbs b) {
    FxSum v{0, 0};
    v.add(a, b);
    return fx_limbs(v.value());
  };
  const Limbs xx = prod(x, x), yy = prod(y, y), zz = prod(z, z);
  const Limbs xy = prod(x, y), xz = prod(x, z), yz = prod(y, z);
  if (GATHER) {   // the fetches of form_gather
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
  int bad = 0;
  long long Y[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double2 q0 = GATHER ? form[3 * c] : Q[3 * c], q1 = GATHER ? form[3 * c + 1] : Q[3 * c + 1],
                  q2 = GATHER ? form[3 * c + 2] : Q[3 * c + 2];
    FxSum r{0, 0};
    r.add(fx_entry(q0.x, bad), xx);
    r.add(fx_entry(q0.y, bad), yy);
    r.add(fx_entry(q1.x, bad), zz);
    r.add(fx_entry(q1.y, bad), xy);
    r.add(fx_entry(q2.x, bad), xz);
    r.add(fx_entry(q2.y, bad), yz);
    Y[c] = r.value();
  }
  if (bad < 0) return false;
#pragma unroll
  for (int c = 0; c < 3; ++c) X[c] = Y[c];
  return true;
}

// The point back to the unit sphere; false where it has no direction.
__device__ __forceinline__ bool renormalise(long long* X) {
  const PointD p = PointX{X}.fp64();
  const double inv_n = rsqrt(p.x * p.x + p.y * p.y + p.z * p.z);
  if (!finite3(p.x * inv_n, p.y * inv_n, p.z * inv_n)) return false;
  X[0] = fx_of(p.x * inv_n);
  X[1] = fx_of(p.y * inv_n);
  X[2] = fx_of(p.z * inv_n);
  return true;
}

// One submap in FP64: its coefficient records (form null), or a form out of
// the fixed-point range; false where the image is not finite.
__device__ __forceinline__ bool form_wide(const MeshView& m, const double* __restrict__ form,
                                          const double* __restrict__ recs, int t, long long* X) {
  const PointD u = PointX{X}.fp64();
  double p[3] = {u.x, u.y, u.z}, P[3];
  if (form) {
    form_value(form, p, P);
  } else {
    record_eval<false>(m, recs, t, p, Pushes{nullptr, 0}, P);
  }
  const double r2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
  if (!(r2 > 0.5 && r2 < 1.4)) {
    const double inv_n = rsqrt(r2);
#pragma unroll
    for (int c = 0; c < 3; ++c) P[c] *= inv_n;
    if (!finite3(P[0], P[1], P[2])) return false;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) X[c] = fx_of(P[c]);
  return true;
}

// A first submap without a form (a driver's current map, ahead of its stack) in
// FP64 from the query's own values -> p its image; false where that is not
// finite.  Through form_wide, the conversions to fixed point and back around it
// made one map of the 525,312 sample points at L = 512 81 us instead of 64, and
// 8,320 points at level 7 23 instead of 15.
__device__ __forceinline__ bool record_first(const MeshView& m, const double* __restrict__ recs, double* p, int* t) {
  *t = locate_row_f(m, PointD{p[0], p[1], p[2]}, to_f32_trunc(p[0]), to_f32_trunc(p[1]), to_f32_trunc(p[2]));
  double P[3];
  record_eval<false>(m, recs, *t, p, Pushes{nullptr, 0}, P);
  const double r2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
  const double sc = r2 > 0.5 && r2 < 1.4 ? 1.0 : rsqrt(r2);
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] = P[c] * sc;
  return finite3(p[0], p[1], p[2]);
}

// The composed point's normalised coordinates; false where it has none.
__device__ __forceinline__ bool store_point(double* p, double* __restrict__ out) {
  const double inv_n = rsqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] *= inv_n;
  if (!finite3(p[0], p[1], p[2])) return false;
#pragma unroll
  for (int c = 0; c < 3; ++c) out[c] = p[c];
  return true;
}
__device__ __forceinline__ bool store_point(const long long* X, double* __restrict__ out) {
  double p[3] = {(double)X[0], (double)X[1], (double)X[2]};   // the units drop out
  return store_point(p, out);
}

__device__ __forceinline__ bool off_sphere(float f0, float f1, float f2) {
  const float n2 = fmaf(f0, f0, fmaf(f1, f1, f2 * f2));
  return !(n2 > 0.5f && n2 < 1.4f);
}

// Every lane loads its own forms.  REC: the first submap has none; the locations
// then stand at the loop's head, the only copy of their code beside the record's
// (with one before the loop, as without REC, 981,400 points through 5 level-7
// maps took 296 us in the shared form, 265 so; without REC the other way round
// 392 against 377, 2^20 grouped queries).
template <class Src, int MINB, bool REC>
__global__ void __launch_bounds__(kBlock, MINB) compose_forms_kernel(MeshView m, Src cp,
                                                                     const double* __restrict__ q, int64_t n,
                                                                     double* __restrict__ out,
                                                                     int32_t* __restrict__ tri,
                                                                     int32_t* __restrict__ tri_all,
                                                                     const int32_t* __restrict__ perm) {
  const int S = cp.count();
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm ? (int64_t)__ldg(perm + j) : j;
    if ((uint64_t)i >= (uint64_t)n) {   // a bad permutation entry
      flag(m, CMM_FLAG_INDEX);
      continue;
    }
    long long X[3];   // the point, units of 2^-58
    int t, s = S - 1;
    Split sp;
    {
      double p[3];
      if (!load_query(q, i, p)) {
        store_nan<false>(m, i, n, S - 1, S, out, tri, tri_all, nullptr);
        continue;
      }
      if (REC) {
        const bool ok = record_first(m, cp.at(s, S), p, &t);
        if (tri) tri[i] = t;
        if (tri_all) tri_all[(int64_t)s * n + i] = t;
        --s;
        if (!ok || (s < 0 && !store_point(p, out + 3 * i))) {
          store_nan<false>(m, i, n, s, S, out, tri, tri_all, nullptr);
          continue;
        }
        if (s < 0) continue;
      }
      if (!REC) {   // the first location from the query's own FP64 values
        t = locate_split(m, PointD{p[0], p[1], p[2]}, to_f32_trunc(p[0]), to_f32_trunc(p[1]), to_f32_trunc(p[2]), &sp);
        if (tri) tri[i] = t;
        if (tri_all) tri_all[(int64_t)s * n + i] = t;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) X[c] = fx_of(p[c]);
    }
    bool lost = false;   // no finite image
    float f0, f1, f2;
    auto floats = [&] { f0 = fx_f32(X[0]), f1 = fx_f32(X[1]), f2 = fx_f32(X[2]); };
    auto locate = [&] {
      floats();
      t = locate_split(m, PointX{X}, f0, f1, f2, &sp);
      if (tri_all) tri_all[(int64_t)s * n + i] = t;
    };
    if (!REC) floats();
    while (true) {
      if (REC) locate();
      if (off_sphere(f0, f1, f2)) {   // rare; the direction, and so the location, stays
        lost = !renormalise(X);
        if (lost) break;
      }
      const double* fr = cp.form(s, S);
      if (fr) fr += (int64_t)t * kFormStride + 18 * kSubIndex[sp.lo][sp.hi];
      if (!fr || !form_fixed<false>(reinterpret_cast<const double2*>(fr), X)) {
        lost = !form_wide(m, fr, fr ? nullptr : cp.at(s, S), t, X);
        if (lost) break;
      }
      if (--s < 0) break;
      if (!REC) locate();
    }
    if (lost || !store_point(X, out + 3 * i)) store_nan<false>(m, i, n, s - 1, S, out, tri, tri_all, nullptr);
  }
}

// A warp fetches its 32 forms together, nine neighbouring lanes' 16 bytes a
// form, through shared memory.  Its loads touch two lines a form where every
// lane's own nine touch nine times 32, and all are in flight without a
// register: scattered queries are bound by the lines (2^22 random points
// through 8 level-7 maps 2.98 ms with own loads at 64 registers, 2.54 at 80,
// 1.76 so; in FP64 2.48).  Grouped queries share lines through the L1, of which
// the staging takes 144 KB: 1.32 own, 1.39 so.  All lanes of a warp stay in the
// loops; `live` marks those with a query and a finite image so far.
template <class Src, int MINB, bool REC>
__global__ void __launch_bounds__(kBlock, MINB) compose_forms_gather_kernel(MeshView m, Src cp,
                                                                            const double* __restrict__ q, int64_t n,
                                                                            double* __restrict__ out,
                                                                            int32_t* __restrict__ tri,
                                                                            int32_t* __restrict__ tri_all,
                                                                            const int32_t* __restrict__ perm) {
  // a form's offset is exchanged as an int (in doubles, a level-10 mesh's last triangles would pass 2^31)
  static_assert((20LL << (2 * kMaxLevel)) * (kFormStride / 2) <= INT32_MAX, "form offsets in double2");
  __shared__ double2 stage[9 * kBlock];
  double2* warp = stage + 9 * (threadIdx.x & ~31u);
  const int S = cp.count(), lane = threadIdx.x & 31;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j - lane < n;
       j += (int64_t)gridDim.x * blockDim.x) {
    bool live = j < n;
    const int64_t i = live && perm ? (int64_t)__ldg(perm + j) : j;
    if (live && (uint64_t)i >= (uint64_t)n) {   // a bad permutation entry
      flag(m, CMM_FLAG_INDEX);
      live = false;
    }
    long long X[3] = {0, 0, 0};
    int t = 0, s = S - 1;
    Split sp{0, 2, 1};
    double p[3] = {0.0, 0.0, 0.0};
    if (live) {
      live = load_query(q, i, p);
      if (!live) store_nan<false>(m, i, n, s, S, out, tri, tri_all, nullptr);
    }
    if (REC) {
      if (live) {
        live = record_first(m, cp.at(s, S), p, &t);
        if (tri) tri[i] = t;
        if (tri_all) tri_all[(int64_t)s * n + i] = t;
        if (!live || (s == 0 && !store_point(p, out + 3 * i))) store_nan<false>(m, i, n, s - 1, S, out, tri, tri_all, nullptr);
      }
      if (--s < 0) continue;
    }
    if (live) {
      if (!REC) {
        t = locate_split(m, PointD{p[0], p[1], p[2]}, to_f32_trunc(p[0]), to_f32_trunc(p[1]), to_f32_trunc(p[2]), &sp);
        if (tri) tri[i] = t;
        if (tri_all) tri_all[(int64_t)s * n + i] = t;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) X[c] = fx_of(p[c]);
    }
    float f0, f1, f2;
    auto floats = [&] { f0 = fx_f32(X[0]), f1 = fx_f32(X[1]), f2 = fx_f32(X[2]); };
    auto locate = [&] {
      if (!live) return;
      floats();
      t = locate_split(m, PointX{X}, f0, f1, f2, &sp);
      if (tri_all) tri_all[(int64_t)s * n + i] = t;
    };
    floats();
    while (true) {
      if (REC) locate();
      bool lost = live && off_sphere(f0, f1, f2) && !renormalise(X);
      const double* fr = cp.form(s, S);
      bool wide = !fr;
      if (fr) {
        const double2* forms = reinterpret_cast<const double2*>(fr);
        const int off = t * (kFormStride / 2) + 9 * kSubIndex[sp.lo][sp.hi];   // in double2
        __syncwarp();   // the last map's forms are read
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const int c = 32 * k + lane, r = c / 9;   // double2 c of the warp's, of lane r's form
          const int o = __shfl_sync(0xffffffffu, off, r) + c - 9 * r;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(warp + c)),
                       "l"(forms + o)
                       : "memory");
        }
        wide = !form_fixed<true>(warp + 9 * lane, X);
        fr += 2 * (int64_t)off;
      }
      if (live && !lost && wide) lost = !form_wide(m, fr, fr ? nullptr : cp.at(s, S), t, X);
      if (lost) {
        store_nan<false>(m, i, n, s - 1, S, out, tri, tri_all, nullptr);
        live = false;
      }
      if (--s < 0) break;
      if (!REC) locate();
    }
    if (live && !store_point(X, out + 3 * i)) store_nan<false>(m, i, n, s - 1, S, out, tri, tri_all, nullptr);
  }
}

__global__ void __launch_bounds__(kBlock) stencil_kernel(MeshView m, const double* __restrict__ coeffs,
                                                         const double* __restrict__ yn,
                                                         const double* __restrict__ st, int64_t nv,
                                                         double* __restrict__ out) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const double x = yn[v], y = yn[nv + v], z = yn[2 * nv + v];
  if (!finite3(x, y, z)) {
    flag(m, CMM_FLAG_NONFINITE);
    for (int k = 0; k < 12; ++k) out[k * nv + v] = nan("");
    return;
  }
  const int t = locate_row(m, x, y, z);
  double Lr[13];
  load_loc(m, t, Lr);
  const Split sp = split_of(bcc_of(Lr, x, y, z));
  Ords<3> o;
  load_ords<3>(coeffs + (int64_t)t * kCoeffStride3, sp, o);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double sx = st[(0 * 4 + k) * nv + v], sy = st[(1 * 4 + k) * nv + v],
                 sz = st[(2 * 4 + k) * nv + v];
    const Gam g = gamma_of(Lr, bcc_of(Lr, sx, sy, sz), sp);
    double P[3];
    sbb<3>(o, g, P);
#pragma unroll
    for (int c = 0; c < 3; ++c) out[(c * 4 + k) * nv + v] = P[c];
  }
}

// ------------------------------------------------------- query order
// Counting sort of the queries by coarse cell (the hierarchy node of level
// kOrderLevel containing the query, FP32 descent, no FP64 filter: any
// cell is a valid bucket) in four passes without global atomics:
// per-block histograms, a scan along each cell's row of blocks, a scan of
// the cell totals, a scatter.  A fifth pass groups each cell's queries by
// cube-map cell (64 bins of 1/128): a warp of the composition then gathers
// the records of a few triangles instead of 32, and stays with neighbours
// through the whole stack (the gathers took 78 % of the L1 throughput with
// the coarse cells alone; 2^22 queries through 8 level-7 maps 1.44 -> 1.33
// ms points only, 2.66 -> 2.28 ms with Jacobians).
constexpr int kOrderLevel = 4;          // 20 * 4^4 = 5120 cells
constexpr int kOrderCells = 20 << (2 * kOrderLevel);
constexpr int kOrderBlock = 1024;       // threads per block of passes 1 and 3
constexpr int kOrderPer = 16;           // most queries per thread
constexpr int kOrderFine = 3;           // bits of each cube-map coordinate in the fifth pass
constexpr int kOrderSpan = 4096;        // most queries grouped by one block of it
// fewer queries: the pass costs more than it gives (375,000 on a level-7
// mesh, one a triangle: the composition 177 us without it, 174 with)
constexpr int64_t kOrderFineMin = 1 << 20;

// Queries per thread of passes 1 and 4: as many blocks as SMs before more
// than one query each (the descent is a serial chain; 10^5 queries in
// blocks of 16 per thread ran on 7 SMs).
int order_per(int64_t n) {
  const int64_t per = (n + (int64_t)kOrderBlock * kNumSMs - 1) / ((int64_t)kOrderBlock * kNumSMs);
  return (int)std::min<int64_t>(kOrderPer, std::max<int64_t>(1, per));
}

// pass 1: keys and per-block histograms hist[cell * nblk + block].  key:
// (cell << 2 fine) | interleaved low bits of the query's cube-map cell.  A
// node's three normals are three aligned float4, loaded together: as nine
// scalars, one test after the other, their L1 gathers took 0.62 of the sort's
// 0.69 ms at 2^24 queries.  (In shared memory the table makes the SMs change
// their L1 split between this kernel and the composition, which stalls a
// pipeline of several streams.)
__global__ void __launch_bounds__(kOrderBlock) order_count_kernel(MeshView m, const double* __restrict__ q,
                                                                  int64_t n, int per, int fine,
                                                                  int32_t* __restrict__ key,
                                                                  int32_t* __restrict__ hist) {
  __shared__ int h[kOrderCells];
  const int lv = m.level < kOrderLevel ? m.level : kOrderLevel;
  for (int k = threadIdx.x; k < kOrderCells; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kOrderBlock * per;
  for (int r = 0; r < per; ++r) {
    const int64_t i = base + (int64_t)r * kOrderBlock + threadIdx.x;
    if (i >= n) break;
    const float fx = (float)q[3 * i], fy = (float)q[3 * i + 1], fz = (float)q[3 * i + 2];
    int f = 0;
    float best = -4.0f;
#pragma unroll 4
    for (int g = 0; g < 20; ++g) {
      const float4 c = __ldg(reinterpret_cast<const float4*>(m.root_f + 12 * g));
      const float d = fmaf(c.x, fx, fmaf(c.y, fy, c.z * fz));
      if (d > best) {
        best = d;
        f = g;
      }
    }
    int off = 0, cnt = 20;
    for (int j = 0; j < lv; ++j) {
      const float4* nf = m.coarse_nf + 3 * (off + f);
      const float4 n0 = __ldg(nf), n1 = __ldg(nf + 1), n2 = __ldg(nf + 2);
      const int c = edge_dot(n0, fx, fy, fz) > 0.f ? 0 : (edge_dot(n1, fx, fy, fz) > 0.f ? 1 : (edge_dot(n2, fx, fy, fz) > 0.f ? 2 : 3));
      off += cnt;
      cnt *= 4;
      f = 4 * f + c;
    }
    f <<= 2 * (kOrderLevel - lv);
    atomicAdd(&h[f], 1);
    int sub = 0;
    if (fine) {   // 256 cells along a cube edge: about 8 across a coarse cell
      const int cell = jump_cell(256, fx, fy, fz);
      for (int b = 0; b < fine; ++b)   // bits kOrderFine-1 down to kOrderFine-fine of u and v
        sub = (sub << 2) | (((cell >> (8 + kOrderFine - 1 - b)) & 1) << 1) | ((cell >> (kOrderFine - 1 - b)) & 1);
    }
    key[i] = (f << (2 * fine)) | sub;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kOrderCells; k += blockDim.x) hist[(int64_t)k * gridDim.x + blockIdx.x] = h[k];
}

// pass 2: per cell (one warp each) the exclusive scan of its row of block
// counts in place, and the cell total
__global__ void __launch_bounds__(256) order_rowscan_kernel(int32_t* __restrict__ hist, int nblk,
                                                            int32_t* __restrict__ total) {
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= kOrderCells) return;
  int32_t* row = hist + (int64_t)c * nblk;
  int carry = 0;
  for (int b0 = 0; b0 < nblk; b0 += 32) {
    const int b = b0 + lane;
    const int v = b < nblk ? row[b] : 0;
    int inc = v;
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += t;
    }
    if (b < nblk) row[b] = carry + inc - v;
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) total[c] = carry;
}

// pass 3: exclusive scan of the cell totals (one block)
__global__ void __launch_bounds__(1024) order_cellscan_kernel(int32_t* __restrict__ total) {
  constexpr int per = (kOrderCells + 1023) / 1024;
  __shared__ int part[1024];
  const int lo = threadIdx.x * per;
  int v[per], s = 0;
  for (int k = 0; k < per; ++k) {
    v[k] = lo + k < kOrderCells ? total[lo + k] : 0;
    s += v[k];
  }
  part[threadIdx.x] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int t = threadIdx.x >= d ? part[threadIdx.x - d] : 0;
    __syncthreads();
    part[threadIdx.x] += t;
    __syncthreads();
  }
  int acc = part[threadIdx.x] - s;
  for (int k = 0; k < per; ++k)
    if (lo + k < kOrderCells) {
      total[lo + k] = acc;
      acc += v[k];
    }
}

// pass 4: scatter the query ids into their cells' ranges, the cube-map bin
// (2 fine bits) packed above the id for the fifth pass
__global__ void __launch_bounds__(kOrderBlock) order_scatter_kernel(const int32_t* __restrict__ key, int64_t n, int per,
                                                                    int fine,
                                                                    const int32_t* __restrict__ hist,
                                                                    const int32_t* __restrict__ cbase,
                                                                    int32_t* __restrict__ perm) {
  __shared__ int h[kOrderCells];
  for (int k = threadIdx.x; k < kOrderCells; k += blockDim.x)
    h[k] = cbase[k] + hist[(int64_t)k * gridDim.x + blockIdx.x];
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kOrderBlock * per;
  for (int r = 0; r < per; ++r) {
    const int64_t i = base + (int64_t)r * kOrderBlock + threadIdx.x;
    if (i < n) {
      const int k = key[i];
      const unsigned sub = fine ? (unsigned)k << (32 - 2 * fine) : 0u;   // the low 2 fine bits, at the top
      perm[atomicAdd(&h[k >> (2 * fine)], 1)] = (int32_t)(sub | (unsigned)i);
    }
  }
}

// pass 5: group by cube-map bin inside each cell, in place.  The array is cut
// at the cells' starts and at the multiples of kOrderSpan (so that queries
// crowded into one cell are shared out too): block c < kOrderCells takes the
// piece from cell c's start, block kOrderCells + w the one from w kOrderSpan
// if that lies inside a cell.
__global__ void __launch_bounds__(256) order_group_kernel(const int32_t* __restrict__ cbase, int64_t n, int fine,
                                                          int32_t* __restrict__ perm) {
  constexpr int kPer = kOrderSpan / 256;
  __shared__ int cur[1 << (2 * kOrderFine)];
  const int tid = threadIdx.x, nb = 1 << (2 * fine), shift = 32 - 2 * fine;
  int c;
  int64_t lo;
  if (blockIdx.x < kOrderCells) {
    c = blockIdx.x;
    lo = cbase[c];
  } else {
    lo = (int64_t)(blockIdx.x - kOrderCells) * kOrderSpan;
    int a = 0, b = kOrderCells;   // the last cell starting at or before lo
    while (b - a > 1) {
      const int mid = (a + b) / 2;
      if (cbase[mid] <= lo) a = mid;
      else b = mid;
    }
    c = a;
    if (cbase[c] == lo) return;   // block c's piece
  }
  const int64_t cell_end = c + 1 < kOrderCells ? cbase[c + 1] : n;
  const int64_t hi = min(cell_end, (lo / kOrderSpan + 1) * kOrderSpan);
  const int cnt = (int)(hi - lo);
  if (cnt <= 0) return;
  for (int k = tid; k < nb; k += 256) cur[k] = 0;
  __syncthreads();
  int val[kPer];   // in registers: all are read before any is written back
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int k = r * 256 + tid;
    if (k < cnt) {
      val[r] = perm[lo + k];
      atomicAdd(&cur[(unsigned)val[r] >> shift], 1);
    }
  }
  __syncthreads();
  if (tid < 32) {   // exclusive scan of the nb <= 64 bins, two per lane
    const int k = 2 * tid;
    const int a = k < nb ? cur[k] : 0, b = k + 1 < nb ? cur[k + 1] : 0;
    int inc = a + b;
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, d);
      if (tid >= d) inc += u;
    }
    if (k < nb) cur[k] = inc - a - b;
    if (k + 1 < nb) cur[k + 1] = inc - b;
  }
  __syncthreads();
  const unsigned mask = (1u << shift) - 1u;
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int k = r * 256 + tid;
    if (k < cnt) {
      const unsigned v = (unsigned)val[r];
      perm[lo + atomicAdd(&cur[v >> shift], 1)] = (int32_t)(v & mask);
    }
  }
}

// Cube-map jump table: the row containing every cell centre, by the
// hierarchy descent (the view passed has no jump table yet).
__global__ void __launch_bounds__(kBlock) jump_table_kernel(MeshView m, int R, int* __restrict__ table) {
  const int64_t n = 6LL * R * R;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
    const int face = (int)(c / ((int64_t)R * R)), iv = (int)((c / R) % R), iu = (int)(c % R);
    const double u = -1.0 + (iu + 0.5) * 2.0 / R, v = -1.0 + (iv + 0.5) * 2.0 / R;
    const double sg = (face & 1) ? -1.0 : 1.0;
    double d[3];
    if (face < 2) {
      d[0] = sg; d[1] = u; d[2] = v;
    } else if (face < 4) {
      d[0] = u; d[1] = sg; d[2] = v;
    } else {
      d[0] = u; d[1] = v; d[2] = sg;
    }
    const double in = 1.0 / sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    table[c] = locate_descent(m, d[0] * in, d[1] * in, d[2] * in);
  }
}

int check_launch(const char* what) {
  note_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CMM_OK : cuda_fail(e, what);
}

}  // namespace

int launch_locate(const MeshView& m, const double* q, int64_t n, int32_t* tri, double* bcc,
                  cudaStream_t s) {
  if (n == 0) return CMM_OK;
  const int b = block_for(m, kTuneLocate, kBlock, n);
  locate_kernel<<<grid_for(n, b), b, 0, s>>>(m, q, n, tri, bcc);
  return check_launch("locate_kernel");
}

int launch_assemble(const MeshView& m, const double* jets, int ncomp, double* coeffs,
                    cudaStream_t s, const BveState* st) {
  const int blocks = (m.nt + kAsmTri - 1) / kAsmTri;
  if (ncomp == 3 && m.rec32)
    assemble_f32_kernel<double><<<blocks, kAsmTri, 0, s>>>(m, jets, (float*)coeffs, st);
  else if (ncomp == 3)
    assemble_kernel<3><<<blocks, 3 * kAsmTri, 0, s>>>(m, jets, coeffs, st);
  else
    assemble_kernel<1><<<blocks, 3 * kAsmTri, 0, s>>>(m, jets, coeffs, st);
  return check_launch("assemble_kernel");
}

int launch_assemble_f32_jets(const MeshView& m, const float* jets, cudaStream_t s, const BveState* st) {
  if (!m.rec32 || !st) {
    set_last_error("assemble from FP32 jets: FP32 records and a device-driven state expected");
    return CMM_ERR_ARG;
  }
  const int blocks = (m.nt + kAsmTri - 1) / kAsmTri;
  assemble_f32_kernel<float><<<blocks, kAsmTri, 0, s>>>(m, jets, nullptr, st);
  return check_launch("assemble_f32_kernel");
}

int launch_compose(const MeshView& m, const double* const* coeffs, int S, const double* q,
                   int64_t n, double* out, int32_t* tri, int32_t* tri_all, double* jac,
                   cudaStream_t s, const int32_t* perm, const double* const* forms,
                   const float* const* forms_ff) {
  if (n == 0) return CMM_OK;
  // the low floats are used when every submap with a form record has them
  bool ff = forms_ff != nullptr;
  for (int k = 0; forms && k < S; ++k)
    if (forms[k] && !(forms_ff && forms_ff[k])) ff = false;
  // points only: lists with records beside a first submap's in FP64, where those
  // are more than a third of the forms.  The fixed-point kernels convert the point
  // around each (level 5, 6 records 250,000 points 200 us, 168 in FP64; 3 of 6
  // level-7 maps 179 and 164; a form costs 15.2 against 20.4 and a record 36
  // against 29).
  int with = 0, without = 0;
  for (int k = 0; forms && k < S; ++k) {
    with += forms[k] != nullptr;
    without += !forms[k] && k < S - 1;
  }
  const bool mixed = without > 0 && 3 * without > with;
  const int b = block_for(m, kTuneCompose, kBlock, n);
  const int vj = m.variant[CMM_VARIANT_COMPOSE_JAC], v = m.variant[CMM_VARIANT_COMPOSE];
  auto run = [&](auto list) {
    using Src = decltype(list);
    list.S = S;
    for (int k = 0; k < S; ++k) {
      list.p[k] = coeffs[k];
      list.f[k] = forms ? forms[k] : nullptr;
      list.g[k] = forms && forms[k] && forms_ff ? forms_ff[k] : nullptr;
    }
    auto go = [&](auto kernel) { kernel<<<grid_for(n, b), b, 0, s>>>(m, list, q, n, out, tri, tri_all, jac, perm); };
    if (jac && forms) {
      // by the queries that the chip holds at 2, 3 or 4 blocks per SM: below
      // that the warps are few, and 128 registers with the components unrolled
      // are faster (level 5, 8 maps, 20,000 queries 39 against 58 us of 4
      // blocks rolled; 100,000: 91 with 2 blocks, 74 with 3, 79 with 4; 2^20: 654,
      // 598, 572).  Scattered low floats want the loads in flight of 3 blocks
      // (2^22 random queries, level 7: 3.88 ms against 4.18 of 4 blocks), but
      // not while a third wave of blocks would be the larger part (250,000
      // at level 5: 199 against 189 us).
      const int v = vj ? vj : n <= 2 * kBlockWave ? 2 : (n <= 3 * kBlockWave || (ff && !perm && n > 8 * kBlockWave)) ? 3 : 4;
      if (ff) {
        if (v == 2) go(compose_kernel<true, Src, 2, kFormsFF, false>);
        else if (v == 3) go(compose_kernel<true, Src, 3, kFormsFF, true>);
        else go(compose_kernel<true, Src, 4, kFormsFF, true>);
      } else {
        if (v == 2) go(compose_kernel<true, Src, 2, kForms, false>);
        else if (v == 3) go(compose_kernel<true, Src, 3, kForms, true>);
        else go(compose_kernel<true, Src, 4, kForms, true>);
      }
    } else if (jac) {
      if (vj == 2) go(compose_kernel<true, Src, 2>);
      else if (vj == 3) go(compose_kernel<true, Src, 3>);
      else go(compose_kernel<true, Src, kComposeJacBlocks>);
    } else if (mixed && with) {
      if (v == 6) go(compose_kernel<false, Src, 6, kForms>);
      else go(compose_kernel<false, Src, kComposeBlocks, kForms>);
    } else if (forms && !mixed && (S > 1 || forms[0])) {
      auto gof = [&](auto kernel) { kernel<<<grid_for(n, b), b, 0, s>>>(m, list, q, n, out, tri, tri_all, perm); };
      // Own loads pay where a warp's queries share records: with several
      // queries per triangle, if they are grouped or a map's forms stay in the
      // L2 (73 MB at level 6, 294 at level 7).  Own against shared fetches:
      // grouped 250,000 / 600,000 / 2^20 / 2^22 queries at level 7 127 / 248 /
      // 382 / 1324 against 118 / 243 / 385 / 1390 us, at level 5 91 / 186 / 296 /
      // 1148 against 98 / 204 / 336 / 1310; caller order, random 250,000 at
      // level 6 69 against 60, 10^6 sample points there 168 against 198,
      // 525,000 at level 7 221 against 205.  One form behind a record is fetched
      // as soon by its lane (2^22 random points, level 7: 731 against 762).  In
      // the caller's order at level 7 the rule stands for scattered points (8
      // maps, 2^22: 2980 against 1744 us); a grid's, 2.1 million, take 650 and
      // 715.  While 3 blocks per SM hold all queries 80 registers are faster
      // (60,000 at level 7: 51 / 50 against 61 / 52).
      const bool far = (int64_t)m.nt * kFormStride * 8 > kL2Bytes;
      const bool scattered = (forms[S - 1] || S > 2) && (perm ? n < 2 * (int64_t)m.nt : far || n < 4 * (int64_t)m.nt);
      auto pick = [&](auto rec) {
        constexpr bool REC = decltype(rec)::value;
        if (v == 6) gof(compose_forms_kernel<Src, 6, REC>);
        else if (v == 4) gof(compose_forms_kernel<Src, 4, REC>);
        else if (n <= 3 * kBlockWave && n > kBlockWave && far) gof(compose_forms_gather_kernel<Src, 3, REC>);
        else if (n <= 3 * kBlockWave) gof(compose_forms_kernel<Src, 3, REC>);
        else if (scattered) gof(compose_forms_gather_kernel<Src, 4, REC>);
        else gof(compose_forms_kernel<Src, 4, REC>);
      };
      if (forms[S - 1]) pick(std::false_type{});
      else pick(std::true_type{});
    } else {
      if (v == 6) go(compose_kernel<false, Src, 6>);
      else go(compose_kernel<false, Src, kComposeBlocks>);
    }
  };
  if (S <= kShortList)
    run(SubmapPtrs<kShortList>{});
  else
    run(SubmapPtrs<CMM_MAX_SUBMAPS>{});
  return check_launch("compose_kernel");
}

int launch_assemble_forms(const MeshView& m, const double* coeffs, double* forms, cudaStream_t s) {
  const int64_t n = 6LL * m.nt;
  assemble_forms_kernel<<<(int)((n + 127) / 128), 128, 0, s>>>(m, coeffs, forms);
  return check_launch("assemble_forms_kernel");
}

int launch_forms_ff(const MeshView& m, const double* forms, float* forms_ff, cudaStream_t s) {
  const int64_t n = 18LL * m.nt;
  forms_ff_kernel<<<(int)((n + 127) / 128), 128, 0, s>>>(m.nt, forms, forms_ff);
  return check_launch("forms_ff_kernel");
}

int launch_remap_forms(const MeshView& m, const BveState* st, int n_maps, int Nt, const double* const* table,
                       double* const* ftable, cudaStream_t s) {
  const int64_t n = 6LL * m.nt;
  remap_forms_kernel<<<(int)((n + 127) / 128), 128, 0, s>>>(m, st, n_maps, Nt, table, ftable);
  return check_launch("remap_forms_kernel");
}

int make_asm_f32(cmm_mesh* mesh) {
  const int64_t n = (int64_t)kAsmFactors * mesh->view.nt;
  const int64_t nl = (int64_t)kLocStride * mesh->view.nt;
  int rc = mesh->tri_asm_f.alloc(n * sizeof(float));
  if (rc || (rc = mesh->tri_loc_f.alloc(nl * sizeof(float)))) return rc;
  to_f32_kernel<<<(int)((n + 255) / 256), 256>>>(mesh->view.tri_asm, n, (float*)mesh->tri_asm_f.p);
  if ((rc = check_launch("to_f32_kernel"))) return rc;
  to_f32_kernel<<<(int)((nl + 255) / 256), 256>>>(mesh->view.tri_loc, nl, (float*)mesh->tri_loc_f.p);
  if ((rc = check_launch("to_f32_kernel"))) return rc;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "make_asm_f32");
  mesh->view.tri_asm_f = (const float*)mesh->tri_asm_f.p;
  mesh->view.tri_loc_f = (const float*)mesh->tri_loc_f.p;
  return CMM_OK;
}

int build_jump_table(cmm_mesh* mesh) {
  MeshView& v = mesh->view;
  const int R = std::min(1024, std::max(16, 4 << v.level));
  const int64_t n = 6LL * R * R;
  int rc = mesh->jump.alloc(n * sizeof(int));
  if (rc) return rc;
  MeshView m = v;
  m.jump = nullptr;
  jump_table_kernel<<<grid_for(n, kBlock), kBlock>>>(m, R, (int*)mesh->jump.p);
  if ((rc = check_launch("jump_table_kernel"))) return rc;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "build_jump_table");
  v.jump = (const int*)mesh->jump.p;
  v.jump_res = R;
  return CMM_OK;
}

// Non-decreasing in n, so that a workspace for the largest call serves every
// smaller one: the block count itself falls wherever order_per steps up, so
// the histogram is sized for the most blocks of any call of up to n queries
// (one query per thread until each SM has a block, never more blocks than SMs
// until kOrderPer queries per thread).
int64_t order_workspace(int64_t n) {
  const int64_t one = (n + kOrderBlock - 1) / kOrderBlock, last = (one + kOrderPer - 1) / kOrderPer;
  const int64_t nblk = std::max<int64_t>({1, last, std::min<int64_t>(one, kNumSMs)});
  return n + (int64_t)kOrderCells * (nblk + 1);
}

int launch_query_order(const MeshView& m, const double* q, int64_t n, int32_t* perm, int32_t* work,
                       cudaStream_t s) {
  if (n == 0) return CMM_OK;
  const int per = order_per(n);
  const int64_t nblk = (n + (int64_t)kOrderBlock * per - 1) / ((int64_t)kOrderBlock * per);
  int32_t* key = work;
  int32_t* hist = work + n;
  int32_t* total = hist + (int64_t)kOrderCells * nblk;
  // bins of the fifth pass: as far as the packed ids leave bits, for enough
  // queries, and where a cell holds more than one triangle (2^24 queries on a
  // level-3 mesh: 581 us with the pass, 555 without, for nothing)
  int fine = m.level > kOrderLevel ? kOrderFine : 0;
  while (fine > 0 && (n < kOrderFineMin || n > (1LL << (32 - 2 * fine)))) --fine;
  order_count_kernel<<<(int)nblk, kOrderBlock, 0, s>>>(m, q, n, per, fine, key, hist);
  int rc = check_launch("order_count_kernel");
  if (rc) return rc;
  order_rowscan_kernel<<<kOrderCells / 8, 256, 0, s>>>(hist, (int)nblk, total);
  if ((rc = check_launch("order_rowscan_kernel"))) return rc;
  order_cellscan_kernel<<<1, 1024, 0, s>>>(total);
  if ((rc = check_launch("order_cellscan_kernel"))) return rc;
  order_scatter_kernel<<<(int)nblk, kOrderBlock, 0, s>>>(key, n, per, fine, hist, total, perm);
  if ((rc = check_launch("order_scatter_kernel")) || !fine) return rc;
  order_group_kernel<<<kOrderCells + (int)((n + kOrderSpan - 1) / kOrderSpan), 256, 0, s>>>(total, n, fine, perm);
  return check_launch("order_group_kernel");
}

int launch_compose_dev(const MeshView& m, const double* const* table, const BveState* st,
                       const double* last, const double* q, int64_t n, double* out, cudaStream_t s,
                       const double* const* ftable) {
  if (n == 0) return CMM_OK;
  DevSubmaps cp{table, ftable, st, last};
  const int b = block_for(m, kTuneCompose, kBlock, n);
  const bool six = m.variant[CMM_VARIANT_COMPOSE] == 6;
  auto go = [&](auto kernel) {
    kernel<<<grid_for(n, b), b, 0, s>>>(m, cp, q, n, out, nullptr, nullptr, nullptr, nullptr);
  };
  auto gof = [&](auto kernel) { kernel<<<grid_for(n, b), b, 0, s>>>(m, cp, q, n, out, nullptr, nullptr, nullptr); };
  if (ftable)
    six ? gof(compose_forms_kernel<DevSubmaps, 6, true>) : gof(compose_forms_kernel<DevSubmaps, kComposeBlocks, true>);
  else
    six ? go(compose_kernel<false, DevSubmaps, 6>) : go(compose_kernel<false, DevSubmaps, kComposeBlocks>);
  return check_launch("compose_kernel");
}

int launch_stencil_eval(const MeshView& m, const double* coeffs, const double* yn,
                        const double* st, int64_t nv, double* out, cudaStream_t s) {
  if (nv == 0) return CMM_OK;
  stencil_kernel<<<(int)((nv + kBlock - 1) / kBlock), kBlock, 0, s>>>(m, coeffs, yn, st, nv, out);
  return check_launch("stencil_kernel");
}

}  // namespace cmm
