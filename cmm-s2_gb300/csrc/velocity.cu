// Velocity interpolant on the MWSS lat-lon mesh, backward integrators and
// the CMM map update (sm_103a).
//
// Location on the lat-lon mesh restates structure_spherical_triangulation
// .inds / .containing_simplex_and_bcc_structured
// (cmm_s2/core/mesh_functions.py:196-282): ring and sector from the angles
// with numpy's floor-division semantics, the reference's near-row
// corrections (theta_c <= 0.03 / > 0.85, great-circle side tests with
// heaviside(0) = 0) and the diagonal side test.  CUDA's atan2/sin/cos are
// not numpy's, so a query exactly on a ring, meridian or diagonal (a
// triangle edge or vertex) may resolve to the other triangle that also
// contains it.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "cmm_internal.h"
#include "device_common.cuh"
#include "fixed.cuh"
#include "geom.h"
#include "integrators.cuh"

namespace cmm {

using namespace dev;

namespace {

constexpr int kBlock = 128;
constexpr int kMaxBlock = 256;   // bound of the tunable advect kernel

// Velocity at q: the Powell-Sabin patch of each time level, combined with
// the stage's Lagrange weights w (spline_interp_velocity.__call__,
// cmm_s2/core/spherical_spline.py:570-615).
struct W3 {
  double a, b, c;
};

// The stage's weights from the kernel parameters or (st) a device-driven
// step's state.
__device__ __forceinline__ W3 stage(const TimeWeights& tw, int s, const BveState* st = nullptr) {
  if (st) return W3{__ldg(&st->tw.w[s][0]), __ldg(&st->tw.w[s][1]), __ldg(&st->tw.w[s][2])};
  return W3{tw.w[s][0], tw.w[s][1], tw.w[s][2]};
}

// FP64 records in FP64: points off the unit sphere, weights of 4 or more,
// ordinates near the ends of the exponent range.
__device__ __noinline__ void velocity_wide(const MeshView& m, const VelPtrs& vc, int nvs, const W3 w, int t, double x,
                                           double y, double z, double* V) {
  V[0] = V[1] = V[2] = 0.0;
  double Lr[13];
  load_loc(m, t, Lr);
  const Bcc b = bcc_of(Lr, x, y, z);
  const Split sp = split_of(b);
  const Gam g = gamma_of(Lr, b, sp);
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    if (l >= nvs) break;
    const double wl = l == 0 ? w.a : (l == 1 ? w.b : w.c);
    Ords<3> o;
    load_ords<3>(vc.p[l] + (int64_t)t * kCoeffStride3, sp, o);
    double P[3];
    sbb<3>(o, g, P);
    V[0] += wl * P[0];
    V[1] += wl * P[1];
    V[2] += wl * P[2];
  }
}


// FP64 records in fixed point (fixed.cuh).  In FP64 an evaluation's ~110
// operations bind the RK4 foot points on GB300 (82 % of the FP64 pipe); here
// the FP64 pipe forms p - v1 only.  The barycentrics b = R (p - v1) + (1,0,0)
// carry no cancellation (R p loses the triangle's inverse size, ~1/h, in
// FP64's last places) and are within 2^(k-55), 2^k the power of two above the
// triangle's largest entry of R (one for the mesh, which the polar triangles
// set, made them 1.5 to 2 times worse than FP64's near the equator: L = 512
// 8e-14).  The Bernstein weights and each level's six ordinates (relative to
// the level's largest) go through 2^-58 steps, and the levels are combined in
// the largest one's scale: from the barycentrics on, a result is within a few
// 2^-57 of the largest ordinate, where the FP64 sum rounds at 2^-53 per term.
__device__ __forceinline__ void velocity_fixed(const MeshView& m, const VelPtrs& vc, int nvs, const W3 w, int t,
                                               double x, double y, double z, double* V) {
  const double* L = m.tri_loc + (int64_t)t * kLocStride;   // R (9), norms (4), v1 (3)
  int bad = 0;
  const Limbs d0 = fx_limbs(fx_of(x - __ldg(L + 13))), d1 = fx_limbs(fx_of(y - __ldg(L + 14))),
              d2 = fx_limbs(fx_of(z - __ldg(L + 15)));
  double R[9];
  int eR = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    R[k] = __ldg(L + k);
    eR = max(eR, fx_exponent(R[k]));
  }
  const int ke = eR - 1022;   // |R| < 2^ke, and ke >= 0: a row's norm is at least 1
  long long b[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    FxSum v{0, 0};
    v.add(fx_scaled(R[3 * r], eR, bad), d0);
    v.add(fx_scaled(R[3 * r + 1], eR, bad), d1);
    v.add(fx_scaled(R[3 * r + 2], eR, bad), d2);
    b[r] = (v.hi << ke) + (v.lo >> (30 - ke));
  }
  b[0] += 1LL << 58;
  // argmin / argmax with the first-index rule (split_of)
  int lo = 0, hi = 0;
  long long bl = b[0], bh = b[0];
  if (b[1] < bl) { bl = b[1]; lo = 1; }
  if (b[2] < bl) { bl = b[2]; lo = 2; }
  if (b[1] > bh) { bh = b[1]; hi = 1; }
  if (b[2] > bh) { bh = b[2]; hi = 2; }
  if (lo == hi) { lo = 1; hi = 0; }
  const int mid = 3 - lo - hi;
  const long long bm = mid == 0 ? b[0] : (mid == 1 ? b[1] : b[2]);
  auto prod = [](Limbs p, Limbs q) {
    FxSum v{0, 0};
    v.add(p, q);
    return v.value();
  };
  // sub-triangle barycentrics; the norms (at most 3) enter as quarters
  const Limbs gV = fx_limbs(bh - bm);
  const int es = hi + mid;
  const double ne = __ldg(L + (es == 1 ? 10 : (es == 3 ? 11 : 12)));
  const Limbs gE = fx_limbs(prod(fx_scaled(ne, 1024, bad), fx_limbs(bm - bl)) << 2);
  const Limbs gC = fx_limbs(prod(fx_scaled(__ldg(L + 9), 1024, bad), fx_limbs(bl)) << 2);
  const Limbs B[6] = {fx_limbs(prod(gV, gV)), fx_limbs(prod(gE, gE)), fx_limbs(prod(gC, gC)),
                      fx_limbs(prod(gV, gE) << 1), fx_limbs(prod(gE, gC) << 1), fx_limbs(prod(gV, gC) << 1)};
  const int* id = kSplitOrd[lo][hi];
  // the levels' patches times their weights (halved, |w| < 4), in the scale
  // 2^(em - 1022) of the largest ordinate so far; one level's code (three
  // unrolled overflow the instruction cache)
  long long U[3] = {0, 0, 0};
  int em = 0;
#pragma unroll 1
  for (int l = 0; l < nvs; ++l) {
    const double* rec = (l == 0 ? vc.p[0] : (l == 1 ? vc.p[1] : vc.p[2])) + (int64_t)t * kCoeffStride3;
    double o[6][3];
    int eb = 0, unused = 0;   // no ordinate is above the largest exponent
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        o[k][c] = __ldg(rec + 3 * id[k] + c);
        eb = max(eb, fx_exponent(o[k][c]));
      }
    const Limbs wl = fx_scaled(l == 0 ? w.a : (l == 1 ? w.b : w.c), 1023, bad);
    const int up = min(max(eb - em, 0), 63), dn = min(max(em - eb, 0), 63);
    em = max(em, eb);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      FxSum v{0, 0};
#pragma unroll
      for (int k = 0; k < 6; ++k) v.add(fx_scaled(o[k][c], eb, unused), B[k]);
      U[c] = (U[c] >> up) + (prod(wl, fx_limbs(v.value())) >> dn);
    }
  }
  if (bad < 0 || em < 100 || em > 1900) {
    velocity_wide(m, vc, nvs, w, t, x, y, z, V);
    return;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) V[c] = fx_to_double(U[c], em + 1);
}

__device__ __forceinline__ void velocity_at(const MeshView& m, const VelPtrs& vc, int nvs,
                                            const W3 w, double x, double y, double z,
                                            double* V) {
  const int t = latlon_locate(m, x, y, z);
  if (m.rec32) {  // FP32 records: barycentrics, patches and time combination in FP32
    const float* Lf = m.tri_loc_f + (int64_t)t * kLocStride;
    float Lr[13];
#pragma unroll
    for (int k = 0; k < 13; ++k) Lr[k] = __ldg(Lf + k);
    const BccF b = bcc_rel_f(m, t, Lr, x, y, z);
    const Split sp = split_of_f(b);
    float gg[3];
    gamma_of_f(Lr, b, sp, gg);
    const float gV = gg[0], gE = gg[1], gC = gg[2];
    float Vf[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      if (l >= nvs) break;
      const float wl = to_f32_trunc(l == 0 ? w.a : (l == 1 ? w.b : w.c));
      OrdsF<3> o;
      load_ords_f<3>((const float*)vc.p[l] + (int64_t)t * kCoeffStride3, sp, o);
      float P[3];
      sbb_f<3>(o, gV, gE, gC, P);
      Vf[0] += wl * P[0];
      Vf[1] += wl * P[1];
      Vf[2] += wl * P[2];
    }
    V[0] = Vf[0];
    V[1] = Vf[1];
    V[2] = Vf[2];
    return;
  }
  const float xf = to_f32_trunc(x), yf = to_f32_trunc(y), zf = to_f32_trunc(z);
  const float n2 = fmaf(xf, xf, fmaf(yf, yf, zf * zf));
  if (n2 > 0.9f && n2 < 1.1f)
    velocity_fixed(m, vc, nvs, w, t, x, y, z, V);
  else
    velocity_wide(m, vc, nvs, w, t, x, y, z, V);
}

// Backward foot point of x under the spline velocity: integrate_back's
// schemes (integrators.cuh) with one copy of the velocity evaluation, whose
// four inlined copies overflow the instruction cache.
__device__ __forceinline__ void integrate_point(const MeshView& m, const VelPtrs& vc, int nvs,
                                                const TimeWeights& tw, int scheme, double dt,
                                                double* x, const BveState* st = nullptr) {
  const int n = scheme == CMM_EULER ? 1 : (scheme == CMM_RK4 ? 4 : 2);
  double s[3] = {x[0], x[1], x[2]}, acc[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    double v[3];
    velocity_at(m, vc, nvs, stage(tw, k, st), s[0], s[1], s[2], v);
    // the stages' sum v1 + 2 v2 + 2 v3 + v4 (RK4), v1 + v2 (improved Euler),
    // the last one alone (Euler, RK2)
    const double f = scheme == CMM_RK4 && (k == 1 || k == 2) ? 2.0 : 1.0;
    const bool add = scheme == CMM_RK4 || scheme == CMM_IMPROVED_EULER;
    for (int c = 0; c < 3; ++c) acc[c] = add ? acc[c] + f * v[c] : v[c];
    const bool last = k == n - 1;
    // the next stage's point, or the foot point
    double a = dt;
    if (last)
      a = scheme == CMM_RK4 ? dt / 6 : (scheme == CMM_IMPROVED_EULER ? dt / 2 : dt);
    else if (scheme == CMM_RK2 || (scheme == CMM_RK4 && k < 2))
      a = dt / 2;
    for (int c = 0; c < 3; ++c) s[c] = x[c] - a * (last ? acc[c] : v[c]);
    sphere_proj(s);
  }
  for (int c = 0; c < 3; ++c) x[c] = s[c];
}

__global__ void __launch_bounds__(kBlock) latlon_locate_kernel(MeshView m, const double* __restrict__ q,
                                                               int64_t n, int32_t* __restrict__ tri,
                                                               double* __restrict__ bcc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double x = q[3 * i], y = q[3 * i + 1], z = q[3 * i + 2];
    if (!finite3(x, y, z)) {
      flag(m, CMM_FLAG_NONFINITE);
      tri[i] = -1;
      if (bcc) bcc[3 * i] = bcc[3 * i + 1] = bcc[3 * i + 2] = nan("");
      continue;
    }
    const int t = latlon_locate(m, x, y, z);
    tri[i] = t;
    if (bcc) {
      const Bcc b = bcc_of(m.tri_loc + (int64_t)t * kLocStride, x, y, z);
      bcc[3 * i] = b.b0;
      bcc[3 * i + 1] = b.b1;
      bcc[3 * i + 2] = b.b2;
    }
  }
}

// x, out: (3,n) component-major, as the reference's (3,N) arrays.
__global__ void __launch_bounds__(kBlock, 4) velocity_kernel(MeshView m, VelPtrs vc, int nvs,
                                                          TimeWeights tw, const double* __restrict__ x,
                                                          int64_t n, double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double px = x[i], py = x[n + i], pz = x[2 * n + i];
    double V[3] = {nan(""), nan(""), nan("")};
    if (finite3(px, py, pz))
      velocity_at(m, vc, nvs, stage(tw, 0), px, py, pz, V);
    else
      flag(m, CMM_FLAG_NONFINITE);
    out[i] = V[0];
    out[n + i] = V[1];
    out[2 * n + i] = V[2];
  }
}

__global__ void __launch_bounds__(kBlock, 4) integrate_kernel(MeshView m, VelPtrs vc, int nvs,
                                                           TimeWeights tw, int scheme, double dt,
                                                           const double* __restrict__ x, int64_t n,
                                                           double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double p[3] = {x[i], x[n + i], x[2 * n + i]};
    if (finite3(p[0], p[1], p[2])) {
      integrate_point(m, vc, nvs, tw, scheme, dt, p);
      if (!finite3(p[0], p[1], p[2])) flag(m, CMM_FLAG_NONFINITE);
    } else {
      flag(m, CMM_FLAG_NONFINITE);
    }
    out[i] = p[0];
    out[n + i] = p[1];
    out[2 * n + i] = p[2];
  }
}

// Foot points of the mesh vertices and of their stencil points
// (advect, cmm_s2/core/evolution_functions.py:117-133).  Five neighbouring
// threads take a vertex and its four stencil points, 1e-5 away: they gather
// the same records at every stage.  work: yn (3,nv) followed by the stencil
// foot points (3,4,nv).  Level 6 / L = 512: 253 us in FP64 with the points
// in array order, ~150 now (issue- and latency-bound: ~3000 instructions per
// velocity, two thirds of them converting the 54 ordinates).
__global__ void __launch_bounds__(kMaxBlock, 2) advect_points_kernel(MeshView mesh, MeshView vm, VelPtrs vc,
                                                               int nvs, TimeWeights tw, int scheme,
                                                               double dt,
                                                               const double* __restrict__ s_pts,
                                                               double* __restrict__ work,
                                                               const BveState* __restrict__ st) {
  if (st) vc = VelPtrs{{st->vel[0], st->vel[1], st->vel[2]}};
  const int64_t nv = mesh.nv, n = 5 * nv;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = i / 5;
    const int k = (int)(i - 5 * v) - 1;   // -1: the vertex, else stencil point k
    const int64_t j = k * nv + v;         // within the (3, 4nv) stencil array
    double p[3];
    if (k < 0) {
      p[0] = mesh.verts[4 * v];
      p[1] = mesh.verts[4 * v + 1];
      p[2] = mesh.verts[4 * v + 2];
    } else {
      p[0] = s_pts[j];
      p[1] = s_pts[4 * nv + j];
      p[2] = s_pts[8 * nv + j];
    }
    integrate_point(vm, vc, nvs, tw, scheme, dt, p, st);
    if (!finite3(p[0], p[1], p[2])) flag(vm, CMM_FLAG_NONFINITE);
    if (k < 0) {
      work[v] = p[0];
      work[nv + v] = p[1];
      work[2 * nv + v] = p[2];
    } else {
      double* sn = work + 3 * nv;
      sn[j] = p[0];
      sn[4 * nv + j] = p[1];
      sn[8 * nv + j] = p[2];
    }
  }
}

// New jets from the stencil images (spline_proj_sphere,
// cmm_s2/core/evolution_functions.py:90-113); with a previous map, the
// images are the previous map evaluated at the stencil foot points in the
// sub-triangle of the vertex foot point, un-normalised (stencil_eval,
// cmm_s2/core/spherical_spline.py:268-298).  Four neighbouring lanes take a
// vertex: lane k evaluates stencil point k, then (k < 3) component k's mean and
// differences and the gradients' slot k.  FP64- and latency-bound: one thread
// per vertex left two warps per SM at level 5 (18 us; level 6: 40 us), a
// quarter of its FP64 work in nine divisions.
__global__ void __launch_bounds__(kBlock) project_jets_kernel(MeshView m, const double* __restrict__ prev,
                                                              const double* __restrict__ yn,
                                                              const double* __restrict__ sn,
                                                              const double* __restrict__ tan,
                                                              double inv4eps, double* __restrict__ jets,
                                                              const BveState* __restrict__ st) {
  const int64_t nv = m.nv;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int k = (int)(i & 3);
  const bool active = (i >> 2) < nv;
  const int64_t v = active ? i >> 2 : nv - 1;   // every lane of the warp takes part in the exchange
  if (st && st->identity) prev = nullptr;
  double P[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) P[c] = sn[(c * 4 + k) * nv + v];
  bool ok = true;
  if (prev) {
    const double x = yn[v], y = yn[nv + v], z = yn[2 * nv + v];
    ok = finite3(x, y, z);
    if (ok) {
      const int t = locate_row(m, x, y, z);
      double Lr[13];
      load_loc(m, t, Lr);
      const Split sp = split_of(bcc_of(Lr, x, y, z));
      Ords<3> o;
      load_ords<3>(prev + (int64_t)t * kCoeffStride3, sp, o);
      const Gam g = gamma_of(Lr, bcc_of(Lr, P[0], P[1], P[2]), sp);
      sbb<3>(o, g, P);
    }
  }
  // component k of the four images (lane 3 repeats component 2)
  double S[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double a = __shfl_sync(0xffffffffu, P[0], q, 4), b = __shfl_sync(0xffffffffu, P[1], q, 4),
                 c = __shfl_sync(0xffffffffu, P[2], q, 4);
    S[q] = k == 0 ? a : (k == 1 ? b : c);
  }
  const double mv = (S[0] + S[1] + S[2] + S[3]) * 0.25;
  const double d1 = (S[1] - S[0] + S[3] - S[2]) * inv4eps;
  const double d2 = (S[2] - S[0] + S[3] - S[1]) * inv4eps;
  const double m0 = __shfl_sync(0xffffffffu, mv, 0, 4), m1 = __shfl_sync(0xffffffffu, mv, 1, 4),
               m2 = __shfl_sync(0xffffffffu, mv, 2, 4);
  if (!active || k == 3) return;
  if (!ok) {
    if (k == 0) flag(m, CMM_FLAG_NONFINITE);
#pragma unroll
    for (int c = 0; c < 3; ++c) jets[(c * 4 + 1 + k) * nv + v] = nan("");
    jets[(k * 4) * nv + v] = nan("");
    return;
  }
  const double* a1 = tan + 3 * v;
  const double* a2 = tan + 3 * (nv + v);
  jets[(k * 4) * nv + v] = mv * rsqrt(m0 * m0 + m1 * m1 + m2 * m2);
#pragma unroll
  for (int c = 0; c < 3; ++c) jets[(c * 4 + 1 + k) * nv + v] = d1 * a1[c] + d2 * a2[c];
  if (!isfinite(mv)) flag(m, CMM_FLAG_NONFINITE);
}

int check_launch(const char* what) {
  note_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CMM_OK : cuda_fail(e, what);
}

}  // namespace

int launch_latlon_locate(const MeshView& vm, const double* q, int64_t n, int32_t* tri, double* bcc,
                         cudaStream_t s) {
  if (n == 0) return CMM_OK;
  latlon_locate_kernel<<<grid_for(n, kBlock), kBlock, 0, s>>>(vm, q, n, tri, bcc);
  return check_launch("latlon_locate_kernel");
}

int launch_velocity_eval(const MeshView& vm, VelPtrs vc, int nvs, const TimeWeights& tw,
                         const double* x, int64_t n, double* out, cudaStream_t s) {
  if (n == 0) return CMM_OK;
  velocity_kernel<<<grid_for(n, kBlock), kBlock, 0, s>>>(vm, vc, nvs, tw, x, n, out);
  return check_launch("velocity_kernel");
}

int launch_integrate(const MeshView& vm, VelPtrs vc, int nvs, const TimeWeights& tw, int scheme,
                     double dt, const double* x, int64_t n, double* out, cudaStream_t s) {
  if (n == 0) return CMM_OK;
  integrate_kernel<<<grid_for(n, kBlock), kBlock, 0, s>>>(vm, vc, nvs, tw, scheme, dt, x, n, out);
  return check_launch("integrate_kernel");
}

int launch_advect_points(const MeshView& mesh, const MeshView& vm, VelPtrs vc, int nvs,
                         const TimeWeights& tw, int scheme, double dt, const double* s_pts,
                         double* work, cudaStream_t s, const BveState* st) {
  const int64_t n = 5LL * mesh.nv;
  const int b = block_for(mesh, kTuneAdvect, kBlock, n);
  advect_points_kernel<<<grid_for(n, b), b, 0, s>>>(mesh, vm, vc, nvs, tw, scheme, dt,
                                                               s_pts, work, st);
  return check_launch("advect_points_kernel");
}

// ---------------------------------------------- allocation-free map update
// Foot-point scratch of advect_project_noalloc: a fixed array in device
// memory that exists on every GPU this library is loaded on, for meshes of
// up to kNoAllocMaxVerts vertices (icosahedral level 5).  Host code must not
// use the name g_advect_scratch as a pointer; the device address of each
// GPU's copy is looked up once per device with cudaGetSymbolAddress.
static __device__ __align__(256) double g_advect_scratch[15 * kNoAllocMaxVerts];

namespace {
constexpr int kMaxDevices = 64;
double* g_scratch_addr[kMaxDevices] = {};
std::mutex g_scratch_mu;
}  // namespace

static int noalloc_scratch(double** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) {
    set_last_error("advect_project_noalloc: device ordinal out of range");
    return CMM_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_advect_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_advect_scratch)");
    g_scratch_addr[dev] = (double*)p;
  }
  *out = g_scratch_addr[dev];
  return CMM_OK;
}

int advect_project_noalloc(const MeshView& mesh, const MeshView& vm, VelPtrs vc, int nvs,
                           const TimeWeights& tw, int scheme, double dt, const double* s_pts,
                           const double* tan, const double* prev_coeffs, double eps,
                           double* jets, cudaStream_t s) {
  if (mesh.nv > kNoAllocMaxVerts) {
    set_last_error("cmm_advect_project_noalloc: mesh has more than " +
                   std::to_string(kNoAllocMaxVerts) +
                   " vertices (icosahedral level 5); use cmm_advect_project with a workspace");
    return CMM_ERR_ARG;
  }
  double* work = nullptr;
  int rc = noalloc_scratch(&work);
  if (rc) return rc;
  // every scratch entry is written by advect_points_kernel before
  // project_jets_kernel reads it, so nothing needs clearing
  if ((rc = launch_advect_points(mesh, vm, vc, nvs, tw, scheme, dt, s_pts, work, s))) return rc;
  return launch_project_jets(mesh, prev_coeffs, work, work + 3 * (int64_t)mesh.nv, tan, eps, jets, s);
}

int launch_project_jets(const MeshView& mesh, const double* prev_coeffs, const double* yn,
                        const double* sn, const double* tan, double eps, double* jets,
                        cudaStream_t s, const BveState* st) {
  const int64_t nv = mesh.nv;
  const int b = small_block(4 * nv, kBlock);
  project_jets_kernel<<<(int)((4 * nv + b - 1) / b), b, 0, s>>>(mesh, prev_coeffs, yn, sn, tan, 1.0 / (4.0 * eps),
                                                                jets, st);
  return check_launch("project_jets_kernel");
}

}  // namespace cmm
