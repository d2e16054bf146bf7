// Pieces of the FP64 velocity inversion shared by its Legendre kernels: the
// coefficient fields, the ring spectra, the Pbar table's layout.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cmm {
namespace sht {

__device__ __forceinline__ double2 cmul(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cmul(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// offset of order m in a table with nj entries per (m, l): nj sum_{m'<m} (L - m')
__device__ __host__ __forceinline__ int64_t tab_off(int m, int L, int nj) {
  return (int64_t)nj * ((int64_t)m * L - (int64_t)m * (m - 1) / 2);
}

__device__ __forceinline__ double2 order_value(const double2* __restrict__ a, int L, int l, int mm, double d) {
  const int k = mm < 0 ? -mm : mm;
  if (k > l) return make_double2(0.0, 0.0);
  const double2 v = cmul(a[(int64_t)k * L + l], d);
  if (k == 0) return make_double2(v.x, 0.0);   // a real field's: an imaginary part means nothing
  if (mm >= 0) return v;   // a_{l,-k} = (-1)^k conj(a_{l,k})
  return (k & 1) ? make_double2(-v.x, v.y) : make_double2(v.x, -v.y);
}

// The six fields at (l, m), l >= m: d scales a to psi, c[k] = sqrt(l(l+1) -
// q(q-1)) / 2 at q = m-1+k.
constexpr int kVelLegendre = 6;

__device__ __forceinline__ void velocity_fields_at(const double2* __restrict__ a, int L, int l, int m, double d,
                                                   const double* c, double2* f) {
  double2 v[5];   // psi at orders m-2 .. m+2
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = order_value(a, L, l, m - 2 + k, d);
  // X = (up + dn) / 2 and Y = (up - dn) / 2 at orders m-1, m, m+1: u_x = i X,
  // u_y = Y
  double2 X[3], Y[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 up = cmul(v[k], c[k]), dn = cmul(v[k + 2], c[k + 1]);
    X[k] = make_double2(up.x + dn.x, up.y + dn.y);
    Y[k] = make_double2(up.x - dn.x, up.y - dn.y);
  }
  const double cu = c[1], cd = c[2];
  f[0] = v[2];
  f[1] = make_double2(-X[1].y, X[1].x);
  f[2] = Y[1];
  // A_x f = i (cu f_{m-1} + cd f_{m+1}) / 2, A_y f = (cu f_{m-1} - cd f_{m+1}) / 2
  f[3] = make_double2(-(cu * X[0].x + cd * X[2].x), -(cu * X[0].y + cd * X[2].y));
  f[4] = make_double2(-(cu * Y[0].y + cd * Y[2].y), cu * Y[0].x + cd * Y[2].x);
  f[5] = make_double2(cu * Y[0].x - cd * Y[2].x, cu * Y[0].y - cd * Y[2].y);
}

// The nine ring spectra (and grid fields) of the velocity in the FP64 form:
// u_x, u_y, u_z, A_x u_x, A_x u_y, A_y u_y, A_z u_x, A_z u_y, A_z u_z.
constexpr int kVelSpectra = 9;

// Spectra of Legendre field f (velocity_fields_at's order) at (t, m),
// value v, into S (9, L+1, L+1); the m = L column is zeroed beside m = 0
// (an out-of-place C2R transform may overwrite its input).
__device__ __forceinline__ void store_velocity_spectra(double2* __restrict__ S, int L, int f, int t, int m,
                                                       double2 v) {
  const int64_t row = L + 1, fs = (int64_t)(L + 1) * row, at = (int64_t)t * row + m;
  const double2 z = make_double2(-(double)m * v.y, (double)m * v.x);   // i m v
  const double2 zero = make_double2(0.0, 0.0);
  const int64_t ny = (int64_t)t * row + L;
  if (f == 0) {          // psi: u_z = i m psi, A_z u_z = -m^2 psi
    S[2 * fs + at] = z;
    S[8 * fs + at] = make_double2(-(double)m * z.y, (double)m * z.x);
    if (m == 0) S[2 * fs + ny] = S[8 * fs + ny] = zero;
  } else if (f <= 2) {   // u_x, u_y and their A_z
    S[(f - 1) * fs + at] = v;
    S[(f + 5) * fs + at] = z;
    if (m == 0) S[(f - 1) * fs + ny] = S[(f + 5) * fs + ny] = zero;
  } else {
    S[f * fs + at] = v;
    if (m == 0) S[f * fs + ny] = zero;
  }
}

}  // namespace sht
}  // namespace cmm
