// Device building blocks shared by the EMI kernels: complex arithmetic over a real type
// T (float or double), block reductions, the Sturm count, the pivoted tridiagonal solve,
// and the common tail of EMI (real tridiagonal scaling, smallest eigenvalue by
// multisection, inverse iteration, back-transformation, normalisation to the reference
// image, temporal coherence).
#pragma once

#include <cfloat>

#include "common.cuh"

namespace mr {
namespace emi {

template <typename T> struct C2;
template <> struct C2<float> { using type = float2; };
template <> struct C2<double> { using type = double2; };

template <typename T> struct Lim;
template <> struct Lim<float> {
  static __device__ __forceinline__ float eps() { return FLT_EPSILON; }
  static __device__ __forceinline__ float tiny() { return FLT_MIN; }
  static __device__ __forceinline__ float huge() { return FLT_MAX; }
};
template <> struct Lim<double> {
  static __device__ __forceinline__ double eps() { return DBL_EPSILON; }
  static __device__ __forceinline__ double tiny() { return DBL_MIN; }
  static __device__ __forceinline__ double huge() { return DBL_MAX; }
};

template <typename T> __device__ __forceinline__ typename C2<T>::type mk(T x, T y) {
  typename C2<T>::type c; c.x = x; c.y = y; return c;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
// a * b
template <typename C> __device__ __forceinline__ C cmul_t(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// a * conj(b)
template <typename C> __device__ __forceinline__ C cmulc_t(C a, C b) {
  C r; r.x = a.x * b.x + a.y * b.y; r.y = a.y * b.x - a.x * b.y; return r;
}

__device__ __forceinline__ float sturm_div(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double sturm_div(double a, double b) { return a / b; }

// Number of eigenvalues of the real symmetric tridiagonal (d, b^2) below sigma. In FP32
// the quotient is the fast approximate division (a few ulp): the count then belongs to a
// tridiagonal perturbed at that level, which the bisection tolerates.
template <typename T>
__device__ __forceinline__ int sturm_count(const T* d, const T* b2, int n, T sigma, T pivmin) {
  int c = 0;
  T q = d[0] - sigma;
  if (fabs(q) < pivmin) q = -pivmin;
  c += (q < 0);
  for (int i = 1; i < n; ++i) {
    q = (d[i] - sigma) - sturm_div(b2[i - 1], q);
    if (fabs(q) < pivmin) q = -pivmin;
    c += (q < 0);
  }
  return c;
}

// Solve (R - lambda I) y = y in place by elimination with row interchanges; R has
// diagonal d and off-diagonal b. dd, du, dl: work arrays of length n.
template <typename T>
__device__ inline void tridiag_solve(const T* d, const T* b, int n, T lambda, T tiny, T* y, T* dd, T* du, T* dl) {
  for (int i = 0; i < n; ++i) {
    dd[i] = d[i] - lambda;
    if (i < n - 1) { du[i] = b[i]; dl[i] = b[i]; }
  }
  // dl[i] on exit holds the second super-diagonal of row i (0 when no interchange)
  for (int i = 0; i < n - 1; ++i) {
    const T sub = dl[i];
    if (fabs(dd[i]) >= fabs(sub)) {
      if (dd[i] == T(0)) dd[i] = tiny;
      const T f = sub / dd[i];
      dd[i + 1] -= f * du[i];
      y[i + 1] -= f * y[i];
      dl[i] = T(0);
    } else {
      const T f = dd[i] / sub;
      dd[i] = sub;
      const T t = dd[i + 1];
      dd[i + 1] = du[i] - f * t;
      if (i < n - 2) {
        dl[i] = du[i + 1];
        du[i + 1] = -f * dl[i];
      } else {
        dl[i] = T(0);
      }
      du[i] = t;
      const T ty = y[i];
      y[i] = y[i + 1];
      y[i + 1] = ty - f * y[i + 1];
    }
  }
  if (dd[n - 1] == T(0)) dd[n - 1] = tiny;
  y[n - 1] /= dd[n - 1];
  if (n > 1) y[n - 2] = (y[n - 2] - du[n - 2] * y[n - 1]) / dd[n - 2];
  for (int i = n - 3; i >= 0; --i) y[i] = (y[i] - du[i] * y[i + 1] - dl[i] * y[i + 2]) / dd[i];
}

}  // namespace emi
}  // namespace mr
