// Device building blocks shared by the EMI kernels: complex arithmetic over a real type
// T (float or double) and the Sturm count.
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
template <class D, typename T>
__device__ __forceinline__ int sturm_count(D d, D b2, int n, T sigma, T pivmin) {
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

}  // namespace emi
}  // namespace mr
