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

// Number of eigenvalues of the real symmetric tridiagonal (d, b^2) below sigma: the negative pivots
// q_i = d_i - sigma - b_{i-1}^2 / q_{i-1} (a q below pivmin counts as -pivmin). In FP32
// the quotient is the fast approximate division (a few ulp): the count then belongs to a
// tridiagonal perturbed at that level, which the bisection tolerates.
template <class D>
__device__ __forceinline__ int sturm_count(D d, D b2, int n, float sigma, float pivmin) {
  int c = 0;
  float q = d[0] - sigma;
  if (fabs(q) < pivmin) q = -pivmin;
  c += (q < 0);
  for (int i = 1; i < n; ++i) {
    q = (d[i] - sigma) - __fdividef(b2[i - 1], q);
    if (fabs(q) < pivmin) q = -pivmin;
    c += (q < 0);
  }
  return c;
}

// In FP64 the same pivots as quotients of the leading minors p_i = (d_i - sigma) p_{i-1} - b_{i-1}^2
// p_{i-2}: q_i = p_i / p_{i-1}, negative where the sign changes. Two FMAs on the serial chain instead of
// a division (134 clocks each). Both minors are scaled by a power of two every other step, so that
// p_{i-1} starts each pair in [1, 2): a pair changes it by at most (1 / eps)^4.
template <class D>
__device__ __forceinline__ int sturm_count(D d, D b2, int n, double sigma, double pivmin) {
  int c = 0;
  double p1 = 1.0, p = d[0] - sigma;
  if (fabs(p) < pivmin) p = -pivmin;
  c += p < 0;
  for (int i = 1; i < n; ++i) {
    if (i & 1) {
      const int e = (__double2hiint(p) >> 20) & 0x7ff;  // 2^(1023 - e), for normal p below 2^1023
      const double s = __hiloint2double(max(2046 - e, 1) << 20, 0);
      p *= s;
      p1 *= s;
    }
    double next = (d[i] - sigma) * p - b2[i - 1] * p1;
    if (fabs(next) < pivmin * fabs(p)) next = -pivmin * p;
    c += (next < 0) != (p < 0);
    p1 = p;
    p = next;
  }
  return c;
}

}  // namespace emi
}  // namespace mr
