// EMI for N <= 128 (moraine/pl.py:46-77: M = inv(|Gamma|) o Gamma, its smallest eigenpair,
// phases referred to image `ref`, fused temporal coherence), in sub-batches of points.
//
// Kernels, each at its own occupancy (the register-bound inverse is not held back by the
// shared memory of the reduction, and the serial O(N) tails of many points overlap on an SM):
//   inverse_kernel<T, NB>  inv(|Gamma|) by Gauss-Jordan with partial pivoting in registers
//                          (gj_tile): the padded 16NB x 16NB matrix on a 16 x 16 thread grid,
//                          rows never swapped, one barrier per step; the result stored
//                          upper-packed in the workspace. FP32 and FP64 EMI, and the FP64
//                          recomputation of routed points.
//   sweep_kernel<NB>       inv(|Gamma|) in FP64 for the refined EMI: the symmetric sweep, two
//                          pivots per barrier, only the lower triangle held.
//   reduce_kernel<T, TA>   M in shared memory as a packed lower triangle, Householder
//                          reduction to a real tridiagonal (tridiag_packed) -> workspace (d, e,
//                          tau, reflectors).
//   tail_kernel<T, TA>     one warp per point: smallest eigenvalue by Sturm multisection,
//                          inverse iteration, back-transformation, normalisation, temporal
//                          coherence.
//   tail_refine_kernel     the refined EMI's tail: FP32 eigenpair of the tridiagonal, one FP64
//                          Newton correction and an FP64 error bound that routes the points
//                          it does not certify to FP64.
//   route_kernel           collects the points to recompute in FP64 over all sub-batches.
#include <algorithm>
#include <atomic>

#include "emi_common.cuh"

namespace mr {
namespace emi {

// Largest sub-batch a caller asked for (mr_set_emi_sub_batch); 0: the default.
std::atomic<int64_t> g_sub_batch_cap{0};

namespace {

constexpr int kMaxFastN = 128;

// Gauss-Jordan thread grid: 16 row lanes (ty) x CX column groups (tx), thread tid = 16 tx + ty;
// thread (tx, ty) holds rows ty + 16 ib (ib < NB) and columns tx + CX jb (jb < NC).
template <int NB, int CX>
struct GjGrid {
  static constexpr int NC = (16 * NB + CX - 1) / CX;
  static constexpr int kThreads = 16 * CX;
  static constexpr int kWarps = kThreads / 32;
};

template <typename T, int NB, int CX>
struct GjShared {
  T col[2][16 * NB];
  int piv[2];
  int piv_of_step[16 * NB];
  int step_of_row[16 * NB];
  T part[GjGrid<NB, CX>::kWarps][16 * NB];  // row sums of |a| per warp (norm estimate)
  T wmax[GjGrid<NB, CX>::kWarps];
};

// max_i sum_j |a_ij| over the n x n block of the register tile (the padding excluded);
// deterministic: fixed reduction order. Whole CTA.
template <typename T, int NB, int CX>
__device__ T max_abs_row_sum(const T (&a)[NB][GjGrid<NB, CX>::NC], int n, int tx, int ty, GjShared<T, NB, CX>& s) {
  constexpr int NC = GjGrid<NB, CX>::NC, W = GjGrid<NB, CX>::kWarps;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
  for (int ib = 0; ib < NB; ++ib) {
    T r = 0;
#pragma unroll
    for (int jb = 0; jb < NC; ++jb)
      if (tx + CX * jb < n) r += fabs(a[ib][jb]);
    r += __shfl_xor_sync(0xffffffffu, r, 16);  // the two column groups tx = 2w, 2w + 1 of this warp
    if (lane < 16) s.part[w][ty + 16 * ib] = r;
  }
  __syncthreads();
  T m = 0;
  for (int i = tid; i < n; i += blockDim.x) {
    T r = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) r += s.part[q][i];
    m = fmax(m, r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) s.wmax[w] = m;
  __syncthreads();
  T r = s.wmax[0];
#pragma unroll
  for (int q = 1; q < W; ++q) r = fmax(r, s.wmax[q]);
  __syncthreads();
  return r;
}

// |Gamma| of point c into the register tile (identity on the padding).
template <typename T, int NB, int CX>
__device__ __forceinline__ void load_abs_gamma(T (&a)[NB][GjGrid<NB, CX>::NC], unsigned& used,
                                               const float2* __restrict__ c, int n, int tx, int ty) {
  constexpr int NC = GjGrid<NB, CX>::NC;
  used = 0;
#pragma unroll
  for (int ib = 0; ib < NB; ++ib) {
    const int i = ty + 16 * ib;
    if (i >= n) used |= 1u << ib;  // padding rows never pivot
#pragma unroll
    for (int jb = 0; jb < NC; ++jb) {
      const int j = tx + CX * jb;
      T v = (i == j) ? T(1) : T(0);
      if (i < n && j < n && i != j) {
        const float2 g = c[i < j ? triu_index(i, j, n) : triu_index(j, i, n)];
        v = (T)sqrt((double)g.x * g.x + (double)g.y * g.y);
      }
      a[ib][jb] = v;
    }
  }
}

__device__ __forceinline__ float recip(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double recip(double x) { return __drcp_rn(x); }  // = 1.0 / x, IEEE round-to-nearest

// One Gauss-Jordan step k = CX KB + kt on the register tile; KB is a compile-time column
// slot, so the pivot column is read and rewritten without dynamic register indexing.
template <typename T, int NB, int CX, int KB>
__device__ __forceinline__ void gj_step(T (&a)[NB][GjGrid<NB, CX>::NC], unsigned& used, int k, int tx, int ty,
                                        bool& singular, GjShared<T, NB, CX>& s) {
  constexpr int NC = GjGrid<NB, CX>::NC;
  const int tid = threadIdx.x;
  const int buf = k & 1;
  const bool owner = tx == (k % CX);
  if (owner) {  // the half-warp owning column k: publish it, find the pivot
    const unsigned half = (tx & 1) ? 0xFFFF0000u : 0x0000FFFFu;
    T best = T(-1);
    int bi = -1;
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
      const T v = a[ib][KB];
      s.col[buf][ty + 16 * ib] = v;
      const T av = fabs(v) == fabs(v) ? fabs(v) : T(-0.5);  // NaN ranks last but is taken
      if (!(used & (1u << ib)) && av > best) { best = av; bi = ty + 16 * ib; }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const T ob = __shfl_xor_sync(half, best, o, 16);
      const int oi = __shfl_xor_sync(half, bi, o, 16);
      if (ob > best || (ob == best && oi >= 0 && (bi < 0 || oi < bi))) { best = ob; bi = oi; }
    }
    if (ty == 0) s.piv[buf] = bi;
  }
  __syncthreads();
  const int p = s.piv[buf];
  T pv = s.col[buf][p];
  if (pv == T(0)) { singular = true; pv = T(1); }
  const T rp = recip(pv);
  if (ty == (p & 15)) used |= 1u << (p >> 4);
  if (tid == 0) { s.piv_of_step[k] = p; s.step_of_row[p] = k; }
  const int pl = p & 15;
  // pivot row (scaled) from row lane pl of this column group; p >> 4 is CTA-uniform
  T r[NC];
  switch (p >> 4) {
#define MR_GJ_ROW(PB)                                                                  \
  case PB:                                                                             \
    if (PB < NB) {                                                                     \
      _Pragma("unroll") for (int jb = 0; jb < NC; ++jb) r[jb] =                        \
          __shfl_sync(0xffffffffu, a[PB < NB ? PB : 0][jb], pl, 16) * rp;              \
    }                                                                                  \
    break;
    MR_GJ_ROW(0) MR_GJ_ROW(1) MR_GJ_ROW(2) MR_GJ_ROW(3) MR_GJ_ROW(4) MR_GJ_ROW(5) MR_GJ_ROW(6)
    default: MR_GJ_ROW(7)
#undef MR_GJ_ROW
  }
  // a -= f_i r_j everywhere, with f_p = pv - 1 so that the pivot row becomes r; then
  // column k becomes delta_ip / pv - f_i / pv
#pragma unroll
  for (int ib = 0; ib < NB; ++ib) {
    const int i = ty + 16 * ib;
    const T fi = s.col[buf][i];
    const T f = (i == p) ? pv - T(1) : fi;
#pragma unroll
    for (int jb = 0; jb < NC; ++jb) a[ib][jb] -= f * r[jb];
    if (owner) a[ib][KB] = (i == p) ? rp : -fi * rp;
  }
}

// In-place Gauss-Jordan inverse with partial pivoting on the register tile. Returns true
// when a zero pivot was met (the matrix is singular).
template <typename T, int NB, int CX>
__device__ bool gj_tile(T (&a)[NB][GjGrid<NB, CX>::NC], unsigned used, int n, int tx, int ty,
                        GjShared<T, NB, CX>& s) {
  constexpr int NC = GjGrid<NB, CX>::NC;
  bool singular = false;
#pragma unroll
  for (int kb = 0; kb < NC; ++kb) {
    for (int kt = 0; kt < CX; ++kt) {
      const int k = CX * kb + kt;
      if (k >= n) break;
      switch (kb) {  // compile-time slot (the loop over kb is unrolled)
        case 0: gj_step<T, NB, CX, 0>(a, used, k, tx, ty, singular, s); break;
        case 1: if (NC > 1) gj_step<T, NB, CX, (1 < NC ? 1 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 2: if (NC > 2) gj_step<T, NB, CX, (2 < NC ? 2 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 3: if (NC > 3) gj_step<T, NB, CX, (3 < NC ? 3 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 4: if (NC > 4) gj_step<T, NB, CX, (4 < NC ? 4 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 5: if (NC > 5) gj_step<T, NB, CX, (5 < NC ? 5 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 6: if (NC > 6) gj_step<T, NB, CX, (6 < NC ? 6 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 7: if (NC > 7) gj_step<T, NB, CX, (7 < NC ? 7 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 8: if (NC > 8) gj_step<T, NB, CX, (8 < NC ? 8 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 9: if (NC > 9) gj_step<T, NB, CX, (9 < NC ? 9 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 10: if (NC > 10) gj_step<T, NB, CX, (10 < NC ? 10 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 11: if (NC > 11) gj_step<T, NB, CX, (11 < NC ? 11 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 12: if (NC > 12) gj_step<T, NB, CX, (12 < NC ? 12 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 13: if (NC > 13) gj_step<T, NB, CX, (13 < NC ? 13 : 0)>(a, used, k, tx, ty, singular, s); break;
        case 14: if (NC > 14) gj_step<T, NB, CX, (14 < NC ? 14 : 0)>(a, used, k, tx, ty, singular, s); break;
        default: if (NC > 15) gj_step<T, NB, CX, (15 < NC ? 15 : 0)>(a, used, k, tx, ty, singular, s); break;
      }
    }
  }
  __syncthreads();
  return singular;
}

// ----------------------------------------------------------------- packed reduction
__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }
__host__ __device__ __forceinline__ int tri(int i) { return i * (i + 1) / 2; }

// a -= ui conj(wj) + wi conj(uj)
template <typename C> __device__ __forceinline__ void rank2(C& a, C ui, C wj, C wi, C uj) {
  // one FMA per product (no separate multiply and add)
  a.x -= ui.x * wj.x; a.x -= ui.y * wj.y; a.x -= wi.x * uj.x; a.x -= wi.y * uj.y;
  a.y -= ui.y * wj.x; a.y += ui.x * wj.y; a.y -= wi.y * uj.x; a.y += wi.x * uj.y;
}

// acc += a b (one FMA per product)
template <typename C> __device__ __forceinline__ void cmac(C& acc, C a, C b) {
  acc.x += a.x * b.x;
  acc.x -= a.y * b.y;
  acc.y += a.x * b.y;
  acc.y += a.y * b.x;
}
// acc += conj(a) b
template <typename C> __device__ __forceinline__ void cmacc(C& acc, C a, C b) {
  acc.x += a.x * b.x;
  acc.x += a.y * b.y;
  acc.y += a.x * b.y;
  acc.y -= a.y * b.x;
}
template <typename C> __device__ __forceinline__ C shfl_xor_c(C v, int o) {
  v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
  v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
  return v;
}

// Sum over the 32 lanes of four per-lane values r[0..3] (reduce-scatter): afterwards lane l
// holds the total of value (l >> 3) & 3 (lanes 0, 8, 16, 24 hold values 0, 1, 2, 3).
template <typename C> __device__ __forceinline__ C warp_sum4(const C (&r)[4]) {
  const int lane = threadIdx.x & 31;
  const bool hi4 = lane & 16, hi3 = lane & 8;
  C k0 = hi4 ? r[2] : r[0], k1 = hi4 ? r[3] : r[1];
  const C s0 = hi4 ? r[0] : r[2], s1 = hi4 ? r[1] : r[3];
  k0 = cadd(k0, shfl_xor_c(s0, 16));
  k1 = cadd(k1, shfl_xor_c(s1, 16));
  C k = hi3 ? k1 : k0;
  k = cadd(k, shfl_xor_c(hi3 ? k0 : k1, 8));
  k = cadd(k, shfl_xor_c(k, 4));
  k = cadd(k, shfl_xor_c(k, 2));
  k = cadd(k, shfl_xor_c(k, 1));
  return k;
}

// Sums over the 16 lanes of each half-warp: lane l holds the total of value (l % 16) / 4 of four, or
// (l % 16) / 8 of two.
template <typename C> __device__ __forceinline__ C half_warp_sum(const C (&r)[2]) {
  const bool hi3 = threadIdx.x & 8;
  C k = hi3 ? r[1] : r[0];
  k = cadd(k, shfl_xor_c(hi3 ? r[0] : r[1], 8));
  k = cadd(k, shfl_xor_c(k, 4));
  k = cadd(k, shfl_xor_c(k, 2));
  return cadd(k, shfl_xor_c(k, 1));
}
template <typename C> __device__ __forceinline__ C half_warp_sum(const C (&r)[4]) {
  const bool hi3 = threadIdx.x & 8, hi2 = threadIdx.x & 4;
  C k0 = hi3 ? r[2] : r[0], k1 = hi3 ? r[3] : r[1];
  const C s0 = hi3 ? r[0] : r[2], s1 = hi3 ? r[1] : r[3];
  k0 = cadd(k0, shfl_xor_c(s0, 8));
  k1 = cadd(k1, shfl_xor_c(s1, 8));
  C k = hi2 ? k1 : k0;
  k = cadd(k, shfl_xor_c(hi2 ? k0 : k1, 4));
  k = cadd(k, shfl_xor_c(k, 2));
  return cadd(k, shfl_xor_c(k, 1));
}

// ----------------------------------------------------------------- workspace layout
// Per point: inv(|Gamma|) in the arithmetic TA of the inverse, packed upper triangle by
// rows like the compressed coherence ((m, j >= m) at tri_up(m, j)); then, in the arithmetic
// T of the reduction, the reflectors (column k rows k+1..n-1, packed by column, nq complex
// T), d and tau (n T each), e (n complex T).
__host__ __device__ __forceinline__ int64_t tri_up(int m, int j, int n) {
  return (int64_t)m * n - ((int64_t)m * (m - 1)) / 2 + (j - m);
}

template <typename T, typename TA = T>
struct PointWs {
  size_t np, nq, bytes;
  __host__ __device__ explicit PointWs(int n) {
    using C = typename C2<T>::type;
    np = (size_t)n * (n + 1) / 2;
    nq = (size_t)n * (n - 1) / 2;
    bytes = align16(np * sizeof(TA)) + align16(nq * sizeof(C)) + align16(2 * (size_t)n * sizeof(T)) +
            align16((size_t)n * sizeof(C));
  }
};

template <typename T, typename TA = T>
struct PointPtr {
  using C = typename C2<T>::type;
  TA* ainv;
  C* refl;
  T* d;
  T* tau;
  C* e;
  __device__ PointPtr(unsigned char* ws, int64_t pt, int n) {
    const PointWs<T, TA> w(n);
    unsigned char* b = ws + (size_t)pt * w.bytes;
    ainv = reinterpret_cast<TA*>(b);
    b += align16(w.np * sizeof(TA));
    refl = reinterpret_cast<C*>(b);
    b += align16(w.nq * sizeof(C));
    d = reinterpret_cast<T*>(b);
    tau = d + n;
    b += align16(2 * (size_t)n * sizeof(T));
    e = reinterpret_cast<C*>(b);
  }
};

__host__ __device__ __forceinline__ size_t refl_off(int k, int n) { return (size_t)k * (n - 1) - (size_t)k * (k - 1) / 2; }

// ----------------------------------------------------------------- kernel 1: inverse
// Route flags of a point (sing[] in the workspace, route[] on output).
constexpr uint8_t kRouteCond = 1;      // cond_1(|Gamma|) estimate above the threshold
constexpr uint8_t kRouteSingular = 2;  // a zero pivot: |Gamma| singular at this precision

// Points of a pass: all n_pc of the sub-batch; or, with a list, list[off + i] for
// i < min(*count - off, n_pc), a window of at most n_pc entries of a list that may be longer.
struct PointSet {
  const int32_t* list;
  const int32_t* count;
  int64_t n_pc;
  const int64_t* dcount;  // without a list: the points are dcount[0] - off, at most n_pc
  int64_t off;
  __device__ __forceinline__ int64_t size() const {
    if (list || dcount) {
      const int64_t c = (list ? (int64_t)*count : *dcount) - off;
      return c < 0 ? 0 : (c < n_pc ? c : n_pc);
    }
    return n_pc;
  }
  __device__ __forceinline__ int64_t operator[](int64_t i) const { return list ? (int64_t)list[off + i] : i; }
};

// TW: arithmetic of the reduction that reads the workspace (the point stride depends on it).
template <typename T, int NB, int CX, typename TW>
__global__ void __launch_bounds__(16 * CX, 1) inverse_kernel(const float2* __restrict__ coh, PointSet pts, int n,
                                                          unsigned char* __restrict__ ws, uint8_t* __restrict__ sing,
                                                          float cond_max) {
  constexpr int NC = GjGrid<NB, CX>::NC;
  __shared__ GjShared<T, NB, CX> gs;
  const int tid = threadIdx.x, tx = tid >> 4, ty = tid & 15;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = blockIdx.x; pt < npt; pt += gridDim.x) {
    const int64_t gp = pts[pt];
    T a[NB][NC];
    unsigned used;
    load_abs_gamma<T, NB, CX>(a, used, coh + gp * npairs, n, tx, ty);
    const T anorm = cond_max > 0.f ? max_abs_row_sum<T, NB, CX>(a, n, tx, ty, gs) : T(0);
    const bool singular = gj_tile<T, NB, CX>(a, used, n, tx, ty, gs);
    uint8_t flag = singular ? kRouteSingular : 0;
    if (cond_max > 0.f && !singular) {
      // cond_1 = ||A||_1 ||inv(A)||_1 (A symmetric: row sums); the register rows of the
      // result are the rows of inv(A) in pivot order
      const T cond = anorm * max_abs_row_sum<T, NB, CX>(a, n, tx, ty, gs);
      if (!(cond <= (T)cond_max)) flag = kRouteCond;
    }
    T* out = PointPtr<TW, T>(ws, pt, n).ainv;
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
      const int r0 = ty + 16 * ib;
      if (r0 >= n) continue;
      const int kr = gs.step_of_row[r0];
#pragma unroll
      for (int jb = 0; jb < NC; ++jb) {
        const int c0 = tx + CX * jb;
        if (c0 >= n) continue;
        const int pc = gs.piv_of_step[c0];
        if (kr >= pc) out[tri_up(pc, kr, n)] = a[ib][jb];  // inv[kr][pc], kept once
      }
    }
    if (tid == 0) sing[pt] = flag;
    __syncthreads();
  }
}

// ----------------------------------------------------------------- kernel 1c: inverse, N > 128
// The same Gauss-Jordan (partial pivoting, rows never swapped) with the matrix in shared memory
// (kIn: up to kBigIn images) or in the CTA's slice of the workspace, one CTA of 32 warps per point.
// Every warp takes the pivot of column k from the 32 warps' candidates, which they left with the
// column's values while they updated it in step k-1, and the scaled pivot row into registers; after
// a barrier the warps update their rows, lanes along the columns. Two barriers per step. Bound by
// shared-memory (or L2) bandwidth, 16 bytes per element and step.
constexpr int kBigThreads = 1024;
constexpr int kBigIn = 160;

template <int Q, bool kIn>
__global__ void __launch_bounds__(kBigThreads, 1) big_inverse_kernel(const float2* __restrict__ coh, PointSet pts, int n,
                                                                     unsigned char* __restrict__ ws,
                                                                     uint8_t* __restrict__ sing,
                                                                     double* __restrict__ slices) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double col[2][32 * Q];
  __shared__ int piv_of_step[32 * Q], step_of_row[32 * Q];
  constexpr int W = kBigThreads / 32;
  static_assert(W == 32, "one candidate per lane");
  __shared__ double cand[W];
  __shared__ int cand_row[W];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int ld = kIn ? n | 1 : n;  // odd: a column's values on different banks
  double* A = kIn ? reinterpret_cast<double*>(smem_raw) : slices + (size_t)blockIdx.x * n * n;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = blockIdx.x; pt < npt; pt += gridDim.x) {
    const float2* c = coh + pts[pt] * npairs;
    for (int i = wid; i < n; i += W) {
      const float2* ci = c + (triu_index(i, i + 1, n) - (i + 1));
      for (int j = i + lane; j < n; j += 32) {
        const float2 g = j == i ? make_float2(1.f, 0.f) : ci[j];
        const double v = sqrt((double)g.x * g.x + (double)g.y * g.y);
        A[i * ld + j] = v;
        A[j * ld + i] = v;
        if (i == 0) col[0][j] = v;
      }
    }
    if (lane == 0) {  // the first column's candidates
      double best = -1.0;
      int at = -1;
      for (int i = wid; i < n; i += W) {
        const float2 g = i ? c[i - 1] : make_float2(1.f, 0.f);
        const double v = sqrt((double)g.x * g.x + (double)g.y * g.y), av = v == v ? v : -0.5;
        if (av > best) { best = av; at = i; }
      }
      cand[wid] = best;
      cand_row[wid] = at;
    }
    unsigned used = 0;  // bit r: this warp's row wid + W r has been a pivot row
    bool singular = false;
    __syncthreads();
    for (int k = 0; k < n; ++k) {
      const double* ck = col[k & 1];
      double best = cand[lane];  // W = 32 candidates, -1 and no row from a warp with none left
      int p = cand_row[lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, p, o);
        if (ob > best || (ob == best && oi >= 0 && (p < 0 || oi < p))) { best = ob; p = oi; }
      }
      double pv = ck[p];
      if (pv == 0.0) { singular = true; pv = 1.0; }
      const double rp = recip(pv);
      double r[Q];  // the pivot row, scaled
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const int j = lane + 32 * t;
        r[t] = j < n ? A[p * ld + j] * rp : 0.0;
      }
      __syncthreads();
      if (tid == 0) {
        step_of_row[p] = k;
        piv_of_step[k] = p;
      }
      if (wid == (p & (W - 1))) used |= 1u << (p / W);
      double* cn = col[(k + 1) & 1];
      double top = -1.0;
      int at = -1;
      for (int i = wid, b = 0; i < n; i += W, ++b) {
        double* row = A + i * ld;
        if (i == p) {
#pragma unroll
          for (int t = 0; t < Q; ++t)
            if (lane + 32 * t < n) row[lane + 32 * t] = r[t];
        } else {
          const double f = ck[i];
#pragma unroll
          for (int t = 0; t < Q; ++t) {
            const int j = lane + 32 * t;
            if (32 * t + 31 < n || j < n) row[j] -= f * r[t];
          }
        }
        __syncwarp();
        if (lane == 0) {  // column k, and column k + 1 with this warp's best unused row for the next step
          row[k] = i == p ? rp : -ck[i] * rp;
          if (k + 1 < n) {
            const double v = row[k + 1], av = fabs(v) == fabs(v) ? fabs(v) : -0.5;  // NaN ranks last but is taken
            cn[i] = v;
            if (!(used >> b & 1) && av > top) { top = av; at = i; }
          }
        }
      }
      if (lane == 0) {
        cand[wid] = top;
        cand_row[wid] = at;
      }
      __syncthreads();
    }
    double* out = PointPtr<double, double>(ws, pt, n).ainv;
    for (int i = wid; i < n; i += W) {
      const int kr = step_of_row[i];
      for (int j = lane; j < n; j += 32) {
        const int pc = piv_of_step[j];
        if (kr >= pc) out[tri_up(pc, kr, n)] = A[i * ld + j];  // inv[kr][pc], kept once
      }
    }
    if (tid == 0) sing[pt] = singular ? kRouteSingular : 0;
    __syncthreads();
  }
}

// ----------------------------------------------------------------- kernel 1b: symmetric sweep
// inv(|Gamma|) for the refined mixed precision, FP64: Gauss-Jordan on the symmetric matrix
// with diagonal pivots in natural order (the sweep operator), which keeps the matrix
// symmetric, so only its lower triangle is held and updated: half the registers of the
// pivoted kernel (two CTAs per SM) and half its FMAs, with no pivot search on the serial
// chain of a step. Step k with column c = A[:, k] (c_k = d):
//   A_ij -= c_i c_j / d (i, j != k);  A_ik = c_i / d (i != k);  A_kk = -1 / d,
// and after all n steps A holds -inv(A). Without interchanges a pivot can become small on
// an indefinite |Gamma|; the kernel flags the point (kRouteCond) when a pivot falls below
// kSweepMinPivot in magnitude, and the refined pass recomputes flagged
// points with the pivoted FP64 kernels. On the c2 scene model the natural order stays
// within about 30 eps cond(|Gamma|) of the pivoted inverse (3.7e-9 relative at worst over
// 1,500 points, 41 % of them indefinite), far below what the refinement needs.
constexpr double kSweepMinPivot = 1e-9;

template <int NB>
struct SweepShared {
  double2 col[2][16 * NB];  // columns k and k + 1 of a pivot pair, (A_ik, A_i,k+1), by pair parity
};

__host__ __device__ constexpr int lt(int ib, int jb) { return ib * (ib + 1) / 2 + jb; }  // jb <= ib

// Thread (tx, ty) of the 16 x 16 grid holds A[i][j] for i = ty + 16 ib, j = tx + 16 jb,
// jb <= ib (NB (NB + 1) / 2 values); in a diagonal block only ty >= tx is the lower triangle
// (the rest is updated like it but never read).
//
// Pivots go in pairs K = {k, k + 1} (k even; with n odd the last pair takes the identity row
// of the padding): with P = A_KK, the two sweeps at once are
//   A_ij -= A_iK inv(P) A_Kj (i, j not in K);  A_iK = A_iK inv(P);  A_KK = -inv(P),
// one barrier per pair, evaluated as the two single sweeps in sequence (sweep_pair). The
// owners of columns k, k + 1 (two lanes of every half-warp) write A_iK, the owners of rows
// k, k + 1 (one whole warp, as ty = k, k + 1 share a warp) write A_Kj and -inv(P). The
// point is flagged when a natural-order pivot (P_00, then P_11 - P_10^2 / P_00) falls below
// kSweepMinPivot.

// Columns k2, k2 + 1 of the matrix into `out`: the lower parts (rows >= k2, >= k2 + 1) from
// the owners of those columns, the upper parts from the owners of rows k2, k2 + 1 (symmetry).
// KBX = k2 >> 4 at compile time.
template <int NB, int KBX>
__device__ __forceinline__ void sweep_publish(const double (&a)[NB * (NB + 1) / 2], int k2, int tx, int ty,
                                              double2* out) {
  const int kt2 = k2 & 15;
  if (tx == kt2 || tx == kt2 + 1) {
    const int c = tx - kt2;
#pragma unroll
    for (int ib = KBX; ib < NB; ++ib) {
      const int i = ty + 16 * ib;
      if (i >= k2 + c) (c ? out[i].y : out[i].x) = a[lt(ib, KBX)];
    }
  }
  if (ty == kt2 || ty == kt2 + 1) {
    const int r = ty - kt2;
#pragma unroll
    for (int jb = 0; jb <= KBX; ++jb) {
      const int j = tx + 16 * jb;
      if (j < k2 + r) (r ? out[j].y : out[j].x) = a[lt(KBX, jb)];
    }
  }
}

template <int NB, int KB>
__device__ __forceinline__ void sweep_pair(double (&a)[NB * (NB + 1) / 2], int k, int n, int tx, int ty,
                                           bool& small, SweepShared<NB>& s) {
  const int buf = (k >> 1) & 1;
  const double2* col = s.col[buf];
  const int kt = k & 15;
  const double2 pk = col[k], pk1 = col[k + 1];
  // the two sweeps in sequence, fused: sweep k turns column k + 1 into c1' = c1 - t c0
  // (t = P_10 / P_00) and its pivot into d1 = P_11 - t P_10; then
  //   A_ij -= g0_i c0_j + g1_i c1'_j,  g0 = c0 / P_00, g1 = c1' / d1,
  // the same two roundings per element as two single sweeps (the product form
  // c_i inv(P) c_j^T instead loses accuracy to cancellation when d1 is small)
  const double r0 = recip(pk.x == 0.0 ? 1.0 : pk.x);
  const double t = pk.y * r0;
  const double d1 = pk1.y - t * pk.y;
  const double r1 = recip(d1 == 0.0 ? 1.0 : d1);
  // natural-order pivots P_00 and d1; NaN compares false and is flagged too
  small |= !(fabs(pk.x) >= kSweepMinPivot && fabs(d1) >= kSweepMinPivot);
  double2 cj[NB];  // (c0_j, c1'_j)
#pragma unroll
  for (int jb = 0; jb < NB; ++jb) {
    const double2 c = col[tx + 16 * jb];
    cj[jb] = make_double2(c.x, c.y - t * c.x);
  }
  const bool colk = tx == kt || tx == kt + 1;  // this lane owns column k or k + 1 (block KB)
#pragma unroll
  for (int ib = 0; ib < NB; ++ib) {
    const double2 ci = col[ty + 16 * ib];
    const double g0 = ci.x * r0, g1 = (ci.y - t * ci.x) * r1;
#pragma unroll
    for (int jb = 0; jb <= ib; ++jb) {
      double& v = a[lt(ib, jb)];
      v -= g0 * cj[jb].x;
      v -= g1 * cj[jb].y;
      if (jb == KB && colk) v = tx == kt ? g0 - t * g1 : g1;  // A_iK = c_i inv(P)
    }
  }
  if (ty == kt || ty == kt + 1) {  // rows k, k + 1: warp-uniform
    const bool row1 = ty != kt;
#pragma unroll
    for (int jb = 0; jb <= KB; ++jb) {
      const double g0 = cj[jb].x * r0, g1 = cj[jb].y * r1;
      double w = row1 ? g1 : g0 - t * g1;  // A_Kj = inv(P) c_j^T
      if (jb == KB && colk)                // -inv(P)
        w = row1 ? (tx == kt ? t * r1 : -r1) : (tx == kt ? -(r0 + t * t * r1) : t * r1);
      a[lt(KB, jb)] = w;
    }
  }
  const int k2 = k + 2;
  if (k2 < n) {
    double2* out = s.col[buf ^ 1];
    if (kt + 2 < 16) sweep_publish<NB, KB>(a, k2, tx, ty, out);
    else if (KB + 1 < NB) sweep_publish<NB, (KB + 1 < NB ? KB + 1 : 0)>(a, k2, tx, ty, out);
  }
  __syncthreads();
}

// TW: arithmetic of the reduction that reads the workspace (the point stride depends on it).
template <int NB, typename TW>
__global__ void __launch_bounds__(256, 2) sweep_kernel(const float2* __restrict__ coh, PointSet pts, int n,
                                                       unsigned char* __restrict__ ws, uint8_t* __restrict__ sing) {
  constexpr int NP = NB * (NB + 1) / 2;
  __shared__ SweepShared<NB> ss;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = blockIdx.x; pt < npt; pt += gridDim.x) {
    const float2* c = coh + pts[pt] * npairs;
    if (tid == 0 && pt + gridDim.x < npt) {  // the next point's coherence into L2 (the part
      // between its first and last 16-byte boundaries; 2 % faster than without)
      const uintptr_t a0 = reinterpret_cast<uintptr_t>(coh + pts[pt + gridDim.x] * npairs);
      const uintptr_t lo = (a0 + 15) & ~uintptr_t(15), hi = (a0 + npairs * 8) & ~uintptr_t(15);
      if (hi > lo) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned)(hi - lo)) : "memory");
    }
    double a[NP];
    // |Gamma| (identity on the padding), lower triangle; a block row's loads are issued
    // together, then converted (7 % faster than loading and converting value by value, which
    // left one L2 round trip per value on the thread's path)
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
      const int i = ty + 16 * ib;
      float2 g[NB];
#pragma unroll
      for (int jb = 0; jb <= ib; ++jb) {
        const int j = tx + 16 * jb;
        g[jb] = (i < n && j < n && i > j) ? c[triu_index(j, i, n)] : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int jb = 0; jb <= ib; ++jb) {
        const int j = tx + 16 * jb;
        a[lt(ib, jb)] = (i == j) ? 1.0 : sqrt((double)g[jb].x * g[jb].x + (double)g[jb].y * g[jb].y);
      }
    }
    sweep_publish<NB, 0>(a, 0, tx, ty, ss.col[0]);
    __syncthreads();
    bool small = false;
#pragma unroll 1
    for (int kb = 0; kb < NB; ++kb) {
      for (int kt = 0; kt < 16; kt += 2) {
        const int k = 16 * kb + kt;
        if (k >= n) break;
        switch (kb) {  // compile-time block for each kb
          case 0: sweep_pair<NB, 0>(a, k, n, tx, ty, small, ss); break;
          case 1: if (NB > 1) sweep_pair<NB, (1 < NB ? 1 : 0)>(a, k, n, tx, ty, small, ss); break;
          case 2: if (NB > 2) sweep_pair<NB, (2 < NB ? 2 : 0)>(a, k, n, tx, ty, small, ss); break;
          case 3: if (NB > 3) sweep_pair<NB, (3 < NB ? 3 : 0)>(a, k, n, tx, ty, small, ss); break;
          case 4: if (NB > 4) sweep_pair<NB, (4 < NB ? 4 : 0)>(a, k, n, tx, ty, small, ss); break;
          case 5: if (NB > 5) sweep_pair<NB, (5 < NB ? 5 : 0)>(a, k, n, tx, ty, small, ss); break;
          case 6: if (NB > 6) sweep_pair<NB, (6 < NB ? 6 : 0)>(a, k, n, tx, ty, small, ss); break;
          default: if (NB > 7) sweep_pair<NB, (7 < NB ? 7 : 0)>(a, k, n, tx, ty, small, ss); break;
        }
      }
    }
    // every thread saw the same pivots: `small` is uniform
    double* out = PointPtr<TW, double>(ws, pt, n).ainv;
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
      const int i = ty + 16 * ib;
#pragma unroll
      for (int jb = 0; jb <= ib; ++jb) {
        const int j = tx + 16 * jb;
        if (i < n && j <= i) out[tri_up(j, i, n)] = -a[lt(ib, jb)];  // inv = -A after the sweep
      }
    }
    if (tid == 0) sing[pt] = small ? kRouteCond : 0;
    __syncthreads();
  }
}

// ----------------------------------------------------------------- kernel 2: reduction
// Householder reduction of M = inv(|Gamma|) o Gamma to a Hermitian tridiagonal (d, e), M in
// shared memory as a packed lower triangle ((i, j <= i) at tri(i) + j). One CTA per point, two
// barriers per step k:
//   A. warp 0 (lane l owns rows l + 32 t): p = tau M u of step k-1 from its partial sums, K = tau/2
//      u^H p, w = p - K u; column k brought up to date; reflector u_k, tau_k from it.
//   B. every warp, over strips of R rows per half-warp (longest first): step k-1's rank-2 update of
//      the rows > k and, on the updated values, both parts of M u_k: the rows' sums over the 16
//      lanes, and the columns' sums of conj(M_ij) u_i, which stay in the lane that owns column j
//      (lanes run along columns k + 1 + lane % 16 + 16 q) until the warp is through its strips.
// Every element is read and written once per step and a row's vectors are read once per strip;
// partial sums are added in a fixed order, so results do not depend on timing. Blocks of 16 columns
// that meet the diagonal run unmasked over the next rows' entries, keep what is theirs and count half
// of the diagonal in either part. Bound by latency: the chain of A (two warp sums, roots and
// divisions) and the short strips of B, hidden only by the other CTAs of the SM. The previous form
// (256 threads, three barriers, groups of four threads on mirrored row pairs, row and column parts in
// separate passes over M): FP32, N = 17, 2,047 points 146 us, now 37; N = 50, 35,627 points 8.4 ms,
// now 3.4; N = 100, 286,294 points 199 ms, now 178; FP64, N = 17, 1,003 points 157 us, now 38; N = 100,
// 4,001 points 6.2 ms, now 5.8.
// Shared memory: the triangle, 16 entries that reads past the end of its last row may touch, (u, w)
// of step k-1 and u_k with kRowPad entries in front (rows above the first of a strip), and each
// warp's part of M u.
constexpr int kRowPad = 8, kColPad = 16;
__host__ __device__ inline size_t reduce_tri(int n) { return (size_t)n * (n + 1) / 2 + kColPad; }
template <typename T>
__host__ __device__ inline size_t reduce_smem(int n, int warps, bool tri_in) {
  return ((tri_in ? reduce_tri(n) : 0) + 3 * (size_t)(n + kRowPad + kColPad) + (size_t)warps * n) *
         sizeof(typename C2<T>::type);
}

template <typename C> struct alignas(2 * sizeof(C)) Pair {
  C u, w;
};

template <typename T, typename TA, int QC, int R, int W, bool kTriIn = true>
__global__ void __launch_bounds__(32 * W, W >= 4 && QC <= 8 ? 16 / W : 1)
    reduce_kernel(const float2* __restrict__ coh, PointSet pts, int n, unsigned char* __restrict__ ws,
                  typename C2<T>::type* __restrict__ slices) {
  using C = typename C2<T>::type;
  constexpr int Q = (QC + 1) / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, lc = lane & 15, wid = tid >> 5;
  constexpr int nw = W;
  Pair<C>* uw = reinterpret_cast<Pair<C>*>(smem_raw) + kRowPad;  // u_{k-1}, w_{k-1}
  C* uc = reinterpret_cast<C*>(uw + n + kColPad) + kRowPad;      // u_k
  C* part = uc + n + kColPad;                                    // [warps][n]: each warp's part of M u
  C* L = kTriIn ? part + nw * n : slices + blockIdx.x * reduce_tri(n);
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int e = tid; e < kRowPad; e += blockDim.x) {
    uw[-1 - e] = {mk<T>(0, 0), mk<T>(0, 0)};
    uc[-1 - e] = mk<T>(0, 0);
  }
  for (int e = tid; e < kColPad; e += blockDim.x) {
    uw[n + e] = {mk<T>(0, 0), mk<T>(0, 0)};
    uc[n + e] = mk<T>(0, 0);
    L[tri(n) + e] = mk<T>(0, 0);
  }
  for (int64_t pt = blockIdx.x; pt < npt; pt += gridDim.x) {
    const float2* c = coh + pts[pt] * npairs;
    PointPtr<T, TA> w(ws, pt, n);
    // M along the upper triangle (inverse and coherence both contiguous there), a warp per row;
    // M_jm = conj(M_mj)
    for (int m = wid; m < n; m += nw) {
      const TA* ai = w.ainv + (tri_up(m, m, n) - m);
      const float2* ci = c + (triu_index(m, m + 1, n) - (m + 1));
      for (int j = m + lane; j < n; j += 32) {
        const TA sc = ai[j];
        const float2 g = j == m ? make_float2(1.f, 0.f) : ci[j];
        L[tri(j) + m] = mk<T>((T)(sc * g.x), (T)(sc * -g.y));
      }
    }
    C u[Q];  // warp 0: u_{k-1}, rows lane + 32 t
#pragma unroll
    for (int t = 0; t < Q; ++t) u[t] = mk<T>(0, 0);
    T tau_prev = 0;
    __syncthreads();
    for (int k = 0; k + 1 < n; ++k) {
      if (wid == 0) {
        C wr[Q];
        T dot = 0;
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const int i = lane + 32 * t;
          wr[t] = mk<T>(0, 0);
          if (tau_prev != T(0) && i >= k && i < n) {
            C p = part[i];
            for (int q = 1; q < nw; ++q) p = cadd(p, part[q * n + i]);
            wr[t] = mk<T>(tau_prev * p.x, tau_prev * p.y);
            dot += u[t].x * wr[t].x + u[t].y * wr[t].y;
          }
        }
        const T K = T(0.5) * tau_prev * warp_sum(dot);
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const int i = lane + 32 * t;
          wr[t].x -= K * u[t].x;
          wr[t].y -= K * u[t].y;
          if (i < n) uw[i] = {u[t], wr[t]};
        }
        __syncwarp();
        const Pair<C> at_k = uw[k];
        C x[Q];
        T xn2 = 0;
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const int i = lane + 32 * t;
          x[t] = mk<T>(0, 0);
          if (i >= k && i < n) {
            x[t] = L[tri(i) + k];
            rank2(x[t], u[t], at_k.w, wr[t], at_k.u);
          }
          if (i >= k + 2) xn2 += x[t].x * x[t].x + x[t].y * x[t].y;
        }
        xn2 = warp_sum(xn2);
        C alpha = x[0];
#pragma unroll
        for (int t = 1; t < Q; ++t)
          if ((k + 1) >> 5 == t) alpha = x[t];
        alpha.x = __shfl_sync(0xffffffffu, alpha.x, (k + 1) & 31);
        alpha.y = __shfl_sync(0xffffffffu, alpha.y, (k + 1) & 31);
        T tau = 0;
        C ek = alpha, v1 = alpha;
        if (xn2 != T(0)) {
          // e_k = -alpha nrm / |alpha|, v_1 = alpha (1 + nrm / |alpha|), tau = 1 / (nrm (nrm + |alpha|)): the
          // two roots and the two divisions side by side
          const T a2 = alpha.x * alpha.x + alpha.y * alpha.y;
          const T aa = sqrt(a2), nrm = sqrt(a2 + xn2);
          tau = T(1) / (nrm * (nrm + aa));
          const T f = nrm / aa;
          if (aa > T(0)) {
            ek = mk<T>(-alpha.x * f, -alpha.y * f);
            v1 = mk<T>(alpha.x - ek.x, alpha.y - ek.y);
          } else {
            ek = mk<T>(-nrm, 0);
            v1 = mk<T>(nrm, 0);
          }
        }
        C* refl = w.refl + refl_off(k, n) - (k + 1);
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const int i = lane + 32 * t;
          if (i == k) w.d[k] = x[t].x;
          if (k + 2 == n && i == n - 1) {  // the last step: what is left of the diagonal
            C a = L[tri(i) + i];
            rank2(a, u[t], wr[t], wr[t], u[t]);
            w.d[i] = a.x;
            w.tau[i] = T(0);
          }
          u[t] = i == k + 1 ? v1 : x[t];
          if (i <= k || tau == T(0)) u[t] = mk<T>(0, 0);
          if (i < n) uc[i] = u[t];
          if (i > k && i < n && k + 2 < n) refl[i] = u[t];
        }
        if (lane == 0) {
          w.e[k] = ek;
          w.tau[k] = tau;
        }
        tau_prev = tau;
      }
      if (k + 2 == n) break;
      __syncthreads();
      // ---- B
      C* mine = part + wid * n;
      C acc[QC];  // column sums, of columns k + 1 + lc + 16 q
#pragma unroll
      for (int q = 0; q < QC; ++q) acc[q] = mk<T>(0, 0);
      const Pair<C>* cuw = uw + (k + 1 + lc);
      const C* cuc = uc + (k + 1 + lc);
      for (int top = n - 1 - 2 * R * wid; top > k; top -= 2 * R * nw) {
        const int hi = top - R * (lane >> 4);  // this half-warp's strip: rows hi - R + 1 .. hi
        Pair<C> rv[R];
        C rc[R], sum[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          rv[r] = uw[hi - r];
          rc[r] = uc[hi - r];
          sum[r] = mk<T>(0, 0);
        }
        C* row0 = L + tri(hi) + (k + 1 + lc);
        // row hi - r starts r hi - r (r - 1) / 2 entries earlier
#pragma unroll
        for (int q = 0; q < QC; ++q) {
          const int j0 = k + 1 + 16 * q;
          if (j0 > top) break;
          const Pair<C> cv = cuw[16 * q];
          const C cc = cuc[16 * q];
          if (j0 + 15 < top - (2 * R - 1)) {  // all lanes left of every diagonal of the two strips
#pragma unroll
            for (int r = 0; r < R; ++r) {
              C* e = row0 - (r * hi - r * (r - 1) / 2) + 16 * q;
              C a = *e;
              rank2(a, rv[r].u, cv.w, rv[r].w, cv.u);
              *e = a;
              cmac(sum[r], a, cc);
              cmacc(acc[q], a, rc[r]);
            }
          } else {
            const int left = hi - (j0 + lc);  // of row hi's diagonal
#pragma unroll
            for (int r = 0; r < R; ++r) {
              C* e = row0 - (r * hi - r * (r - 1) / 2) + 16 * q;
              C a = *e;  // past the diagonal: the next row's, not kept
              rank2(a, rv[r].u, cv.w, rv[r].w, cv.u);
              if (left >= r) *e = a;
              // half of the diagonal in either part, nothing beyond it
              a.x = left > r ? a.x : left == r ? T(0.5) * a.x : T(0);
              a.y = left > r ? a.y : T(0);
              cmac(sum[r], a, cc);
              cmacc(acc[q], a, rc[r]);
            }
          }
        }
        const C tot = half_warp_sum(sum);
        const int i = hi - (lane & 15) / (16 / R);
        if (lane % (16 / R) == 0 && i > k) mine[i] = tot;
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        const int j = k + 1 + lc + 16 * q;
        acc[q] = cadd(acc[q], shfl_xor_c(acc[q], 16));
        if (lane < 16 && j < n) {
          if (((n - 1 - j) / (2 * R)) % nw == wid) acc[q] = cadd(acc[q], mine[j]);  // a row of this warp's strips
          mine[j] = acc[q];
        }
      }
      __syncthreads();
    }
    __syncthreads();  // L and the vectors are rewritten for the next point
  }
}

// Reflector k of a point (its scalar and the lane's four entries, zero past its end) into
// registers.
template <typename T, typename TA, int NR>
__device__ __forceinline__ void load_refl(const PointPtr<T, TA>& w, int n, int k, int lane,
                                          typename C2<T>::type (&u)[NR], T& tau) {
  tau = w.tau[k];
  const typename C2<T>::type* src = w.refl + refl_off(k, n);
  const int m = n - k - 1;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    const int i = lane + 32 * t;
    u[t] = i < m ? src[i] : mk<T>(0, 0);
  }
}

// ----------------------------------------------------------------- kernel 3: tail, one warp per point
constexpr int kTailWarps = 8;

template <typename T>
__host__ __device__ inline size_t tail_warp_bytes(int n) {
  using C = typename C2<T>::type;
  return align16(6 * (size_t)n * sizeof(T)) + align16((size_t)n * sizeof(C)) + align16((size_t)n * sizeof(double2));
}

// NR: rows per lane (32 NR >= n); W warps per CTA.
template <typename T, typename TA, int NR, int W>
__global__ void __launch_bounds__(32 * W, NR <= 4 ? 3 : 1) tail_kernel(const float2* __restrict__ coh, PointSet pts, int n,
                                                              int ref, const unsigned char* __restrict__ ws,
                                                              const uint8_t* __restrict__ sing,
                                                              float2* __restrict__ ph, float* __restrict__ quality,
                                                              float* __restrict__ tcoh) {
  using C = typename C2<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char* mine = smem_raw + (size_t)wid * tail_warp_bytes<T>(n);
  T* d = reinterpret_cast<T*>(mine);
  T* b = d + n;
  T* b2 = b + n;
  T* y = b2 + n;
  T* w1 = y + n;
  T* w2 = w1 + n;
  C* z = reinterpret_cast<C*>(mine + align16(6 * (size_t)n * sizeof(T)));
  double2* phs = reinterpret_cast<double2*>(mine + align16(6 * (size_t)n * sizeof(T)) + align16((size_t)n * sizeof(C)));
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const float fnan = __int_as_float(0x7fffffff);
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * W + wid; pt < npt; pt += (int64_t)gridDim.x * W) {
    const int64_t gp = pts[pt];
    const PointPtr<T, TA> w(const_cast<unsigned char*>(ws), pt, n);
    // real tridiagonal: b = |e|, phases delta_{k+1} = delta_k e_k/|e_k| (warp prefix product)
    C carry = mk<T>(1, 0);
    for (int k0 = 0; k0 < n; k0 += 32) {
      const int k = k0 + lane;
      if (k < n) d[k] = w.d[k];
      C f = mk<T>(1, 0);
      if (k + 1 < n) {
        const C ek = w.e[k];
        const T a = sqrt(ek.x * ek.x + ek.y * ek.y);
        b[k] = a;
        b2[k] = a * a;
        if (a > T(0)) f = mk<T>(ek.x / a, ek.y / a);
      }
      // inclusive scan of the factors f over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const T ox = __shfl_up_sync(0xffffffffu, f.x, o), oy = __shfl_up_sync(0xffffffffu, f.y, o);
        if (lane >= o) f = cmul_t(mk<T>(ox, oy), f);
      }
      const C dl = cmul_t(carry, f);  // delta_{k+1}
      if (k0 == 0 && lane == 0) z[0] = mk<T>(1, 0);
      if (k + 1 < n) z[k + 1] = dl;
      carry = mk<T>(__shfl_sync(0xffffffffu, dl.x, 31), __shfl_sync(0xffffffffu, dl.y, 31));
    }
    __syncwarp();
    // lambda_min by multisection
    T lo = Lim<T>::huge(), hi = -Lim<T>::huge(), tnorm = 0;
    for (int i = lane; i < n; i += 32) {
      const T r = (i > 0 ? b[i - 1] : T(0)) + (i + 1 < n ? b[i] : T(0));
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
      tnorm = fmax(tnorm, fabs(d[i]) + r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
    }
    const T eps = Lim<T>::eps();
    const T pivmin = fmax(Lim<T>::tiny(), eps * eps * tnorm * tnorm) + Lim<T>::tiny();
    const T pad = T(2) * eps * fmax(tnorm, Lim<T>::tiny()) + T(2) * pivmin;
    lo -= pad;
    hi += pad;
    for (int it = 0; it < 64; ++it) {
      const T width = hi - lo;
      if (!(width > T(2) * eps * fmax(fabs(lo), fabs(hi)) + T(4) * pivmin)) break;
      const T sg = lo + width * (T)(lane + 1) / T(33);
      const int cnt = sturm_count(d, b2, n, sg, pivmin);
      const unsigned ball = __ballot_sync(0xffffffffu, cnt >= 1);
      const int first = ball ? __ffs(ball) - 1 : 32;
      const T nlo = (first == 0) ? lo : lo + width * (T)first / T(33);
      const T nhi = (first == 32) ? hi : lo + width * (T)(first + 1) / T(33);
      lo = nlo;
      hi = nhi;
    }
    const T lam = T(0.5) * (lo + hi);
    // eigenvector of the real tridiagonal by inverse iteration (lane 0)
    for (int i = lane; i < n; i += 32) y[i] = T(1) + T(0.25) * (T)((i * 37) % 11) / T(11);
    __syncwarp();
    if (lane == 0) {
      const T tiny = eps * fmax(tnorm, Lim<T>::tiny());
      for (int it = 0; it < 2; ++it) {
        tridiag_solve(d, b, n, lam, tiny, y, w1, w2, b2);  // b2 is free after the bisection
        T sc = 0;
        for (int i = 0; i < n; ++i) sc = fmax(sc, fabs(y[i]));
        if (!(sc > T(0)) || !isfinite(sc)) break;
        const T r = T(1) / sc;
        for (int i = 0; i < n; ++i) y[i] *= r;
      }
    }
    __syncwarp();
    // v = Q D y
    for (int i = lane; i < n; i += 32) { const C dl = z[i]; z[i] = mk<T>(dl.x * y[i], dl.y * y[i]); }
    __syncwarp();
    // reflectors applied from the last; the next one's values are loaded while the current
    // one is applied, so the serial chain does not wait on memory
    {
      C uu[NR], nu[NR];
      T tau = 0, ntau = 0;
      if (n >= 3) load_refl(w, n, n - 3, lane, uu, tau);
      for (int k = n - 3; k >= 0; --k) {
        if (k > 0) load_refl(w, n, k - 1, lane, nu, ntau);
        if (tau != T(0)) {
          const int m = n - k - 1;
          C sacc = mk<T>(0, 0);
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            const int i = lane + 32 * t;
            if (i < m) {
              const C zi = z[k + 1 + i];
              sacc.x += uu[t].x * zi.x + uu[t].y * zi.y;
              sacc.y += uu[t].x * zi.y - uu[t].y * zi.x;
            }
          }
          sacc.x = warp_sum(sacc.x);
          sacc.y = warp_sum(sacc.y);
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            const int i = lane + 32 * t;
            if (i < m) {
              const C tt = cmul_t(uu[t], sacc);
              z[k + 1 + i].x -= tau * tt.x;
              z[k + 1 + i].y -= tau * tt.y;
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int t = 0; t < NR; ++t) uu[t] = nu[t];
        tau = ntau;
      }
    }
    // normalise to the reference image
    const bool singular = (sing[pt] & kRouteSingular) != 0;
    const C zr = z[ref];
    for (int i = lane; i < n; i += 32) {
      const C v = cmulc_t(z[i], zr);
      const double vx = v.x, vy = v.y, a = sqrt(vx * vx + vy * vy);
      float2 o = make_float2((float)(vx / a), (float)(vy / a));
      if (singular) o = make_float2(fnan, fnan);
      ph[gp * n + i] = o;
      phs[i] = make_double2(o.x, o.y);
    }
    if (lane == 0) quality[gp] = singular ? fnan : (float)lam;
    __syncwarp();
    if (tcoh) {  // |sum_q coh_q/|coh_q| conj(ph_m) ph_j| / n_pairs
      const float2* c = coh + gp * npairs;
      double tx = 0, ty = 0;
      int mm = 0, jj = 1 + lane;
      while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
      for (int64_t q = lane; q < npairs; q += 32) {
        const int m0 = mm, j0 = jj;
        jj += 32;
        while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
        const float2 g = c[q];
        const double ga = sqrt((double)g.x * g.x + (double)g.y * g.y);
        const double2 v = cmul(make_double2(g.x / ga, g.y / ga), cmulc(phs[j0], phs[m0]));
        tx += v.x;
        ty += v.y;
      }
      tx = warp_sum(tx);
      ty = warp_sum(ty);
      if (lane == 0) tcoh[gp] = (float)(sqrt(tx * tx + ty * ty) / (double)npairs);
    }
    __syncwarp();
  }
}


// ----------------------------------------------------------------- kernel 3b: refined tail
// For the refined mixed precision (FP64 inverse, FP32 reduction): the FP32 eigenvector is
// improved by one step of a Newton (Jacobi-Davidson) correction in FP64,
//   r = M v - lambda v (lambda = v^H M v, M = inv(|Gamma|) o Gamma from the FP64 inverse),
//   (M - lambda I) dv = r solved approximately through the FP32 factors M ~ Q D R D^H Q^H,
//   dv = Q D P (R - lambda I)^-1 P D^H Q^H r, P the projector orthogonal to R's eigenvector,
// which divides the error by about eps32 ||M|| / gap. Then the refined pair is checked in
// FP64: with residual r', gap g = lambda_2(R) - lambda and smallest component |v_i|, the
// phase error of every date is at most |r'| / (g min|v_i|); points above `tol` are flagged
// for an FP64 recomputation. One warp per point.
constexpr int kRefineWarps = 4;

__host__ __device__ inline size_t refine_warp_bytes(int n) {
  return align16(6 * (size_t)n * sizeof(float)) + align16(6 * (size_t)n * sizeof(double)) +
         3 * align16((size_t)n * sizeof(double2));
}

// Solve (R - lambda I) x = y in place, R real symmetric tridiagonal (d, b), by elimination
// with row interchanges, for a real (V = T) or complex (V = C2<T>) right-hand side. Each
// row's final pivot is inverted once and kept in dd, so the back substitution multiplies:
// one reciprocal per row on the serial chain instead of a division per row and component.
// dd, du, dl: work arrays of length n; dl ends as the second super-diagonal of each row.
template <typename T> __device__ __forceinline__ void axpy_r(T& y, T f, const T& x) { y -= f * x; }
template <typename T> __device__ __forceinline__ void axpy_r(typename C2<T>::type& y, T f,
                                                              const typename C2<T>::type& x) {
  y.x -= f * x.x;
  y.y -= f * x.y;
}
template <typename T> __device__ __forceinline__ void scale_r(T& y, T f) { y *= f; }
template <typename T> __device__ __forceinline__ void scale_r(typename C2<T>::type& y, T f) {
  y.x *= f;
  y.y *= f;
}

template <typename T, typename V>
__device__ inline void tridiag_solve_rcp(const T* d, const T* b, int n, T lambda, T tiny, V* y, T* dd, T* du,
                                         T* dl) {
  for (int i = 0; i < n; ++i) {
    dd[i] = d[i] - lambda;
    if (i < n - 1) { du[i] = b[i]; dl[i] = b[i]; }
  }
  for (int i = 0; i < n - 1; ++i) {
    const T sub = dl[i];
    if (fabs(dd[i]) >= fabs(sub)) {
      if (dd[i] == T(0)) dd[i] = tiny;
      const T r = recip(dd[i]);
      const T f = sub * r;
      dd[i + 1] -= f * du[i];
      axpy_r<T>(y[i + 1], f, y[i]);
      dl[i] = T(0);
      dd[i] = r;
    } else {
      const T r = recip(sub);
      const T f = dd[i] * r;
      const T t = dd[i + 1];
      dd[i + 1] = du[i] - f * t;
      if (i < n - 2) {
        dl[i] = du[i + 1];
        du[i + 1] = -f * dl[i];
      } else {
        dl[i] = T(0);
      }
      du[i] = t;
      const V ty = y[i];
      y[i] = y[i + 1];
      y[i + 1] = ty;
      axpy_r<T>(y[i + 1], f, y[i]);
      dd[i] = r;
    }
  }
  if (dd[n - 1] == T(0)) dd[n - 1] = tiny;
  scale_r<T>(y[n - 1], recip(dd[n - 1]));
  if (n > 1) {
    axpy_r<T>(y[n - 2], du[n - 2], y[n - 1]);
    scale_r<T>(y[n - 2], dd[n - 2]);
  }
  for (int i = n - 3; i >= 0; --i) {
    axpy_r<T>(y[i], du[i], y[i + 1]);
    axpy_r<T>(y[i], dl[i], y[i + 2]);
    scale_r<T>(y[i], dd[i]);
  }
}

// out = M v for M = inv(|Gamma|) o Gamma (Hermitian), read along the upper triangle: the
// element (m, j > m) adds M_mj v_j to row m and conj(M_mj) v_m to row j. Lanes own columns
// j = lane + 32 c; rows go four at a time through warp_sum4. One warp.
__device__ void herm_matvec(const double* __restrict__ ainv, const float2* __restrict__ c, int n,
                            const double2* v, double2* out) {
  constexpr int NC = (kMaxFastN + 31) / 32;
  const int lane = threadIdx.x & 31;
  double2 vj[NC], cacc[NC];
#pragma unroll
  for (int t = 0; t < NC; ++t) {
    const int j = lane + 32 * t;
    vj[t] = j < n ? v[j] : make_double2(0, 0);
    cacc[t] = make_double2(0, 0);
  }
  for (int m0 = 0; m0 < n; m0 += 4) {
    double2 racc[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      racc[r] = make_double2(0, 0);
      const int m = m0 + r;
      if (m >= n) continue;  // warp-uniform
      const double2 vm = v[m];
      const int64_t um = tri_up(m, m, n), qm = um - (m + 1);
#pragma unroll
      for (int t = 0; t < NC; ++t) {
        const int j = lane + 32 * t;
        if (j < m || j >= n) continue;
        const double s = ainv[um + (j - m)];
        if (j == m) {
          racc[r].x += s * vm.x;
          racc[r].y += s * vm.y;
        } else {
          const float2 g = c[qm + (j - m)];
          const double2 a = make_double2(s * (double)g.x, s * (double)g.y);  // M_mj
          cmac(racc[r], a, vj[t]);
          cmacc(cacc[t], a, vm);
        }
      }
    }
    const double2 tot = warp_sum4(racc);
    const int r = lane >> 3;
    if ((lane & 7) == 0 && m0 + r < n) out[m0 + r] = tot;
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < NC; ++t) {
    const int j = lane + 32 * t;
    if (j < n) out[j] = cadd(out[j], cacc[t]);
  }
  __syncwarp();
}

// z <- H_k z for the reflectors of the workspace, k ascending (forward, Q^H z) or
// descending (back, Q z), in the arithmetic V of z (float2 or double2); the reflectors'
// stored values are used exactly. One warp.
template <typename V, typename T, typename TA>
__device__ void apply_q(const PointPtr<T, TA>& w, int n, typename C2<V>::type* z, bool forward) {
  using C = typename C2<T>::type;
  using CV = typename C2<V>::type;
  const int lane = threadIdx.x & 31;
  if (n < 3) return;
  C cu[4], nu[4];
  T ct = 0, nt = 0;
  load_refl(w, n, forward ? 0 : n - 3, lane, cu, ct);
  for (int s = 0; s + 2 < n; ++s) {
    const int k = forward ? s : n - 3 - s;
    if (s + 3 < n) load_refl(w, n, forward ? s + 1 : n - 4 - s, lane, nu, nt);  // the next one, early
    const V tau = (V)ct;
    if (tau != V(0)) {
      const int m = n - k - 1;
      CV acc = mk<V>(0, 0), uu[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int i = lane + 32 * t;
        uu[t] = mk<V>((V)cu[t].x, (V)cu[t].y);
        if (i < m) cmacc(acc, uu[t], z[k + 1 + i]);  // u^H z
      }
      acc.x = warp_sum(acc.x);
      acc.y = warp_sum(acc.y);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int i = lane + 32 * t;
        if (i < m) {
          const CV tt = cmul(uu[t], acc);
          z[k + 1 + i].x -= tau * tt.x;
          z[k + 1 + i].y -= tau * tt.y;
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) cu[t] = nu[t];
    ct = nt;
  }
}

// Smallest sigma (to the bisection's resolution) with at least `target` eigenvalues of the
// real tridiagonal (d, b2) at or below it, by multisection over the warp from [lo, hi].
template <typename T>
__device__ T multisect(const T* d, const T* b2, int n, T lo, T hi, int target, T pivmin, int rounds) {
  const int lane = threadIdx.x & 31;
  const T eps = Lim<T>::eps();
  for (int it = 0; it < rounds; ++it) {
    const T width = hi - lo;
    if (!(width > T(2) * eps * fmax(fabs(lo), fabs(hi)) + T(4) * pivmin)) break;
    const T sg = lo + width * (T)(lane + 1) / T(33);
    const int cnt = sturm_count(d, b2, n, sg, pivmin);
    const unsigned ball = __ballot_sync(0xffffffffu, cnt >= target);
    const int first = ball ? __ffs(ball) - 1 : 32;
    const T nlo = (first == 0) ? lo : lo + width * (T)first / T(33);
    const T nhi = (first == 32) ? hi : lo + width * (T)(first + 1) / T(33);
    lo = nlo;
    hi = nhi;
  }
  return T(0.5) * (lo + hi);
}

template <typename T>
__global__ void __launch_bounds__(32 * kRefineWarps, 4) tail_refine_kernel(
    const float2* __restrict__ coh, PointSet pts, int n, int ref, const unsigned char* __restrict__ ws,
    uint8_t* __restrict__ sing, float2* __restrict__ ph, float* __restrict__ quality, float* __restrict__ tcoh,
    double tol) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char* mine = smem_raw + (size_t)wid * refine_warp_bytes(n);
  T* d = reinterpret_cast<T*>(mine);
  T* b = d + n;
  T* b2 = b + n;
  T* y = b2 + n;
  T* w1 = y + n;
  T* w2 = w1 + n;
  double* dd = reinterpret_cast<double*>(mine + align16(6 * (size_t)n * sizeof(float)));
  double* bd = dd + n;
  double* yd = bd + n;
  double* s1 = yd + n;
  double* s2 = s1 + n;
  double* s3 = s2 + n;
  float2* z32 = reinterpret_cast<float2*>(s1);  // FP32 work vector; s1 is scratch only inside the solve
  double2* dph = reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(dd) + align16(6 * (size_t)n * sizeof(double)));
  double2* v = dph + n;
  double2* t1 = v + n;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const float fnan = __int_as_float(0x7fffffff);
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * kRefineWarps + wid; pt < npt; pt += (int64_t)gridDim.x * kRefineWarps) {
    const int64_t gp = pts[pt];
    const PointPtr<T, double> w(const_cast<unsigned char*>(ws), pt, n);
    const float2* c = coh + gp * npairs;
    // real tridiagonal R: b = |e|, phases delta_{k+1} = delta_k e_k/|e_k| (warp prefix product, FP64)
    double2 carry = make_double2(1, 0);
    for (int k0 = 0; k0 < n; k0 += 32) {
      const int k = k0 + lane;
      if (k < n) { d[k] = w.d[k]; dd[k] = (double)w.d[k]; }
      double2 f = make_double2(1, 0);
      if (k + 1 < n) {
        const typename C2<T>::type ek = w.e[k];
        const double ex = ek.x, ey = ek.y, a = sqrt(ex * ex + ey * ey);
        b[k] = (T)a;
        b2[k] = (T)a * (T)a;
        bd[k] = a;
        if (a > 0.0) f = make_double2(ex / a, ey / a);
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double ox = __shfl_up_sync(0xffffffffu, f.x, o), oy = __shfl_up_sync(0xffffffffu, f.y, o);
        if (lane >= o) f = cmul(make_double2(ox, oy), f);
      }
      const double2 dl = cmul(carry, f);
      if (k0 == 0 && lane == 0) dph[0] = make_double2(1, 0);
      if (k + 1 < n) dph[k + 1] = dl;
      carry = make_double2(__shfl_sync(0xffffffffu, dl.x, 31), __shfl_sync(0xffffffffu, dl.y, 31));
    }
    __syncwarp();
    // lambda_1 and lambda_2 of R (FP32 Sturm counts)
    T lo = Lim<T>::huge(), hi = -Lim<T>::huge(), tnorm = 0;
    for (int i = lane; i < n; i += 32) {
      const T r = (i > 0 ? b[i - 1] : T(0)) + (i + 1 < n ? b[i] : T(0));
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
      tnorm = fmax(tnorm, fabs(d[i]) + r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
    }
    const T eps = Lim<T>::eps();
    const T pivmin = fmax(Lim<T>::tiny(), eps * eps * tnorm * tnorm) + Lim<T>::tiny();
    const T pad = T(2) * eps * fmax(tnorm, Lim<T>::tiny()) + T(2) * pivmin;
    lo -= pad;
    hi += pad;
    const T lam1 = multisect(d, b2, n, lo, hi, 1, pivmin, 64);
    // eigenvector y of R by inverse iteration (FP32, lane 0)
    for (int i = lane; i < n; i += 32) y[i] = T(1) + T(0.25) * (T)((i * 37) % 11) / T(11);
    __syncwarp();
    if (lane == 0) {
      const T tiny = eps * fmax(tnorm, Lim<T>::tiny());
      for (int it = 0; it < 2; ++it) {
        tridiag_solve_rcp(d, b, n, lam1, tiny, y, w1, w2, b2);  // b2 is free after the bisections
        T sc = 0;
        for (int i = 0; i < n; ++i) sc = fmax(sc, fabs(y[i]));
        if (!(sc > T(0)) || !isfinite(sc)) break;
        const T r = T(1) / sc;
        for (int i = 0; i < n; ++i) y[i] *= r;
      }
    }
    __syncwarp();
    // y to unit length in FP64; v = Q D y
    double yn = 0;
    for (int i = lane; i < n; i += 32) { yd[i] = (double)y[i]; yn += yd[i] * yd[i]; }
    yn = 1.0 / sqrt(warp_sum(yn));
    for (int i = lane; i < n; i += 32) {
      yd[i] *= yn;
      z32[i] = make_float2((float)(dph[i].x * yd[i]), (float)(dph[i].y * yd[i]));
    }
    __syncwarp();
    apply_q<float>(w, n, z32, false);
    for (int i = lane; i < n; i += 32) v[i] = make_double2(z32[i].x, z32[i].y);
    __syncwarp();
    // one correction step, then the check
    double lam = 0, rn = 0;
    for (int pass = 0; pass < 2; ++pass) {
      herm_matvec(w.ainv, c, n, v, t1);
      double vmv = 0, vv = 0;
      for (int i = lane; i < n; i += 32) {
        vmv += v[i].x * t1[i].x + v[i].y * t1[i].y;
        vv += v[i].x * v[i].x + v[i].y * v[i].y;
      }
      vv = warp_sum(vv);
      lam = warp_sum(vmv) / vv;
      double r2 = 0;
      for (int i = lane; i < n; i += 32) {
        t1[i] = make_double2(t1[i].x - lam * v[i].x, t1[i].y - lam * v[i].y);
        r2 += t1[i].x * t1[i].x + t1[i].y * t1[i].y;
      }
      rn = sqrt(warp_sum(r2) / vv);
      __syncwarp();
      if (pass == 1) break;
      // dv = Q D P (R - lam I)^-1 P D^H Q^H r; the reflectors are applied in FP32 (the factors
      // hold M only to FP32 accuracy anyway), the projected solve runs in FP64
      for (int i = lane; i < n; i += 32) z32[i] = make_float2((float)t1[i].x, (float)t1[i].y);
      __syncwarp();
      apply_q<float>(w, n, z32, true);
      double2 pr = make_double2(0, 0);
      for (int i = lane; i < n; i += 32) {
        t1[i] = cmulc(make_double2(z32[i].x, z32[i].y), dph[i]);  // D^H: times conj(delta_i)
        pr.x += yd[i] * t1[i].x;
        pr.y += yd[i] * t1[i].y;
      }
      pr.x = warp_sum(pr.x);
      pr.y = warp_sum(pr.y);
      for (int i = lane; i < n; i += 32) { t1[i].x -= yd[i] * pr.x; t1[i].y -= yd[i] * pr.y; }
      __syncwarp();
      if (lane == 0) tridiag_solve_rcp(dd, bd, n, lam, DBL_EPSILON * (double)tnorm + DBL_MIN, t1, s1, s2, s3);
      __syncwarp();
      pr = make_double2(0, 0);
      for (int i = lane; i < n; i += 32) { pr.x += yd[i] * t1[i].x; pr.y += yd[i] * t1[i].y; }
      pr.x = warp_sum(pr.x);
      pr.y = warp_sum(pr.y);
      for (int i = lane; i < n; i += 32) {
        const double2 x = cmul(make_double2(t1[i].x - yd[i] * pr.x, t1[i].y - yd[i] * pr.y), dph[i]);
        z32[i] = make_float2((float)x.x, (float)x.y);
      }
      __syncwarp();
      apply_q<float>(w, n, z32, false);
      double vn = 0;
      for (int i = lane; i < n; i += 32) {
        v[i] = make_double2(v[i].x - (double)z32[i].x, v[i].y - (double)z32[i].y);
        vn += v[i].x * v[i].x + v[i].y * v[i].y;
      }
      vn = 1.0 / sqrt(warp_sum(vn));
      for (int i = lane; i < n; i += 32) v[i] = make_double2(v[i].x * vn, v[i].y * vn);
      __syncwarp();
    }
    // phase error bound of the refined vector (v has unit length)
    double vmin = 1e300;
    for (int i = lane; i < n; i += 32) vmin = fmin(vmin, sqrt(v[i].x * v[i].x + v[i].y * v[i].y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmin = fmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
    // |r'| / (gap min|v_i|) <= tol with gap = lambda_2(R) - lam - margin holds exactly when
    // lambda_2(R) >= sig = lam + margin + |r'| / (tol min|v_i|): one Sturm count at sig
    // (rounded up to FP32) answers it, without locating lambda_2
    const double sig = lam + 4.0 * (double)eps * (double)n * (double)tnorm + rn / (tol * vmin);
    for (int i = lane; i + 1 < n; i += 32) b2[i] = b[i] * b[i];  // b2 was the solves' scratch
    __syncwarp();
    float sg = (float)sig;
    if ((double)sg < sig) sg = nextafterf(sg, 3.4e38f);
    const bool gap_ok = sig < 3.0e38 && sturm_count(d, b2, n, (T)sg, pivmin) <= 1;  // NaN: false
    const bool singular = (sing[pt] & kRouteSingular) != 0;
    const bool small_pivot = (sing[pt] & kRouteCond) != 0;  // the sweep's inverse is not trusted
    const bool ok = singular || (!small_pivot && gap_ok);
    // normalise to the reference image
    const double2 zr = v[ref];
    for (int i = lane; i < n; i += 32) {
      const double2 q = cmulc(v[i], zr);
      const double a = sqrt(q.x * q.x + q.y * q.y);
      float2 o = make_float2((float)(q.x / a), (float)(q.y / a));
      if (singular) o = make_float2(fnan, fnan);
      ph[gp * n + i] = o;
      t1[i] = make_double2(o.x, o.y);
    }
    __syncwarp();
    if (lane == 0) {
      quality[gp] = singular ? fnan : (float)lam;
      sing[pt] = singular ? kRouteSingular : (ok ? 0 : kRouteCond);
    }
    if (tcoh) {  // |sum_q coh_q/|coh_q| conj(ph_m) ph_j| / n_pairs
      double tx = 0, ty = 0;
      int mm = 0, jj = 1 + lane;
      while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
      for (int64_t q = lane; q < npairs; q += 32) {
        const int m0 = mm, j0 = jj;
        jj += 32;
        while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
        const float2 g = c[q];
        const double ga = sqrt((double)g.x * g.x + (double)g.y * g.y);
        const double2 q2 = cmul(make_double2(g.x / ga, g.y / ga), cmulc(t1[j0], t1[m0]));
        tx += q2.x;
        ty += q2.y;
      }
      tx = warp_sum(tx);
      ty = warp_sum(ty);
      if (lane == 0) tcoh[gp] = (float)(sqrt(tx * tx + ty * ty) / (double)npairs);
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------- host side
template <class K>
int occupancy(K kernel, int threads, size_t smem) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess) return 0;
  return occ;
}

// Most points of a sub-batch: its per-point workspace within 4 GiB (about 34,600 points at
// N = 100), so that each launch has enough points to keep every SM busy to its end.
template <typename T>
int64_t sub_batch(int n) {
  const PointWs<T> w(n);  // FP64 sub-batches also fit the refined layout (it is smaller)
  const int64_t def = (int64_t)std::max<size_t>(1024, std::min<size_t>(1 << 17, (size_t)(1ull << 32) / (w.bytes + 1)));
  const int64_t cap = g_sub_batch_cap.load();
  return cap > 0 ? std::min(cap, def) : def;
}

// Workspace of one sub-batch of `sub` points: per-point state of the widest arithmetic
// used and the route flags of the FP32 and FP64 passes; then, for all `n_list` points of the
// call, the list of points to redo in FP64 and its count. The redo runs once after every
// sub-batch, so the few routed points of a call share launches instead of running a
// nearly empty pass per sub-batch.
struct SubWs {
  unsigned char* pts;
  uint8_t* sing;
  uint8_t* sing2;
  int32_t* list;
  int32_t* count;
  unsigned char* slices;  // above kReduceIn images: per-CTA matrices
  static size_t bytes(int64_t sub, size_t point_bytes, int64_t n_list) {
    return align16((size_t)sub * point_bytes) + 2 * align16((size_t)sub) + align16(4 * (size_t)n_list) + 16;
  }
  SubWs(unsigned char* ws, int64_t sub, size_t point_bytes, int64_t n_list) {
    unsigned char* b = ws;
    pts = b;
    b += align16((size_t)sub * point_bytes);
    sing = b;
    b += align16((size_t)sub);
    sing2 = b;
    b += align16((size_t)sub);
    list = reinterpret_cast<int32_t*>(b);
    b += align16(4 * (size_t)n_list);
    count = reinterpret_cast<int32_t*>(b);
    slices = b + 16;
  }
};

// Appends the points of a sub-batch (global indices b0 + i) that are to be redone in FP64 to
// the list. `refined`: points singular in the (already FP64) inverse are not redone. With a
// device-held point count (dcount, the sub-batch starting at point doff of it) only the
// points below it are read.
__global__ void route_kernel(const uint8_t* __restrict__ sing, int64_t nb, int64_t b0, int32_t* __restrict__ list,
                             int32_t* __restrict__ count, uint8_t* __restrict__ route, bool refined,
                             const int64_t* __restrict__ dcount, int64_t doff) {
  if (dcount) {
    const int64_t c = *dcount - doff;
    nb = c < 0 ? 0 : (c < nb ? c : nb);
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t f = sing[i];
    if (route) route[i] = f;
    if (f && !(refined && f == kRouteSingular)) list[atomicAdd(count, 1)] = (int32_t)(b0 + i);  // order is free
  }
}

// Column groups of the Gauss-Jordan grid. 32 groups (512 threads, half the registers per
// thread) measured no faster than 16 in FP32 or FP64: one point per SM either way, and its
// serial pivot steps set the pace. With look-ahead pivoting the 512-thread tile stayed in
// local memory (128 registers per thread), twice as slow.
template <typename T>
constexpr int gj_cx() { return 16; }

template <typename T, int NB, typename TW>
int launch_inverse(const float2* coh, PointSet pts, int64_t grid_cap, int n, unsigned char* ws, uint8_t* sing,
                   float cond_max, cudaStream_t s) {
  constexpr int CX = gj_cx<T>();
  const int occ = std::max(1, occupancy(inverse_kernel<T, NB, CX, TW>, 16 * CX, 0));
  const int64_t grid = std::min<int64_t>(grid_cap, (int64_t)sm_count() * occ);
  KernelTimer kt(pts.list ? "emi inverse rerun" : sizeof(T) == 8 ? "emi inverse fp64" : "emi inverse fp32", s);
  inverse_kernel<T, NB, CX, TW><<<(unsigned)grid, 16 * CX, 0, s>>>(coh, pts, n, ws, sing, cond_max);
  return check_launch("emi inverse");
}

// inv(|Gamma|) in arithmetic TA into a workspace laid out for a reduction in T.
// Most images with the reduction's FP64 triangle in shared memory.
constexpr int kReduceIn = 158;

template <int Q, bool kIn>
int launch_big_inverse(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, void* slices,
                       cudaStream_t s) {
  const size_t smem = kIn ? (size_t)n * (n | 1) * sizeof(double) : 0;
  auto kernel = big_inverse_kernel<Q, kIn>;
  if (int rc = allow_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  KernelTimer kt("emi inverse fp64", s);
  kernel<<<(unsigned)std::min<int64_t>(pts.n_pc, sm_count()), kBigThreads, smem, s>>>(c, pts, n, ws, sing,
                                                                                     static_cast<double*>(slices));
  return check_launch("emi inverse");
}

int run_big_inverse(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, void* slices,
                    cudaStream_t s) {
  if (n <= kBigIn) return launch_big_inverse<5, true>(c, pts, n, ws, sing, slices, s);
  if (n <= 192) return launch_big_inverse<6, false>(c, pts, n, ws, sing, slices, s);
  if (n <= 256) return launch_big_inverse<8, false>(c, pts, n, ws, sing, slices, s);
  return launch_big_inverse<16, false>(c, pts, n, ws, sing, slices, s);
}

// Bytes of one CTA's slice (inverse: n x n; reduction: its triangle), one per SM; none where both
// kernels have their matrix in shared memory.
size_t slice_bytes(int n) {
  if (n <= kReduceIn) return 0;
  return align16(std::max((size_t)n * n * sizeof(double), reduce_tri(n) * sizeof(double2)));
}

template <typename TA, typename T>
int run_inverse(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, float cond_max,
                cudaStream_t s) {
  const int64_t cap = pts.n_pc;  // grid bound: the most points this pass can see
  switch ((n + 15) / 16) {
    case 1: case 2: return launch_inverse<TA, 2, T>(c, pts, cap, n, ws, sing, cond_max, s);
    case 3: return launch_inverse<TA, 3, T>(c, pts, cap, n, ws, sing, cond_max, s);
    case 4: return launch_inverse<TA, 4, T>(c, pts, cap, n, ws, sing, cond_max, s);
    case 5: return launch_inverse<TA, 5, T>(c, pts, cap, n, ws, sing, cond_max, s);
    case 6: return launch_inverse<TA, 6, T>(c, pts, cap, n, ws, sing, cond_max, s);
    case 7: return launch_inverse<TA, 7, T>(c, pts, cap, n, ws, sing, cond_max, s);
    default: return launch_inverse<TA, 8, T>(c, pts, cap, n, ws, sing, cond_max, s);
  }
}

template <typename T, typename TA, int QC, int R, int W, bool kTriIn = true>
int launch_reduce(const float2* c, PointSet pts, int n, unsigned char* ws, cudaStream_t s,
                  typename C2<T>::type* slices = nullptr) {
  const size_t rsmem = reduce_smem<T>(n, W, kTriIn);
  auto kernel = reduce_kernel<T, TA, QC, R, W, kTriIn>;
  if (int rc_ = allow_smem(reinterpret_cast<const void*>(kernel), rsmem)) return rc_;
  const int rocc = occupancy(kernel, 32 * W, rsmem);
  if (rocc < 1) return fail(MR_ERR_UNSUPPORTED, "emi: %zu bytes of shared memory per CTA do not fit", rsmem);
  KernelTimer kt(pts.list ? "emi reduce rerun" : sizeof(T) == 8 ? "emi reduce fp64" : "emi reduce fp32", s);
  // one slice of the workspace per SM where the triangle is not in shared memory
  const int64_t most = (int64_t)sm_count() * (kTriIn ? rocc : 1);
  kernel<<<(unsigned)std::min<int64_t>(pts.n_pc, most), 32 * W, rsmem, s>>>(c, pts, n, ws, slices);
  return check_launch("emi reduce");
}

template <typename T, typename TA>
int run_reduce(const float2* c, PointSet pts, int n, unsigned char* ws, cudaStream_t s) {
  // Warps per point and rows per half-warp strip. Up to 64 images one warp (FP64: two above 32)
  // needs no or little waiting on other warps and an SM holds many points; above, shared memory
  // holds two to four points per SM, and more warps each hide their latencies: N = 100, FP32, 1, 2, 4,
  // 8 warps of 4 rows: 243, 222, 178, 285 ms for 286,294 points; FP64, 4 and 8 warps of 4 rows 6.5 and
  // 6.2, of 2 rows (128 registers, two CTAs of 8 warps) 6.4 and 5.8 ms for 4,001 points.
  constexpr bool f64 = sizeof(T) == 8;
  constexpr int W4 = f64 ? 2 : 1, W8 = f64 ? 8 : 4, R8 = f64 ? 2 : 4;
  switch ((n + 15) / 16) {
    case 1: return launch_reduce<T, TA, 1, 4, 1>(c, pts, n, ws, s);
    case 2: return launch_reduce<T, TA, 2, 4, 1>(c, pts, n, ws, s);
    case 3: return launch_reduce<T, TA, 3, 4, W4>(c, pts, n, ws, s);
    case 4: return launch_reduce<T, TA, 4, 4, W4>(c, pts, n, ws, s);
    case 5: return launch_reduce<T, TA, 5, R8, W8>(c, pts, n, ws, s);
    case 6: return launch_reduce<T, TA, 6, R8, W8>(c, pts, n, ws, s);
    case 7: return launch_reduce<T, TA, 7, R8, W8>(c, pts, n, ws, s);
    default: return launch_reduce<T, TA, 8, R8, W8>(c, pts, n, ws, s);
  }
}

// The reduction above kMaxFastN images, FP64: the triangle in shared memory up to kReduceIn images.
int run_big_reduce(const float2* c, PointSet pts, int n, unsigned char* ws, void* slices, cudaStream_t s) {
  auto* sl = static_cast<double2*>(slices);
  if (n <= 144) return launch_reduce<double, double, 9, 4, 8>(c, pts, n, ws, s);
  if (n <= kReduceIn) return launch_reduce<double, double, 10, 4, 8>(c, pts, n, ws, s);
  if (n <= 160) return launch_reduce<double, double, 10, 4, 8, false>(c, pts, n, ws, s, sl);
  if (n <= 192) return launch_reduce<double, double, 12, 4, 8, false>(c, pts, n, ws, s, sl);
  if (n <= 256) return launch_reduce<double, double, 16, 4, 8, false>(c, pts, n, ws, s, sl);
  return launch_reduce<double, double, 32, 2, 8, false>(c, pts, n, ws, s, sl);
}

// One pass of the three kernels over a sub-batch (pts.list == nullptr: all pts.n_pc points;
// else the listed ones, whose count is read on the device), inverse and reduction both in
// T. cond_max > 0 flags the points whose condition estimate exceeds it.
template <typename T, int NR, int W>
int launch_tail(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
                const unsigned char* ws, const uint8_t* sing, cudaStream_t s) {
  const size_t tsmem = W * tail_warp_bytes<T>(n);
  auto kernel = tail_kernel<T, T, NR, W>;
  if (int rc_ = allow_smem(reinterpret_cast<const void*>(kernel), tsmem)) return rc_;
  const int tocc = std::max(1, occupancy(kernel, 32 * W, tsmem));
  const int64_t tgrid = std::min<int64_t>((pts.n_pc + W - 1) / W, (int64_t)sm_count() * tocc);
  KernelTimer kt(pts.list ? "emi tail rerun" : sizeof(T) == 8 ? "emi tail fp64" : "emi tail fp32", s);
  kernel<<<(unsigned)tgrid, 32 * W, tsmem, s>>>(c, pts, n, ref, ws, sing, ph, quality, tcoh);
  return check_launch("emi tail");
}

template <typename T>
int run_pass(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
             unsigned char* ws, uint8_t* sing, float cond_max, void* slices, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    if (n > kMaxFastN) {
      if (int rc = run_big_inverse(c, pts, n, ws, sing, slices, s)) return rc;
      if (int rc = run_big_reduce(c, pts, n, ws, slices, s)) return rc;
      return n <= 160   ? launch_tail<T, 5, 4>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s)
             : n <= 256 ? launch_tail<T, 8, 4>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s)
                        : launch_tail<T, 16, 4>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s);
    }
  }
  if (int rc = run_inverse<T, T>(c, pts, n, ws, sing, cond_max, s)) return rc;
  if (int rc = run_reduce<T, T>(c, pts, n, ws, s)) return rc;
  return launch_tail<T, 4, kTailWarps>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s);
}

template <int NB>
int launch_sweep(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, cudaStream_t s) {
  const int occ = std::max(1, occupancy(sweep_kernel<NB, float>, 256, 0));
  const int64_t grid = std::min<int64_t>(pts.n_pc, (int64_t)sm_count() * occ);
  KernelTimer kt(pts.list ? "emi sweep rerun" : "emi sweep fp64", s);
  sweep_kernel<NB, float><<<(unsigned)grid, 256, 0, s>>>(c, pts, n, ws, sing);
  return check_launch("emi sweep");
}

int run_sweep(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, cudaStream_t s) {
  switch ((n + 15) / 16) {
    case 1: case 2: return launch_sweep<2>(c, pts, n, ws, sing, s);
    case 3: return launch_sweep<3>(c, pts, n, ws, sing, s);
    case 4: return launch_sweep<4>(c, pts, n, ws, sing, s);
    case 5: return launch_sweep<5>(c, pts, n, ws, sing, s);
    case 6: return launch_sweep<6>(c, pts, n, ws, sing, s);
    case 7: return launch_sweep<7>(c, pts, n, ws, sing, s);
    default: return launch_sweep<8>(c, pts, n, ws, sing, s);
  }
}

// The refined pass: FP64 inverse (symmetric sweep), FP32 reduction, FP64-refined tail;
// sing[] ends with the points whose sweep met a small pivot or whose refined error bound
// exceeds `tol` flagged kRouteCond.
int run_refine_pass(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
                    unsigned char* ws, uint8_t* sing, double tol, cudaStream_t s) {
  if (int rc = run_sweep(c, pts, n, ws, sing, s)) return rc;
  if (int rc = run_reduce<float, double>(c, pts, n, ws, s)) return rc;
  const size_t tsmem = kRefineWarps * refine_warp_bytes(n);
  if (int rc_ = allow_smem(reinterpret_cast<const void*>(tail_refine_kernel<float>), tsmem)) return rc_;
  const int tocc = std::max(1, occupancy(tail_refine_kernel<float>, 32 * kRefineWarps, tsmem));
  const int64_t tgrid = std::min<int64_t>((pts.n_pc + kRefineWarps - 1) / kRefineWarps, (int64_t)sm_count() * tocc);
  KernelTimer kt("emi refine tail", s);
  tail_refine_kernel<float><<<(unsigned)tgrid, 32 * kRefineWarps, tsmem, s>>>(c, pts, n, ref, ws, sing, ph,
                                                                                quality, tcoh, tol);
  return check_launch("emi refine tail");
}

size_t point_bytes_max(int n) {
  return std::max({PointWs<float>(n).bytes, PointWs<double>(n).bytes, PointWs<float, double>(n).bytes});
}

}  // namespace

size_t fast_workspace_bytes(int64_t n_pc, int n) {
  if (n > kMaxFastN)
    return SubWs::bytes(std::min<int64_t>(n_pc, sub_batch<double>(n)), PointWs<double>(n).bytes, n_pc) +
           std::min<int64_t>(n_pc, sm_count()) * slice_bytes(n);
  const int64_t s32 = std::min<int64_t>(n_pc, sub_batch<float>(n));
  const int64_t s64 = std::min<int64_t>(n_pc, sub_batch<double>(n));
  return std::max(SubWs::bytes(s32, PointWs<float>(n).bytes, n_pc), SubWs::bytes(s64, point_bytes_max(n), n_pc));
}

int fast_run(const float2* coh, int64_t n_pc, int n, int ref, int precision, float cond_max, float2* ph,
             float* quality, float* tcoh, uint8_t* route, void* workspace, cudaStream_t s,
             const int64_t* dcount, int64_t doff) {
  const bool f64 = precision == MR_PREC_FP64;
  const bool mixed = precision == MR_PREC_MIXED;
  const bool refine = precision == MR_PREC_REFINE;
  if (dcount && mixed) return fail(MR_ERR_UNSUPPORTED, "emi: device-counted points run in FP32, FP64 or refined");
  auto* ws = static_cast<unsigned char*>(workspace);
  // a mixed or refined sub-batch must hold its points in FP64 when all of them are routed
  const bool wide = f64 || mixed || refine;
  // sub-batches of equal size (none left nearly empty at the end)
  const int64_t cap = wide ? sub_batch<double>(n) : sub_batch<float>(n);
  const int64_t nsub = (n_pc + cap - 1) / cap;
  const int64_t sub = nsub > 0 ? (n_pc + nsub - 1) / nsub : 0;
  const SubWs w(ws, sub, wide ? point_bytes_max(n) : PointWs<float>(n).bytes, n_pc);
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const bool routed = mixed || refine;
  if (routed) MR_CUDA_TRY(cudaMemsetAsync(w.count, 0, sizeof(int32_t), s));
  for (int64_t b0 = 0; b0 < n_pc; b0 += sub) {
    const int64_t nb = std::min<int64_t>(sub, n_pc - b0);
    const float2* c = coh + b0 * npairs;
    float2* p = ph + b0 * n;
    float* q = quality + b0;
    float* t = tcoh ? tcoh + b0 : nullptr;
    const PointSet all{nullptr, nullptr, nb, dcount, doff + b0};
    int rc;
    if (f64) {
      rc = run_pass<double>(c, all, n, ref, p, q, t, w.pts, w.sing, 0.f, w.slices, s);
      if (!rc && route) MR_CUDA_TRY(cudaMemsetAsync(route + b0, 1, (size_t)nb, s));
    } else {
      rc = refine ? run_refine_pass(c, all, n, ref, p, q, t, w.pts, w.sing, (double)cond_max, s)
                  : run_pass<float>(c, all, n, ref, p, q, t, w.pts, w.sing, mixed ? cond_max : 0.f, nullptr, s);
      if (!rc && routed) {
        const int grid = (int)std::min<int64_t>((nb + 255) / 256, (int64_t)sm_count() * 8);
        route_kernel<<<grid, 256, 0, s>>>(w.sing, nb, b0, w.list, w.count, route ? route + b0 : nullptr, refine,
                                          dcount, doff + b0);
        rc = check_launch("emi route");
      } else if (!rc && route) {
        MR_CUDA_TRY(cudaMemsetAsync(route + b0, 0, (size_t)nb, s));
      }
    }
    if (rc) return rc;
  }
  // the routed points of every sub-batch, in FP64, in windows of `sub` list entries (the
  // count is known only on the device: windows past it exit at once)
  if (routed) {
    for (int64_t l0 = 0; l0 < n_pc; l0 += sub) {
      const int rc = run_pass<double>(coh, PointSet{w.list, w.count, sub, nullptr, l0}, n, ref, ph, quality, tcoh,
                                      w.pts, w.sing2, 0.f, nullptr, s);
      if (rc) return rc;
    }
  }
  return MR_OK;
}

}  // namespace emi
}  // namespace mr
