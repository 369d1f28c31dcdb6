// EMI (moraine/pl.py:46-77: M = inv(|Gamma|) o Gamma, its smallest eigenpair, phases referred to
// image `ref`, fused temporal coherence), in sub-batches of points: in FP32, FP64 or refined up
// to 128 images, in FP64 above.
//
// Kernels, each at its own occupancy (the register-bound inverse is not held back by the
// shared memory of the reduction, and serial recurrences of many points share a warp):
//   inverse_kernel         inv(|Gamma|) by Gauss-Jordan with partial pivoting in registers
//                          (gj_tile): the padded 16NB x 16NB matrix on a 16 x 16 thread grid,
//                          rows never swapped, one barrier per step; the result stored
//                          upper-packed in the workspace. FP32 and FP64 EMI, and the FP64
//                          recomputation of routed points.
//   sweep_kernel           inv(|Gamma|) in FP64 for the refined EMI: the symmetric sweep, two
//                          pivots per barrier, only the lower triangle held.
//   big_inverse_kernel     the pivoted inverse above 128 images, in shared memory or L2.
//   reduce_kernel          M in shared memory as a packed lower triangle, Householder
//                          reduction to a Hermitian tridiagonal -> workspace (d, e, tau,
//                          reflectors).
//   tri_eig_kernel         smallest eigenpair of the real tridiagonal: Sturm counts and inverse
//                          iteration (two solves), several points per warp.
//   tail_kernel            one warp per point: back-transformation, normalisation, temporal
//                          coherence.
//   refine_*_kernel        the refined EMI's tail: one FP64 Newton correction of the FP32
//                          eigenvector and an FP64 error bound that routes the points
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
// T), d and tau (n T each), e (n complex T). The reduction has all of M in its triangle before it
// writes the first reflector, so above 128 images (kBig), where the workspace is kept small, the
// reflectors take the inverse's place: n (n + 1) / 2 reals in n (n - 1) / 2 pairs of them. (Up to 128
// images that would save a third of 4 GiB, and the refined tail reads the inverse again.)
__host__ __device__ __forceinline__ int64_t tri_up(int m, int j, int n) {
  return (int64_t)m * n - ((int64_t)m * (m - 1)) / 2 + (j - m);
}

template <typename T, typename TA = T, bool kBig = false>
struct PointWs {
  size_t np, nq, bytes;
  __host__ __device__ explicit PointWs(int n) {
    using C = typename C2<T>::type;
    np = (size_t)n * (n + 1) / 2;
    nq = (size_t)n * (n - 1) / 2;
    bytes = (kBig ? 0 : align16(np * sizeof(TA))) + align16(nq * sizeof(C)) + align16(2 * (size_t)n * sizeof(T)) +
            align16((size_t)n * sizeof(C)) + align16(((size_t)n + 2) * sizeof(T)) +
            (kRefined ? (2 * (size_t)n + 1) * sizeof(double2) : 0);
  }
  static constexpr bool kRefined = sizeof(T) == 4 && sizeof(TA) == 8;
};

template <typename T, typename TA = T, bool kBig = false>
struct PointPtr {
  using C = typename C2<T>::type;
  TA* ainv;
  C* refl;
  T* d;
  T* tau;
  C* e;
  T* y;        // eigenvector of the real tridiagonal
  T* scal;     // its eigenvalue; the tridiagonal's largest row sum
  double2* v;  // refined EMI: eigenvector of M,
  double2* x;  // right-hand side and solution of the projected solve,
  double* lam; // Rayleigh quotient
  __device__ PointPtr(unsigned char* ws, int64_t pt, int n) {
    const PointWs<T, TA, kBig> w(n);
    unsigned char* b = ws + (size_t)pt * w.bytes;
    ainv = reinterpret_cast<TA*>(b);
    if (!kBig) b += align16(w.np * sizeof(TA));
    refl = reinterpret_cast<C*>(b);
    b += align16(w.nq * sizeof(C));
    d = reinterpret_cast<T*>(b);
    tau = d + n;
    b += align16(2 * (size_t)n * sizeof(T));
    e = reinterpret_cast<C*>(b);
    b += align16((size_t)n * sizeof(C));
    y = reinterpret_cast<T*>(b);
    scal = y + n;
    b += align16(((size_t)n + 2) * sizeof(T));
    v = reinterpret_cast<double2*>(b);
    x = v + n;
    lam = reinterpret_cast<double*>(x + n);
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

// CTAs per SM that the registers are cut to: left alone the unrolled steps take up to 254 registers
// and one CTA waits out its pivot chain alone. 4,000 points, one CTA (natural) against this: FP64,
// N = 64 1.5 and 0.70 ms, N = 100 3.46 and 2.89, where the spills of a third CTA cost more than it
// gives, as those of a second do above 112; FP32, N = 64 two, three and four CTAs 0.71, 0.57, 0.51.
template <typename T, int NB> constexpr int gj_ctas() {
  return sizeof(T) == 4 ? (NB <= 7 ? 4 : 3) : NB <= 3 ? 5 : NB == 4 ? 4 : NB == 5 ? 3 : NB <= 7 ? 2 : 1;
}

// TW: arithmetic of the reduction that reads the workspace (the point stride depends on it).
template <typename T, int NB, int CX, typename TW>
__global__ void __launch_bounds__(16 * CX, gj_ctas<T, NB>()) inverse_kernel(const float2* __restrict__ coh, PointSet pts, int n,
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

// ----------------------------------------------------------------- kernel 1a: inverse, N <= 32
// The same Gauss-Jordan with one warp per point: lane i holds row i in registers (the padding is
// identity and never pivots), the pivot is a warp argmax over the lanes' entries of column k, and the
// pivot row goes to all lanes by shuffles. No barrier, and as many points per SM as it has warps:
// on the 16 x 16 grid a 17 x 17 matrix used 289 of the CTA's 1,024 entries and waited for a
// barrier per step. FP64, N = 17, 1,003 points: 23 us against 42.
constexpr int kWarpInvWarps = 4;

template <typename T, int NM, typename TW>
__global__ void __launch_bounds__(32 * kWarpInvWarps) warp_inverse_kernel(const float2* __restrict__ coh, PointSet pts,
                                                                          int n, unsigned char* __restrict__ ws,
                                                                          uint8_t* __restrict__ sing, float cond_max) {
  const int lane = threadIdx.x & 31;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * kWarpInvWarps + (threadIdx.x >> 5); pt < npt;
       pt += (int64_t)gridDim.x * kWarpInvWarps) {
    const float2* c = coh + pts[pt] * npairs;
    T a[NM];
#pragma unroll
    for (int j = 0; j < NM; ++j) {
      float2 g = make_float2(lane == j ? 1.f : 0.f, 0.f);
      if (lane < n && j < n && lane != j) g = c[lane < j ? triu_index(lane, j, n) : triu_index(j, lane, n)];
      a[j] = (T)sqrt((double)g.x * g.x + (double)g.y * g.y);
    }
    auto norm = [&]() {  // max over the rows of the sum of |a_ij|
      T r = 0;
#pragma unroll
      for (int j = 0; j < NM; ++j)
        if (j < n) r += fabs(a[j]);
      if (lane >= n) r = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
      return r;
    };
    const T anorm = cond_max > 0.f ? norm() : T(0);
    bool used = lane >= n, singular = false;
    int step = 0;       // of this row
    int piv_mine = 0;   // lane k: pivot row of step k
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      if (k >= n) break;
      T best = used ? T(-1) : fabs(a[k]) == fabs(a[k]) ? fabs(a[k]) : T(-0.5);  // NaN ranks last but is taken
      int p = used ? 32 : lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const T ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, p, o);
        if (ob > best || (ob == best && oi < p)) { best = ob; p = oi; }
      }
      T pv = __shfl_sync(0xffffffffu, a[k], p);
      if (pv == T(0)) { singular = true; pv = T(1); }
      const T rp = recip(pv);
      const bool is_p = lane == p;
      if (is_p) { used = true; step = k; }
      if (lane == k) piv_mine = p;
      // a -= f r everywhere, with f_p = pv - 1 so that the pivot row becomes r
      const T fi = a[k], f = is_p ? pv - T(1) : fi;
#pragma unroll
      for (int j = 0; j < NM; ++j) a[j] -= f * (__shfl_sync(0xffffffffu, a[j], p) * rp);
      a[k] = is_p ? rp : -fi * rp;
    }
    uint8_t flag = singular ? kRouteSingular : 0;
    if (cond_max > 0.f && !singular) {
      const T cond = anorm * norm();
      if (!(cond <= (T)cond_max)) flag = kRouteCond;
    }
    T* out = PointPtr<TW, T>(ws, pt, n).ainv;
#pragma unroll
    for (int j = 0; j < NM; ++j) {  // row `step` of the inverse; column j belongs to pivot row j's step
      if (j >= n) break;
      const int pc = __shfl_sync(0xffffffffu, piv_mine, j);
      if (lane < n && step >= pc) out[tri_up(pc, step, n)] = a[j];  // inv[step][pc], kept once
    }
    if (lane == 0) sing[pt] = flag;
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
    double* out = PointPtr<double, double, true>(ws, pt, n).ainv;
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
// partial sums are added in a fixed order, so results do not depend on timing. In blocks of 16 columns
// that meet the diagonal a lane reads and writes only entries of its own row (what lies past the
// diagonal belongs to the next row, and to another half-warp) and counts half of the diagonal in
// either part. Bound by latency: the chain of A (two warp sums, roots and
// divisions) and the short strips of B, hidden only by the other CTAs of the SM. The previous form
// (256 threads, three barriers, groups of four threads on mirrored row pairs, row and column parts in
// separate passes over M): FP32, N = 17, 2,047 points 146 us, now 37; N = 50, 35,627 points 8.4 ms,
// now 3.6; N = 100, 286,294 points 199 ms, now 165; FP64, N = 17, 1,003 points 157 us, now 37; N = 100,
// 4,001 points 6.2 ms, now 5.1. FP32 in packed pairs (fma.f32x2 on rows and columns laid out twice)
// was slower, 204 ms: its sums and doubled vectors cost registers and shared memory.
// The vectors of a step, one record per row: kRowPad zero records in front (rows above the first of a
// strip) and kColPad behind (columns past the last). u, w: of step k-1; c: u_k.
constexpr int kRowPad = 8, kColPad = 16;
template <typename C> struct Rec {
  C u, w, c;
};

// Shared memory: the step's records, each warp's column sums, the row sums, and the triangle.
__host__ __device__ inline size_t reduce_tri(int n) { return (size_t)n * (n + 1) / 2; }
template <typename T>
__host__ __device__ inline size_t reduce_smem(int n, int warps, bool tri_in) {
  return (n + kRowPad + kColPad) * sizeof(Rec<typename C2<T>::type>) +
         ((tri_in ? reduce_tri(n) : 0) + (size_t)(warps + 1) * n) * sizeof(typename C2<T>::type);
}

template <typename T, typename TA, int QC, int R, int W, bool kTriIn = true>
__global__ void __launch_bounds__(32 * W, W >= 3 && QC <= 8 ? (sizeof(T) == 8 ? 2 : 16 / W) : 1)
    reduce_kernel(const float2* __restrict__ coh, PointSet pts, int n, unsigned char* __restrict__ ws,
                  typename C2<T>::type* __restrict__ slices) {
  using C = typename C2<T>::type;
  constexpr int Q = (QC + 1) / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, lc = lane & 15, wid = tid >> 5;
  constexpr int nw = W;
  Rec<C>* rec = reinterpret_cast<Rec<C>*>(smem_raw) + kRowPad;
  C* part = reinterpret_cast<C*>(rec + n + kColPad);  // [warps][n]: each warp's column sums
  C* rows = part + nw * n;                             // row sums
  C* L = kTriIn ? rows + n : slices + blockIdx.x * reduce_tri(n);
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int e = tid; e < kRowPad + kColPad; e += blockDim.x) {
    rec[e < kRowPad ? -1 - e : n + e - kRowPad] = {mk<T>(0, 0), mk<T>(0, 0), mk<T>(0, 0)};
  }
  for (int64_t pt = blockIdx.x; pt < npt; pt += gridDim.x) {
    const float2* c = coh + pts[pt] * npairs;
    PointPtr<T, TA, (QC > 8)> w(ws, pt, n);
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
            C p = rows[i];
#pragma unroll
            for (int q = 0; q < nw; ++q) p = cadd(p, part[q * n + i]);
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
          if (i < n) { rec[i].u = u[t]; rec[i].w = wr[t]; }
        }
        __syncwarp();
        const C uk = rec[k].u, wk = rec[k].w;
        C x[Q];
        T xn2 = 0;
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const int i = lane + 32 * t;
          x[t] = mk<T>(0, 0);
          if (i >= k && i < n) {
            x[t] = L[tri(i) + k];
            rank2(x[t], u[t], wk, wr[t], uk);
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
          if (i < n) rec[i].c = u[t];
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
      const Rec<C>* crec = rec + (k + 1 + lc);
      for (int top = n - 1 - 2 * R * wid; top > k; top -= 2 * R * nw) {
        const int hi = top - R * (lane >> 4);  // this half-warp's strip: rows hi - R + 1 .. hi
        Rec<C> rv[R];
        C sum[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          rv[r] = rec[hi - r];
          sum[r] = mk<T>(0, 0);
        }
        C* row0 = L + tri(hi) + (k + 1 + lc);
        // row hi - r starts r hi - r (r - 1) / 2 entries earlier
#pragma unroll
        for (int q = 0; q < QC; ++q) {
          const int j0 = k + 1 + 16 * q;
          if (j0 > top) break;
          const Rec<C> cv = crec[16 * q];
          if (j0 + 15 < top - (2 * R - 1)) {  // all lanes left of every diagonal of the two strips
#pragma unroll
            for (int r = 0; r < R; ++r) {
              C* e = row0 - (r * hi - r * (r - 1) / 2) + 16 * q;
              C a = *e;
              rank2(a, rv[r].u, cv.w, rv[r].w, cv.u);
              *e = a;
              cmac(sum[r], a, cv.c);
              cmacc(acc[q], a, rv[r].c);
            }
          } else {
            const int left = hi - (j0 + lc);  // of row hi's diagonal
#pragma unroll
            for (int r = 0; r < R; ++r) {
              C* e = row0 - (r * hi - r * (r - 1) / 2) + 16 * q;
              const bool own = left >= r;  // else the next row's entry, which its own half-warp may be writing
              C a = own ? *e : mk<T>(0, 0);
              rank2(a, rv[r].u, cv.w, rv[r].w, cv.u);
              if (own) *e = a;
              // half of the diagonal in either part, nothing beyond it
              a.x = left > r ? a.x : left == r ? T(0.5) * a.x : T(0);
              a.y = left > r ? a.y : T(0);
              cmac(sum[r], a, cv.c);
              cmacc(acc[q], a, rv[r].c);
            }
          }
        }
        const C tot = half_warp_sum(sum);
        const int i = hi - (lane & 15) / (16 / R);
        if (lane % (16 / R) == 0 && i > k) rows[i] = tot;
      }
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        const int j0 = k + 1 + 16 * q;
        if (j0 >= n) break;
        const C col = cadd(acc[q], shfl_xor_c(acc[q], 16));
        if (lane < 16 && j0 + lane < n) mine[j0 + lane] = col;
      }
      __syncthreads();
    }
    __syncthreads();  // L and the vectors are rewritten for the next point
  }
}

// Reflector k of a point (its scalar and the lane's entries, of rows lane + 32 t) into registers.
template <typename T, typename TA, bool kBig, int NR>
__device__ __forceinline__ void load_refl(const PointPtr<T, TA, kBig>& w, int n, int k, int lane,
                                          typename C2<T>::type (&u)[NR], T& tau) {
  tau = w.tau[k];
  const typename C2<T>::type* src = w.refl + refl_off(k, n) - (k + 1);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    const int i = lane + 32 * t;
    u[t] = i > k && i < n ? src[i] : mk<T>(0, 0);
  }
}

// z <- H_k z for the reflectors of the workspace, k ascending (forward, Q^H z) or descending (back,
// Q z), z in registers (row lane + 32 t). A ring of D reflectors is on its way while one is applied,
// so that the serial chain does not wait on memory. One warp.
template <typename T, typename TA, bool kBig, int NR>
__device__ __forceinline__ void apply_q(const PointPtr<T, TA, kBig>& w, int n, typename C2<T>::type (&z)[NR], bool forward) {
  using C = typename C2<T>::type;
  constexpr int D = NR * sizeof(C) <= 16 ? 4 : NR * sizeof(C) <= 64 ? 2 : 1;
  const int lane = threadIdx.x & 31, steps = n - 2;
  C u[D][NR];
  T tau[D];
#pragma unroll
  for (int r = 0; r < D; ++r) {
    tau[r] = T(0);
    if (r < steps) load_refl(w, n, forward ? r : n - 3 - r, lane, u[r], tau[r]);
  }
  for (int s0 = 0; s0 < steps; s0 += D) {
#pragma unroll
    for (int r = 0; r < D; ++r) {
      const int s = s0 + r;
      if (s >= steps) break;
      C acc = mk<T>(0, 0);
#pragma unroll
      for (int t = 0; t < NR; ++t) cmacc(acc, u[r][t], z[t]);  // u^H z
      acc.x = tau[r] * warp_sum(acc.x);
      acc.y = tau[r] * warp_sum(acc.y);
#pragma unroll
      for (int t = 0; t < NR; ++t) {
        z[t].x -= u[r][t].x * acc.x;
        z[t].x += u[r][t].y * acc.y;
        z[t].y -= u[r][t].x * acc.y;
        z[t].y -= u[r][t].y * acc.x;
      }
      if (s + D < steps) load_refl(w, n, forward ? s + D : n - 3 - s - D, lane, u[r], tau[r]);
    }
  }
}

// Phases of the real tridiagonal R = D^H T D: delta_0 = 1, delta_{k+1} = delta_k e_k / |e_k|, as a warp
// prefix product; lane l gets delta of rows l + 32 t. One warp.
template <typename V, typename T, typename TA, bool kBig, int NR>
__device__ __forceinline__ void row_phases(const PointPtr<T, TA, kBig>& w, int n, typename C2<V>::type (&dl)[NR]) {
  using C = typename C2<V>::type;
  const int lane = threadIdx.x & 31;
  C carry = mk<V>(1, 0);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    const int i = lane + 32 * t;
    C f = mk<V>(1, 0);
    if (i > 0 && i < n) {
      const V x = w.e[i - 1].x, y = w.e[i - 1].y, a = sqrt(x * x + y * y);
      if (a > V(0)) f = mk<V>(x / a, y / a);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V ox = __shfl_up_sync(0xffffffffu, f.x, o), oy = __shfl_up_sync(0xffffffffu, f.y, o);
      if (lane >= o) f = cmul_t(mk<V>(ox, oy), f);
    }
    dl[t] = cmul_t(carry, f);
    carry = mk<V>(__shfl_sync(0xffffffffu, dl[t].x, 31), __shfl_sync(0xffffffffu, dl[t].y, 31));
  }
}

// ----------------------------------------------------------------- kernel 3: tridiagonal eigenpair
// Elements of many points' vectors in shared memory: entry i of point p at [i * stride + p].
template <typename V> struct Strided {
  V* p;
  int stride;
  __device__ __forceinline__ V& operator[](int i) const { return p[i * stride]; }
};

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

// Solve (R - lambda I) x = scale y in place, R real symmetric tridiagonal with diagonal d(i) and
// off-diagonal b(i), by elimination with row interchanges, for a real (V = T) or complex (V = C2<T>)
// right-hand side. Each row's final pivot is inverted once and kept in dd, so the back substitution
// multiplies: one reciprocal per row on the serial chain; the row under elimination stays in
// registers. dd, du, dl: work arrays of length n (dl: the second super-diagonal). One thread.
template <typename T, typename V, class D, class B>
__device__ __forceinline__ void tridiag_solve(D d, B b, int n, T lambda, T tiny, T scale, Strided<V> y, Strided<T> dd,
                                              Strided<T> du, Strided<T> dl) {
  T di = d(0) - lambda, dui = b(0);
  V yi = y[0];
  scale_r<T>(yi, scale);
  for (int i = 0; i < n - 1; ++i) {
    const T sub = b(i), dn = d(i + 1) - lambda, dun = i < n - 2 ? b(i + 1) : T(0);
    V yn = y[i + 1];
    scale_r<T>(yn, scale);
    if (fabs(di) >= fabs(sub)) {
      if (di == T(0)) di = tiny;
      const T r = recip(di), f = sub * r;
      dd[i] = r;
      du[i] = dui;
      dl[i] = T(0);
      y[i] = yi;
      di = dn - f * dui;
      dui = dun;
      axpy_r<T>(yn, f, yi);
      yi = yn;
    } else {
      const T r = recip(sub), f = di * r;
      dd[i] = r;
      du[i] = dn;
      dl[i] = dun;
      y[i] = yn;
      di = dui - f * dn;
      dui = -f * dun;
      axpy_r<T>(yi, f, yn);
    }
  }
  if (di == T(0)) di = tiny;
  V y1 = yi, y2 = yi;
  scale_r<T>(y1, recip(di));
  y[n - 1] = y1;
  for (int i = n - 2; i >= 0; --i) {
    V v = y[i];
    axpy_r<T>(v, du[i], y1);
    if (i < n - 2) axpy_r<T>(v, dl[i], y2);
    scale_r<T>(v, dd[i]);
    y[i] = v;
    y2 = y1;
    y1 = v;
  }
}

// Smallest eigenvalue of the real tridiagonal (by sections of a bracket, G Sturm counts at a time) and
// its eigenvector y (two inverse iterations, one lane), G lanes per point and kEigThreads / G points
// per CTA, everything in shared memory. A warp per point left its other lanes idle in the solves,
// and 33 sections a round cost 5 times the operations of 5: the serial recurrences of a point
// take as long either way, but here a warp runs those of 32 / G points at once (286,294 points,
// N = 100: 2.9 ms). Results (lambda, max row sum, y) go to the workspace.
constexpr int kEigThreads = 128;

template <typename T> inline size_t eig_smem(int n, int g) { return 6 * (size_t)n * (kEigThreads / g + 1) * sizeof(T); }

template <typename T, typename TA, int G, bool kBig>
__global__ void __launch_bounds__(kEigThreads) tri_eig_kernel(PointSet pts, int n, unsigned char* __restrict__ ws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int P = kEigThreads / G, S = P + 1;
  const int tid = threadIdx.x, lane = tid & 31, p = tid / G, g = tid % G;
  T* d0 = reinterpret_cast<T*>(smem_raw);
  T* b0 = d0 + n * S;
  const int64_t npt = pts.size();
  for (int64_t base = (int64_t)blockIdx.x * P; base < npt; base += (int64_t)gridDim.x * P) {
    const int here = (int)(npt - base < P ? npt - base : P);
#pragma unroll 4
    for (int f = tid; f < here * n; f += kEigThreads) {
      const int q = f / n, i = f - q * n;
      const PointPtr<T, TA, kBig> w(ws, base + q, n);
      d0[i * S + q] = w.d[i];
      const typename C2<T>::type e = w.e[min(i, n - 2)];
      b0[i * S + q] = sqrt(e.x * e.x + e.y * e.y);  // entry n - 1 is not used
    }
    __syncthreads();
    const bool live = base + p < npt;
    const Strided<T> d{d0 + p, S}, b{b0 + p, S}, y{b0 + n * S + p, S}, dd{b0 + 2 * n * S + p, S},
        du{b0 + 3 * n * S + p, S}, dl{b0 + 4 * n * S + p, S};
    T lo = Lim<T>::huge(), hi = -Lim<T>::huge(), tnorm = 0;
    if (live)
      for (int i = g; i < n; i += G) {
        const T r = (i > 0 ? b[i - 1] : T(0)) + (i + 1 < n ? b[i] : T(0));
        lo = fmin(lo, d[i] - r);
        hi = fmax(hi, d[i] + r);
        tnorm = fmax(tnorm, fabs(d[i]) + r);
        if (i + 1 < n) dd[i] = b[i] * b[i];
        y[i] = T(1) + T(0.25) * (T)((i * 37) % 11) / T(11);
      }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
    }
    __syncwarp();
    const T eps = Lim<T>::eps();
    const T pivmin = fmax(Lim<T>::tiny(), eps * eps * tnorm * tnorm) + Lim<T>::tiny();
    const T pad = T(2) * eps * fmax(tnorm, Lim<T>::tiny()) + T(2) * pivmin;
    lo -= pad;
    hi += pad;
    for (int it = 0; it < 64; ++it) {
      const T width = hi - lo;
      const bool open = live && width > T(2) * eps * fmax(fabs(lo), fabs(hi)) + T(4) * pivmin;
      if (!__any_sync(0xffffffffu, open)) break;
      int cnt = 0;
      if (open) cnt = sturm_count(d, dd, n, lo + width * (T)(g + 1) / T(G + 1), pivmin);
      const unsigned ball = __ballot_sync(0xffffffffu, cnt >= 1) >> (lane & ~(G - 1));
      const unsigned mine = G == 32 ? ball : ball & ((1u << (G & 31)) - 1u);
      if (open) {
        const int first = mine ? __ffs(mine) - 1 : G;
        const T nlo = first == 0 ? lo : lo + width * (T)first / T(G + 1);
        hi = first == G ? hi : lo + width * (T)(first + 1) / T(G + 1);
        lo = nlo;
      }
    }
    const T lam = T(0.5) * (lo + hi);
    __syncwarp();
    if (g == 0 && live) {
      const T tiny = eps * fmax(tnorm, Lim<T>::tiny());
      T scale = 1;
      for (int it = 0; it < 2; ++it) {
        tridiag_solve<T>([&](int i) { return d[i]; }, [&](int i) { return b[i]; }, n, lam, tiny, scale, y, dd, du, dl);
        T sc = 0;
        for (int i = 0; i < n; ++i) sc = fmax(sc, fabs(y[i]));
        scale = T(1) / sc;
        if (!(sc > T(0)) || !isfinite(sc)) { scale = T(1); break; }
      }
      du[0] = scale;  // for the group's other lanes
    }
    __syncwarp();
    if (live) {
      const PointPtr<T, TA, kBig> w(ws, base + p, n);
      const T scale = du[0];
      for (int i = g; i < n; i += G) w.y[i] = y[i] * scale;
      if (g == 0) {
        w.scal[0] = lam;
        w.scal[1] = tnorm;
      }
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------- kernel 4: phases from the eigenvector
constexpr int kTailWarps = 8;

// 1 / sqrt(x) in FP64 from the FP32 root: two Newton steps, to about an FP64 ulp. x within FP32's
// normal range, else the quotient.
__device__ __forceinline__ double inv_sqrt(double x) {
  if (!(x > 1.2e-38 && x < 3.0e38)) return 1.0 / sqrt(x);
  double y = (double)rsqrtf((float)x);
  const double h = 0.5 * x;
  y = y * fma(-h * y, y, 1.5);
  return y * fma(-h * y, y, 1.5);
}

// |sum_q coh_q / |coh_q| conj(ph_m) ph_j| / n_pairs of one point, phs its phases. One warp; lane 0's value.
__device__ __forceinline__ float temp_coh_of(const float2* __restrict__ c, const double2* phs, int n) {
  const int lane = threadIdx.x & 31;
  const int npairs = n * (n - 1) / 2;
  double tx = 0, ty = 0;
  int mm = 0, jj = 1 + lane;
  while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
  auto add = [&](float2 g) {
    const int m0 = mm, j0 = jj;
    jj += 32;
    while (jj >= n && mm < n - 1) { mm += 1; jj = jj - n + mm + 1; }
    const double gx = g.x, gy = g.y;
    const double r = inv_sqrt(gx * gx + gy * gy);
    const double2 v = cmul(make_double2(gx, gy), cmulc(phs[j0], phs[m0]));
    tx = fma(v.x, r, tx);
    ty = fma(v.y, r, ty);
  };
  int q = lane;
  for (; q + 96 < npairs; q += 128) {  // four coherences on their way at a time
    const float2 g0 = c[q], g1 = c[q + 32], g2 = c[q + 64], g3 = c[q + 96];
    add(g0);
    add(g1);
    add(g2);
    add(g3);
  }
  for (; q < npairs; q += 32) add(c[q]);
  tx = warp_sum(tx);
  ty = warp_sum(ty);
  return (float)(sqrt(tx * tx + ty * ty) / (double)npairs);
}

// Value of row `ref` of a vector held by rows lane + 32 t.
template <typename C, int NR> __device__ __forceinline__ C row_value(const C (&v)[NR], int ref) {
  C r = v[0];
#pragma unroll
  for (int t = 1; t < NR; ++t)
    if (ref >> 5 == t) r = v[t];
  r.x = __shfl_sync(0xffffffffu, r.x, ref & 31);
  r.y = __shfl_sync(0xffffffffu, r.y, ref & 31);
  return r;
}

// ph = v conj(v[ref]) / |.| of one point (NaN where singular) to global memory and to phs.
template <typename C, int NR>
__device__ __forceinline__ void write_phases(const C (&v)[NR], int n, int ref, bool singular, float2* __restrict__ ph,
                                             double2* phs) {
  const int lane = threadIdx.x & 31;
  const float fnan = __int_as_float(0x7fffffff);
  const C zr = row_value(v, ref);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    const int i = lane + 32 * t;
    const C q = cmulc_t(v[t], zr);
    const double vx = q.x, vy = q.y, a = sqrt(vx * vx + vy * vy);
    float2 o = make_float2((float)(vx / a), (float)(vy / a));
    if (singular) o = make_float2(fnan, fnan);
    if (i < n) {
      ph[i] = o;
      phs[i] = make_double2(o.x, o.y);
    }
  }
  __syncwarp();
}

// One warp per point: v = Q D y, normalisation, temporal coherence. NR: rows per lane (32 NR >= n).
template <typename T, typename TA, int NR>
__global__ void __launch_bounds__(32 * kTailWarps) tail_kernel(const float2* __restrict__ coh, PointSet pts, int n,
                                                               int ref, unsigned char* __restrict__ ws,
                                                               const uint8_t* __restrict__ sing,
                                                               float2* __restrict__ ph, float* __restrict__ quality,
                                                               float* __restrict__ tcoh) {
  using C = typename C2<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double2* phs = reinterpret_cast<double2*>(smem_raw) + wid * n;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * kTailWarps + wid; pt < npt; pt += (int64_t)gridDim.x * kTailWarps) {
    const int64_t gp = pts[pt];
    const PointPtr<T, TA, (NR > 4)> w(ws, pt, n);
    C z[NR];
    row_phases<T>(w, n, z);
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const int i = lane + 32 * t;
      const T yi = i < n ? w.y[i] : T(0);
      z[t] = mk<T>(z[t].x * yi, z[t].y * yi);
    }
    apply_q(w, n, z, false);
    const bool singular = (sing[pt] & kRouteSingular) != 0;
    write_phases(z, n, ref, singular, ph + gp * n, phs);
    if (lane == 0) quality[gp] = singular ? __int_as_float(0x7fffffff) : (float)w.scal[0];
    if (tcoh) {
      const float t = temp_coh_of(coh + gp * npairs, phs, n);
      if (lane == 0) tcoh[gp] = t;
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------- kernels 4a-c: refined tail
// For the refined mixed precision (FP64 inverse, FP32 reduction): the FP32 eigenvector is
// improved by one step of a Newton (Jacobi-Davidson) correction in FP64,
//   r = M v - lambda v (lambda = v^H M v, M = inv(|Gamma|) o Gamma from the FP64 inverse),
//   (M - lambda I) dv = r solved approximately through the FP32 factors M ~ Q D R D^H Q^H,
//   dv = Q D P (R - lambda I)^-1 P D^H Q^H r, P the projector orthogonal to R's eigenvector,
// which divides the error by about eps32 ||M|| / gap. Then the refined pair is checked in
// FP64: with residual r', gap g = lambda_2(R) - lambda and smallest component |v_i|, the
// phase error of every date is at most |r'| / (g min|v_i|); points above `tol` are flagged
// for an FP64 recomputation. Two kernels of one warp per point (residual; correction and check),
// the projected solve between them with one thread per point. The reflectors are applied in FP32
// (the factors hold M only to FP32 accuracy anyway), the projected solve runs in FP64. Bound by the
// latency of the reads of M and the reflectors at 16 to 20 warps per SM; a group of four matvec rows
// fetches its values together, without a branch in between (fetched value by value, or two rows at a
// time behind their bounds tests: 33 and 35 against 22 ms for the residual). 286,294 points, N = 100:
// 54 ms in all, against 89 for one kernel of a warp per point with the eigenpair and the solves on one
// lane; 35,627 points, N = 50: 2.0 against 4.8 ms.
constexpr int kRefineWarps = 4;

// out = M v for M = inv(|Gamma|) o Gamma (Hermitian), read along the upper triangle: the
// element (m, j > m) adds M_mj v_j to row m and conj(M_mj) v_m to row j. Lanes own columns
// j = lane + 32 t (vj: v's values there); rows go four at a time through warp_sum4, row values of v
// and the sums through shared memory. One warp.
template <int NR>
__device__ __forceinline__ void herm_matvec(const double* __restrict__ ainv, const float2* __restrict__ c, int n,
                                            const double2 (&vj)[NR], double2* v, double2* sums, double2 (&out)[NR]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    if (lane + 32 * t < n) v[lane + 32 * t] = vj[t];
    out[t] = make_double2(0, 0);
  }
  __syncwarp();
  for (int m0 = 0; m0 < n; m0 += 4) {
    double2 racc[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) racc[r] = make_double2(0, 0);
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      if (32 * t + 31 < m0) continue;  // warp-uniform
      const int j = lane + 32 * t;
      double sc[4];
      float2 g[4];
      // the four rows' values are fetched together, without a branch: what is outside the triangle
      // reads an element of its row and counts nothing
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = min(m0 + r, n - 1), um = (int)tri_up(m, m, n) - m;
        sc[r] = ainv[um + max(min(j, n - 1), m)];
        g[r] = c[max(um - (m + 1) + max(min(j, n - 1), min(m + 1, n - 1)), 0)];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = m0 + r;
        const double s = j >= m && j < n && m < n ? sc[r] : 0.0;
        if (j == m) g[r] = make_float2(1.f, 0.f);
        const double2 a = make_double2(s * (double)g[r].x, s * (double)g[r].y);  // M_mj
        cmac(racc[r], a, vj[t]);
        const double2 vm = v[min(m, n - 1)];
        if (j > m) cmacc(out[t], a, vm);
      }
    }
    const double2 tot = warp_sum4(racc);
    const int r = lane >> 3;
    if ((lane & 7) == 0 && m0 + r < n) sums[m0 + r] = tot;
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < NR; ++t)
    if (lane + 32 * t < n) out[t] = cadd(out[t], sums[lane + 32 * t]);
  __syncwarp();
}

// v^H M v / v^H v into lam; mv becomes the residual M v - lam v; its norm relative to |v| returned.
template <int NR>
__device__ __forceinline__ double residual(const double2 (&v)[NR], double2 (&mv)[NR], double& lam) {
  double vmv = 0, vv = 0, r2 = 0;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    vmv += v[t].x * mv[t].x + v[t].y * mv[t].y;
    vv += v[t].x * v[t].x + v[t].y * v[t].y;
  }
  vv = warp_sum(vv);
  lam = warp_sum(vmv) / vv;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    mv[t] = make_double2(mv[t].x - lam * v[t].x, mv[t].y - lam * v[t].y);
    r2 += mv[t].x * mv[t].x + mv[t].y * mv[t].y;
  }
  return sqrt(warp_sum(r2) / vv);
}

// y of unit length in FP64, rows lane + 32 t.
template <int NR>
__device__ __forceinline__ void unit_y(const float* y, int n, double (&yd)[NR]) {
  const int lane = threadIdx.x & 31;
  double yn = 0;
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    yd[t] = lane + 32 * t < n ? (double)y[lane + 32 * t] : 0.0;
    yn += yd[t] * yd[t];
  }
  yn = 1.0 / sqrt(warp_sum(yn));
#pragma unroll
  for (int t = 0; t < NR; ++t) yd[t] *= yn;
}

// x - yd (yd . x): the projector P.
template <int NR> __device__ __forceinline__ void project(const double (&yd)[NR], double2 (&x)[NR]) {
  double2 pr = make_double2(0, 0);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    pr.x += yd[t] * x[t].x;
    pr.y += yd[t] * x[t].y;
  }
  pr.x = warp_sum(pr.x);
  pr.y = warp_sum(pr.y);
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    x[t].x -= yd[t] * pr.x;
    x[t].y -= yd[t] * pr.y;
  }
}

template <int NR>
__global__ void __launch_bounds__(32 * kRefineWarps, NR <= 2 ? 5 : 4) refine_residual_kernel(
    const float2* __restrict__ coh, PointSet pts, int n, unsigned char* __restrict__ ws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double2* sv = reinterpret_cast<double2*>(smem_raw) + 3 * n * wid;
  double2* sd = sv + 2 * n;  // the rows' phases, out of the registers' way
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * kRefineWarps + wid; pt < npt; pt += (int64_t)gridDim.x * kRefineWarps) {
    const PointPtr<float, double> w(ws, pt, n);
    float2 z[NR];  // v = Q D y
    {
      double2 dph[NR];
      double yd[NR];
      row_phases<double>(w, n, dph);
      unit_y(w.y, n, yd);
#pragma unroll
      for (int t = 0; t < NR; ++t) {
        if (lane + 32 * t < n) sd[lane + 32 * t] = dph[t];
        z[t] = make_float2((float)(dph[t].x * yd[t]), (float)(dph[t].y * yd[t]));
      }
    }
    double2 v[NR], mv[NR];
    apply_q(w, n, z, false);
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      v[t] = make_double2(z[t].x, z[t].y);
      if (lane + 32 * t < n) w.v[lane + 32 * t] = v[t];
    }
    herm_matvec(w.ainv, coh + pts[pt] * npairs, n, v, sv, sv + n, mv);
    double lam;
    residual(v, mv, lam);
#pragma unroll
    for (int t = 0; t < NR; ++t) z[t] = make_float2((float)mv[t].x, (float)mv[t].y);
    apply_q(w, n, z, true);
#pragma unroll
    for (int t = 0; t < NR; ++t)  // D^H: times conj(delta_i)
      mv[t] = lane + 32 * t < n ? cmulc(make_double2(z[t].x, z[t].y), sd[lane + 32 * t]) : make_double2(0, 0);
    double yd[NR];
    unit_y(w.y, n, yd);
    project(yd, mv);
#pragma unroll
    for (int t = 0; t < NR; ++t)
      if (lane + 32 * t < n) w.x[lane + 32 * t] = mv[t];
    if (lane == 0) *w.lam = lam;
    __syncwarp();
  }
}

// x <- (R - lambda I)^-1 x of each point, one thread per point: kSolvePoints points per warp, their
// vectors in shared memory.
constexpr int kSolvePoints = 16;
inline size_t solve_smem(int n) { return (size_t)n * (kSolvePoints + 1) * (3 * sizeof(double) + sizeof(double2)); }

constexpr int kSolveThreads = 128;  // to fetch and store; kSolvePoints of them solve

__global__ void __launch_bounds__(kSolveThreads) refine_solve_kernel(PointSet pts, int n, unsigned char* __restrict__ ws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int P = kSolvePoints, S = P + 1;
  double2* x0 = reinterpret_cast<double2*>(smem_raw);
  double* s0 = reinterpret_cast<double*>(x0 + n * S);
  const int tid = threadIdx.x;
  const int64_t npt = pts.size();
  for (int64_t base = (int64_t)blockIdx.x * P; base < npt; base += (int64_t)gridDim.x * P) {
    const int here = (int)(npt - base < P ? npt - base : P);
#pragma unroll 4
    for (int f = tid; f < here * n; f += kSolveThreads) {
      const int q = f / n, i = f - q * n;
      const PointPtr<float, double> w(ws, base + q, n);
      x0[i * S + q] = w.x[i];
      s0[i * S + q] = (double)w.d[i];
      const float2 e = w.e[min(i, n - 2)];
      const double ex = e.x, ey = e.y;
      s0[(n + i) * S + q] = sqrt(ex * ex + ey * ey);  // entry n - 1 is not used
    }
    __syncthreads();
    if (tid < here) {
      const PointPtr<float, double> w(ws, base + tid, n);
      const double tiny = DBL_EPSILON * (double)w.scal[1] + DBL_MIN;
      // row i of d and b is read before the elimination overwrites it with its reciprocal pivot and
      // super-diagonal
      const double *d = s0 + tid, *b = s0 + n * S + tid;
      tridiag_solve<double>([&](int i) { return d[i * S]; }, [&](int i) { return b[i * S]; }, n, *w.lam, tiny, 1.0,
                            Strided<double2>{x0 + tid, S}, Strided<double>{s0 + tid, S},
                            Strided<double>{s0 + n * S + tid, S}, Strided<double>{s0 + 2 * n * S + tid, S});
    }
    __syncthreads();
#pragma unroll 4
    for (int f = tid; f < here * n; f += kSolveThreads) {
      const int q = f / n, i = f - q * n;
      const PointPtr<float, double> w(ws, base + q, n);
      w.x[i] = x0[i * S + q];
    }
    __syncthreads();
  }
}

template <int NR>
__global__ void __launch_bounds__(32 * kRefineWarps, 5) refine_check_kernel(
    const float2* __restrict__ coh, PointSet pts, int n, int ref, unsigned char* __restrict__ ws,
    uint8_t* __restrict__ sing, float2* __restrict__ ph, float* __restrict__ quality, float* __restrict__ tcoh,
    double tol) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double2* sv = reinterpret_cast<double2*>(smem_raw) + 2 * n * wid;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int64_t npt = pts.size();
  for (int64_t pt = (int64_t)blockIdx.x * kRefineWarps + wid; pt < npt; pt += (int64_t)gridDim.x * kRefineWarps) {
    const int64_t gp = pts[pt];
    const PointPtr<float, double> w(ws, pt, n);
    const float2* c = coh + gp * npairs;
    double2 v[NR], x[NR], dph[NR];
    double yd[NR];
    row_phases<double>(w, n, dph);
    unit_y(w.y, n, yd);
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const int i = lane + 32 * t;
      x[t] = i < n ? w.x[i] : make_double2(0, 0);
      v[t] = i < n ? w.v[i] : make_double2(0, 0);
    }
    project(yd, x);
    float2 z[NR];
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const double2 q = cmul(x[t], dph[t]);
      z[t] = make_float2((float)q.x, (float)q.y);
    }
    apply_q(w, n, z, false);
    double vn = 0;
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      v[t] = make_double2(v[t].x - (double)z[t].x, v[t].y - (double)z[t].y);
      vn += v[t].x * v[t].x + v[t].y * v[t].y;
    }
    vn = 1.0 / sqrt(warp_sum(vn));
#pragma unroll
    for (int t = 0; t < NR; ++t) v[t] = make_double2(v[t].x * vn, v[t].y * vn);
    double2 mv[NR];
    herm_matvec(w.ainv, c, n, v, sv, sv + n, mv);
    double lam;
    const double rn = residual(v, mv, lam);
    // phase error bound of the refined vector (v has unit length)
    double vmin = 1e300;
#pragma unroll
    for (int t = 0; t < NR; ++t)
      if (lane + 32 * t < n) vmin = fmin(vmin, sqrt(v[t].x * v[t].x + v[t].y * v[t].y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmin = fmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
    // |r'| / (gap min|v_i|) <= tol with gap = lambda_2(R) - lam - margin holds exactly when
    // lambda_2(R) >= sig = lam + margin + |r'| / (tol min|v_i|): one Sturm count at sig
    // (rounded up to FP32) answers it, without locating lambda_2
    const float eps = Lim<float>::eps(), tnorm = w.scal[1];
    const float pivmin = fmaxf(Lim<float>::tiny(), eps * eps * tnorm * tnorm) + Lim<float>::tiny();
    const double sig = lam + 4.0 * (double)eps * (double)n * (double)tnorm + rn / (tol * vmin);
    float* d = reinterpret_cast<float*>(sv);
    float* b2 = d + n;
    for (int i = lane; i < n; i += 32) {
      d[i] = w.d[i];
      if (i + 1 < n) {
        const double ex = w.e[i].x, ey = w.e[i].y;
        const float b = (float)sqrt(ex * ex + ey * ey);
        b2[i] = b * b;
      }
    }
    __syncwarp();
    float sg = (float)sig;
    if ((double)sg < sig) sg = nextafterf(sg, 3.4e38f);
    const bool gap_ok = sig < 3.0e38 && sturm_count(d, b2, n, sg, pivmin) <= 1;  // NaN: false
    const bool singular = (sing[pt] & kRouteSingular) != 0;
    const bool small_pivot = (sing[pt] & kRouteCond) != 0;  // the sweep's inverse is not trusted
    const bool ok = singular || (!small_pivot && gap_ok);
    __syncwarp();
    write_phases(v, n, ref, singular, ph + gp * n, sv);
    if (lane == 0) {
      quality[gp] = singular ? __int_as_float(0x7fffffff) : (float)lam;
      sing[pt] = singular ? kRouteSingular : (ok ? 0 : kRouteCond);
    }
    if (tcoh) {
      const float t = temp_coh_of(c, sv, n);
      if (lane == 0) tcoh[gp] = t;
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

// CTAs of a launch that walks `ctas` CTAs' worth of points: no more than are resident at once. One per SM
// always are, so that calls of few points, whose time is their launches', do not ask the runtime.
template <class K>
unsigned resident_grid(K kernel, int threads, size_t smem, int64_t ctas) {
  const int64_t sms = sm_count();
  return (unsigned)(ctas <= sms ? ctas : std::min<int64_t>(ctas, sms * std::max(1, occupancy(kernel, threads, smem))));
}

size_t point_bytes_max(int n) {
  return std::max({PointWs<float>(n).bytes, PointWs<double>(n).bytes, PointWs<float, double>(n).bytes});
}

// Most points of a sub-batch. Up to 128 images: per-point workspace within 4 GiB (about 34,000 points
// at N = 100), so that each launch has enough points to keep every SM busy to its end. Above, where a
// point has an SM to itself: whole waves of one point per SM, as many as 256 MiB hold, at least four
// (from 200 images on; with the slices less than the dense matrices of two points per SM). A sub-batch
// more costs its eigenpair and tail kernels' latency, 0.27 ms at N = 150: 5,224 points take 42.3 ms in
// one sub-batch (1,372 MiB with the inverse kept beside the reflectors), 43.0 as set here (235 MiB),
// 44.3 in waves of five (131 MiB). 1,000 points at N = 400 543 ms either way (2,026 and 911 MiB).
template <typename T>
int64_t sub_batch(int n) {
  const int64_t cap = g_sub_batch_cap.load();
  int64_t def;
  if (n > kMaxFastN) {
    const int64_t sms = sm_count(), wave = sms * (int64_t)PointWs<double, double, true>(n).bytes;
    def = std::max<int64_t>(4, ((int64_t)1 << 28) / wave) * sms;
  } else {
    const size_t bytes = sizeof(T) == 4 ? PointWs<float>(n).bytes : point_bytes_max(n);
    def = (int64_t)std::max<size_t>(1024, std::min<size_t>(1 << 17, ((size_t)1 << 32) / bytes));
  }
  return cap > 0 ? std::min(cap, def) : def;
}

// Workspace of one sub-batch of `sub` points: per-point state of the widest arithmetic
// used and the route flags of the FP32 and FP64 passes; then, for all `n_list` points of the
// call, the list of points to redo in FP64 and its count. The redo runs once after every
// sub-batch, so the few routed points of a call share launches instead of running a
// nearly empty pass per sub-batch.
// Slices start on a line of L2, whatever the points before them: a row's reads otherwise take a sector more
// each where n is a multiple of 4 (1,480 points, N = 176 39 ms at 16 or 48 bytes off, 33.5 on a line; 2,960, N =
// 200 140 and 112 ms).
constexpr size_t kSliceAlign = 128;

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
    const uintptr_t at = reinterpret_cast<uintptr_t>(b) + 16;
    slices = reinterpret_cast<unsigned char*>((at + kSliceAlign - 1) / kSliceAlign * kSliceAlign);
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
// thread) measured no faster than 16 in FP32 or FP64 with one point per SM, whose serial pivot
// steps set the pace. With look-ahead pivoting the 512-thread tile stayed in
// local memory (128 registers per thread), twice as slow.
template <typename T>
constexpr int gj_cx() { return 16; }

template <typename T, int NB, typename TW>
int launch_inverse(const float2* coh, PointSet pts, int64_t grid_cap, int n, unsigned char* ws, uint8_t* sing,
                   float cond_max, cudaStream_t s) {
  constexpr int CX = gj_cx<T>();
  const unsigned grid = resident_grid(inverse_kernel<T, NB, CX, TW>, 16 * CX, 0, grid_cap);
  KernelTimer kt(pts.list ? "emi inverse rerun" : sizeof(T) == 8 ? "emi inverse fp64" : "emi inverse fp32", s);
  inverse_kernel<T, NB, CX, TW><<<grid, 16 * CX, 0, s>>>(coh, pts, n, ws, sing, cond_max);
  return check_launch("emi inverse");
}

template <typename T, int NM, typename TW>
int launch_warp_inverse(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, float cond_max,
                        cudaStream_t s) {
  auto kernel = warp_inverse_kernel<T, NM, TW>;
  const int64_t ctas = (pts.n_pc + kWarpInvWarps - 1) / kWarpInvWarps;
  KernelTimer kt(pts.list ? "emi inverse rerun" : sizeof(T) == 8 ? "emi inverse fp64" : "emi inverse fp32", s);
  kernel<<<resident_grid(kernel, 32 * kWarpInvWarps, 0, ctas), 32 * kWarpInvWarps, 0, s>>>(c, pts, n, ws, sing,
                                                                                          cond_max);
  return check_launch("emi inverse");
}

// Most images with the reduction's FP64 triangle in shared memory.
constexpr int kReduceIn = 157;

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

// inv(|Gamma|) in arithmetic TA into a workspace laid out for a reduction in T.
template <typename TA, typename T>
int run_inverse(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, float cond_max,
                cudaStream_t s) {
  const int64_t cap = pts.n_pc;  // grid bound: the most points this pass can see
  switch ((n + 15) / 16) {
    case 1: return launch_warp_inverse<TA, 16, T>(c, pts, n, ws, sing, cond_max, s);
    case 2: return n <= 24 ? launch_warp_inverse<TA, 24, T>(c, pts, n, ws, sing, cond_max, s)
                           : launch_warp_inverse<TA, 32, T>(c, pts, n, ws, sing, cond_max, s);
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
  KernelTimer kt(pts.list ? "emi reduce rerun" : sizeof(T) == 8 ? "emi reduce fp64" : "emi reduce fp32", s);
  // one slice of the workspace per SM where the triangle is not in shared memory
  const int64_t most = kTriIn ? pts.n_pc : std::min<int64_t>(pts.n_pc, sm_count());
  kernel<<<resident_grid(kernel, 32 * W, rsmem, most), 32 * W, rsmem, s>>>(c, pts, n, ws, slices);
  return check_launch("emi reduce");
}

template <typename T, typename TA>
int run_reduce(const float2* c, PointSet pts, int n, unsigned char* ws, cudaStream_t s) {
  // Warps per point and rows per half-warp strip. Up to 64 images one warp needs no waiting on other
  // warps and an SM holds many points (FP64, N = 50, 4,001 points: one warp 0.78 ms, two 1.02);
  // above, shared memory holds two to four points per SM, and more warps each hide their latencies
  // (times of a build before the row sums had their own array; it takes 165 and 5.1 ms now):
  // N = 100, FP32, 1, 2, 4, 8 warps of 4 rows: 243, 222, 178, 285 ms for 286,294 points; FP64, 4 and 8
  // warps of 4 rows 6.5 and 6.2, of 2 rows (128 registers, two CTAs of 8 warps) 6.4 and 5.8 ms for
  // 4,001 points.
  constexpr bool f64 = sizeof(T) == 8;
  constexpr int W4 = 1, W8 = f64 ? 8 : 4, R8 = f64 ? 2 : 4;
  switch ((n + 15) / 16) {
    case 1: return launch_reduce<T, TA, 1, 4, 1>(c, pts, n, ws, s);
    case 2: return launch_reduce<T, TA, 2, 4, 1>(c, pts, n, ws, s);
    case 3: return launch_reduce<T, TA, 3, 4, W4>(c, pts, n, ws, s);
    case 4: return launch_reduce<T, TA, 4, 4, W4>(c, pts, n, ws, s);
    case 5: return launch_reduce<T, TA, 5, R8, W8>(c, pts, n, ws, s);
    case 6: return launch_reduce<T, TA, 6, R8, W8>(c, pts, n, ws, s);
    case 7:
      if constexpr (f64) {
        // The most warps with which two CTAs fit an SM's 228 KB (1 KB of each CTA is reserved): 8 up to
        // 107 images, 6 up to 109, 4 up to 111, 3 at 112. One CTA of 8 warps against these, 3,000
        // points: N = 108 7.44 and 4.46 ms, N = 110 (4 warps) 7.64 and 4.96, N = 112 7.86 and 5.78.
        auto two_fit = [&](int warps) { return 2 * (reduce_smem<T>(n, warps, true) + 1024) <= 228 * 1024; };
        if (!two_fit(8))
          return two_fit(6)   ? launch_reduce<T, TA, 7, 2, 6>(c, pts, n, ws, s)
                 : two_fit(4) ? launch_reduce<T, TA, 7, 4, 4>(c, pts, n, ws, s)
                              : launch_reduce<T, TA, 7, 4, 3>(c, pts, n, ws, s);
      }
      return launch_reduce<T, TA, 7, R8, W8>(c, pts, n, ws, s);
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

// Eigenpair of each point's tridiagonal.
template <typename T, typename TA, int G, bool kBig>
int launch_tri_eig(PointSet pts, int n, unsigned char* ws, cudaStream_t s) {
  const size_t smem = eig_smem<T>(n, G);
  auto kernel = tri_eig_kernel<T, TA, G, kBig>;
  if (int rc = allow_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  const int64_t ctas = (pts.n_pc + kEigThreads / G - 1) / (kEigThreads / G);
  kernel<<<resident_grid(kernel, kEigThreads, smem, ctas), kEigThreads, smem, s>>>(pts, n, ws);
  return check_launch("emi eigenpair");
}

template <typename T, typename TA, bool kBig = false>
int run_tri_eig(PointSet pts, int n, unsigned char* ws, cudaStream_t s) {
  // Lanes per point by the arithmetic alone: another number of sections moves the last bits of the
  // eigenvalue, and a point's result does not depend on the batch that it is in. FP32 8 (30,000 points at
  // N = 100: 4, 8, 16, 32 lanes 354, 275, 402, 673 us; 35,000 at N = 50 121, 146, 253, 400). FP64 16, of
  // 8, 16 and 32: few points are faster with more lanes (1,003 at N = 17 34, 30, 26 us; 1,332 at N = 150
  // 187, 165, 154), many with fewer (30,000 at N = 100 942, 904, 1,515; 35,000 at N = 50 339, 549, 893).
  return launch_tri_eig<T, TA, sizeof(T) == 4 ? 8 : 16, kBig>(pts, n, ws, s);
}

template <typename T, int NR>
int launch_tail(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
                unsigned char* ws, const uint8_t* sing, cudaStream_t s) {
  KernelTimer kt(pts.list ? "emi tail rerun" : sizeof(T) == 8 ? "emi tail fp64" : "emi tail fp32", s);
  if (int rc = run_tri_eig<T, T, (NR > 4)>(pts, n, ws, s)) return rc;
  const size_t tsmem = kTailWarps * (size_t)n * sizeof(double2);
  auto kernel = tail_kernel<T, T, NR>;
  if (int rc = allow_smem(reinterpret_cast<const void*>(kernel), tsmem)) return rc;
  const unsigned tgrid = resident_grid(kernel, 32 * kTailWarps, tsmem, (pts.n_pc + kTailWarps - 1) / kTailWarps);
  kernel<<<tgrid, 32 * kTailWarps, tsmem, s>>>(c, pts, n, ref, ws, sing, ph, quality, tcoh);
  return check_launch("emi tail");
}

// One pass of inverse, reduction, eigenpair and tail over a sub-batch (pts.list == nullptr: all
// pts.n_pc points; else the listed ones, whose count is read on the device), inverse and reduction
// both in T. cond_max > 0 flags the points whose condition estimate exceeds it.
template <typename T>
int run_pass(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
             unsigned char* ws, uint8_t* sing, float cond_max, void* slices, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    if (n > kMaxFastN) {
      if (int rc = run_big_inverse(c, pts, n, ws, sing, slices, s)) return rc;
      if (int rc = run_big_reduce(c, pts, n, ws, slices, s)) return rc;
      return n <= 256 ? launch_tail<T, 8>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s)
                      : launch_tail<T, 16>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s);
    }
  }
  if (int rc = run_inverse<T, T>(c, pts, n, ws, sing, cond_max, s)) return rc;
  if (int rc = run_reduce<T, T>(c, pts, n, ws, s)) return rc;
  return n <= 32   ? launch_tail<T, 1>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s)
         : n <= 64 ? launch_tail<T, 2>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s)
                   : launch_tail<T, 4>(c, pts, n, ref, ph, quality, tcoh, ws, sing, s);
}

template <int NB>
int launch_sweep(const float2* c, PointSet pts, int n, unsigned char* ws, uint8_t* sing, cudaStream_t s) {
  const unsigned grid = resident_grid(sweep_kernel<NB, float>, 256, 0, pts.n_pc);
  KernelTimer kt(pts.list ? "emi sweep rerun" : "emi sweep fp64", s);
  sweep_kernel<NB, float><<<grid, 256, 0, s>>>(c, pts, n, ws, sing);
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

template <int NR>
int launch_refine(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
                  unsigned char* ws, uint8_t* sing, double tol, cudaStream_t s) {
  KernelTimer kt("emi refine tail", s);
  if (int rc = run_tri_eig<float, double>(pts, n, ws, s)) return rc;
  const size_t wsmem = kRefineWarps * 3 * (size_t)n * sizeof(double2), ssmem = solve_smem(n);
  auto ka = refine_residual_kernel<NR>;
  auto kb = refine_check_kernel<NR>;
  if (int rc = allow_smem(reinterpret_cast<const void*>(ka), wsmem)) return rc;
  if (int rc = allow_smem(reinterpret_cast<const void*>(kb), wsmem)) return rc;
  if (int rc = allow_smem(reinterpret_cast<const void*>(refine_solve_kernel), ssmem)) return rc;
  auto grid = [&](auto kernel, int threads, size_t smem, int points) {
    return resident_grid(kernel, threads, smem, (pts.n_pc + points - 1) / points);
  };
  ka<<<grid(ka, 32 * kRefineWarps, wsmem, kRefineWarps), 32 * kRefineWarps, wsmem, s>>>(c, pts, n, ws);
  refine_solve_kernel<<<grid(refine_solve_kernel, kSolveThreads, ssmem, kSolvePoints), kSolveThreads, ssmem, s>>>(
      pts, n, ws);
  kb<<<grid(kb, 32 * kRefineWarps, wsmem, kRefineWarps), 32 * kRefineWarps, wsmem, s>>>(c, pts, n, ref, ws, sing, ph,
                                                                                       quality, tcoh, tol);
  return check_launch("emi refine tail", 3);
}

// The refined pass: FP64 inverse (symmetric sweep), FP32 reduction, FP64-refined tail;
// sing[] ends with the points whose sweep met a small pivot or whose refined error bound
// exceeds `tol` flagged kRouteCond.
int run_refine_pass(const float2* c, PointSet pts, int n, int ref, float2* ph, float* quality, float* tcoh,
                    unsigned char* ws, uint8_t* sing, double tol, cudaStream_t s) {
  if (int rc = run_sweep(c, pts, n, ws, sing, s)) return rc;
  if (int rc = run_reduce<float, double>(c, pts, n, ws, s)) return rc;
  return n <= 32   ? launch_refine<1>(c, pts, n, ref, ph, quality, tcoh, ws, sing, tol, s)
         : n <= 64 ? launch_refine<2>(c, pts, n, ref, ph, quality, tcoh, ws, sing, tol, s)
                   : launch_refine<4>(c, pts, n, ref, ph, quality, tcoh, ws, sing, tol, s);
}

}  // namespace

size_t fast_workspace_bytes(int64_t n_pc, int n) {
  if (n > kMaxFastN)  // FP64 only: no list of points to redo
    return SubWs::bytes(std::min<int64_t>(n_pc, sub_batch<double>(n)), PointWs<double, double, true>(n).bytes, 0) +
           std::min<int64_t>(n_pc, sm_count()) * slice_bytes(n) + kSliceAlign;
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
  const int64_t cap = wide ? sub_batch<double>(n) : sub_batch<float>(n);
  // sub-batches of equal size (none left nearly empty at the end); above 128 images full waves of one
  // point per SM and the rest
  const int64_t nsub = (n_pc + cap - 1) / cap;
  const int64_t sub = n > kMaxFastN ? std::min(cap, n_pc) : nsub > 0 ? (n_pc + nsub - 1) / nsub : 0;
  const size_t point = n > kMaxFastN ? PointWs<double, double, true>(n).bytes
                       : wide        ? point_bytes_max(n) : PointWs<float>(n).bytes;
  const SubWs w(ws, sub, point, n > kMaxFastN ? 0 : n_pc);
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
