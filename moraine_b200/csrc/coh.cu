// Coherence estimation on SIMT cores: the SHP-masked complex Gram of every point,
// normalised to coherence (point-cloud, upper-triangle compressed) or to covariance and
// coherence (raster, full N x N).
//
// Reference behaviour followed (kanglcn/moraine):
//   moraine/co.py:164-187  coh[i,q] = sum z_m conj(z_j) / sqrt(sum|z_m|^2 sum|z_j|^2) over the
//                          window pixels with pc_is_shp set that lie inside the image,
//                          summed in window order (row-major over the az x r window)
//   moraine/co.py:83-110   raster: cov = sum / n_shp, coh as above, every (m, j)
#include <algorithm>

#include "common.cuh"

namespace mr {
namespace {

// SHP rows staged per pass: `most`, or fewer (a power of two, at least 4) where `row_bytes` each
// would take more than 64 KiB.
int chunk_rows(int most, size_t row_bytes) {
  while (most > 4 && most * row_bytes > 64 * 1024) most >>= 1;
  return most;
}

// Block-wide compaction of a window mask into the linear pixel indices of the SHPs that
// lie inside the image, in window order. Returns the count (same in every thread).
__device__ int collect_shps(const uint8_t* __restrict__ mask, int az_win, int r_win, int ra, int rr,
                            int nlines, int width, int* __restrict__ s_pos, int* __restrict__ s_tmp) {
  const int win = az_win * r_win;
  const int azh = az_win / 2, rh = r_win / 2;
  const int per = (win + blockDim.x - 1) / blockDim.x;
  const int e0 = threadIdx.x * per, e1 = min(win, e0 + per);
  const int k0 = e0 / r_win, l0 = e0 - k0 * r_win;
  int c = 0;
  for (int e = e0, k = k0, l = l0; e < e1; ++e) {
    const int sa = ra - azh + k, sr = rr - rh + l;
    c += (mask[e] && sa >= 0 && sa < nlines && sr >= 0 && sr < width);
    if (++l == r_win) { l = 0; ++k; }
  }
  // block exclusive scan of c
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_tmp[wid] = incl;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    if (w < wid) before += s_tmp[w];
    total += s_tmp[w];
  }
  int pos = before + incl - c;
  for (int e = e0, k = k0, l = l0; e < e1; ++e) {
    const int sa = ra - azh + k, sr = rr - rh + l;
    if (mask[e] && sa >= 0 && sa < nlines && sr >= 0 && sr < width) s_pos[pos++] = sa * width + sr;
    if (++l == r_win) { l = 0; ++k; }
  }
  __syncthreads();
  return total;
}

// Out of line: called for a few values in 10^7, from a hundred places of an unrolled epilogue.
__device__ __noinline__ double quotient(double num, const double* am, const double* aj) {
  return num / sqrt(*am * *aj);
}

// (re, im) / sqrt(am aj) rounded to FP32, from f ~ 1 / sqrt(am aj): products in place of an FP64 root
// and two divisions, which are computed only where a product is within 16 FP64 ulps of the middle
// between two floats (its error is a few). The same floats as the quotients'.
__device__ __forceinline__ float2 normalised(double re, double im, double f, const double* am, const double* aj) {
  double x = re * f, y = im * f;
  const unsigned lx = (unsigned)__double2loint(x) & 0x1fffffffu, ly = (unsigned)__double2loint(y) & 0x1fffffffu;
  if (lx - 0x0ffffff0u < 32u || ly - 0x0ffffff0u < 32u) {
    x = quotient(re, am, aj);
    y = quotient(im, am, aj);
  }
  return make_float2((float)x, (float)y);
}

__device__ __forceinline__ void copy8(float2* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// One CTA per point (grid-stride), a 4 x 4 block of the Gram's upper triangle per thread and
// round, over the point's SHPs staged kc rows at a time. The launch gives a point only as many
// warps as its blocks fill; several CTAs share an SM.
// kOut = kTriu  : writes coh (n_pc, Q) in triu order.
// kOut = kRaster: writes cov and coh (npix, N, N) (raster form), the lower blocks as conjugates;
//        kRasterPairs: two values to a store (raster_pairs).
//
// A staged row holds its images in the arithmetic A, permuted so that the 16-byte words
// that a thread reads lie 16 bytes from its neighbour's (no bank conflict): image 4 b + r at
// position (r / V) V nb + V b + r % V, V images to a word.
// FP32: cp.async into two buffers; the products re re, im im, im re and re im are summed apart, S
// roundings each on partial sums of half the size: four FMAs per complex product (the sum of both
// products rounded into one accumulator took six instructions and was less exact). FP64: fetched
// by cp.async as stored, widened once when staged (at 16 conversions per clock and SM, widening at
// each use cost as much time as the products themselves), one FMA chain per component. The sums
// |z|^2 are the Gram's own diagonal in FP32 (blocks (b, b) come first, in round 0), and
// summed from the staged rows in FP64.
// FP32 is bound by its issue slots, FP64 by shared memory (eight 16-byte reads, four wavefronts
// each, take as long as their 64 FP64 FMAs). FP32, N = 50, 15 x 31 window, 30,011 points: 1.65 ms
// against 2.9 with a separate pass for |z|^2 and 256-thread CTAs; N = 20 raster of 123 x 131: 0.16
// against 0.38 ms. FP64 at N = 150, 8,000 points of 95 SHPs: 4.7 against 5.0 ms.
//
// A CTA has up to 192 threads, or up to 256, two of them per SM, where that takes a round less. FP32: N = 80,
// 4,000 points, 11 x 21 window 444 against 331 us, N = 112 735 and 620, N = 200 2,129 and 1,736 (with the
// same rounds the 256 lost: N = 68 74 against 76 % of the time of the kernel before). FP64, 15 x 31 window:
// 900 points, N = 150 1,153 against 960 us, N = 190 2,058 and 1,792, N = 320 6,457 and 5,549; 3,000 points,
// N = 174 4,739 and 3,873; one CTA of 256 threads and up to 255 registers was no faster than the 192.
constexpr int kGramThreads = 192, kWideGramThreads = 256;

template <typename A> struct GramAcc;
template <> struct GramAcc<float> {
  float rr, ii, ir, ri;
  __device__ __forceinline__ void add(float2 m, float2 j) {  // z_m conj(z_j)
    rr = fmaf(m.x, j.x, rr);
    ii = fmaf(m.y, j.y, ii);
    ir = fmaf(m.y, j.x, ir);
    ri = fmaf(m.x, j.y, ri);
  }
  __device__ __forceinline__ float re() const { return rr + ii; }
  __device__ __forceinline__ float im() const { return ir - ri; }
};
template <> struct GramAcc<double> {
  double x, y;
  __device__ __forceinline__ void add(double2 m, double2 j) {
    x = fma(m.x, j.x, x);
    x = fma(m.y, j.y, x);
    y = fma(m.y, j.x, y);
    y = fma(-m.x, j.y, y);
  }
  __device__ __forceinline__ double re() const { return x; }
  __device__ __forceinline__ double im() const { return y; }
};

// amp2[c] (+)= sum of |z|^2 of each image over ns staged rows (image c at at(c)), each |z|^2 rounded
// once (its two products are exact in FP64) and added in row order.
template <class At>
__device__ __forceinline__ void sum_squares(const double2* rows, int stride, int n, int ns, bool first, double* amp2,
                                            At at) {
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    const double2* z = rows + at(c);
    double s = first ? 0.0 : amp2[c];
#pragma unroll 4
    for (int t = 0; t < ns; ++t) s += fma(z[t * stride].x, z[t * stride].x, z[t * stride].y * z[t * stride].y);
    amp2[c] = s;
  }
}

// Images 4 b .. 4 b + 3 of a staged row.
__device__ __forceinline__ void load_block(const float2* row, int nb, int b, float2 (&z)[4]) {
  const float4 u = reinterpret_cast<const float4*>(row)[b], v = reinterpret_cast<const float4*>(row)[nb + b];
  z[0] = make_float2(u.x, u.y);
  z[1] = make_float2(u.z, u.w);
  z[2] = make_float2(v.x, v.y);
  z[3] = make_float2(v.z, v.w);
}
__device__ __forceinline__ void load_block(const double2* row, int nb, int b, double2 (&z)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) z[r] = row[r * nb + b];
}

enum GramOut { kTriu, kRaster, kRasterPairs };

// Columns col and col + 1 of a row of n values, n even and the row 16-byte aligned.
__device__ __forceinline__ void put2(float2* row, int col, int n, float px, float py, float qx, float qy) {
  if (col < n) *reinterpret_cast<float4*>(row + col) = make_float4(px, py, qx, qy);
}

// Rows 4 bm + a and the next of a finished block of coherence (rr, ii) and covariance (ir, ri), and off the
// diagonal their conjugate transpose.
__device__ __forceinline__ void write_rows(float2* coh, float2* cov, int n, int bm, int bj, int a,
                                           const GramAcc<float> (&v)[2][4]) {
  const int m = 4 * bm + a, j = 4 * bj;
  if (m >= n) return;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int b = 0; b < 4; b += 2) {
      const GramAcc<float> &p = v[r][b], &q = v[r][b + 1];
      put2(coh + (m + r) * n, j + b, n, p.rr, p.ii, q.rr, q.ii);
      put2(cov + (m + r) * n, j + b, n, p.ir, p.ri, q.ir, q.ri);
    }
  if (bm == bj) return;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (j + b < n) {
      const GramAcc<float> &p = v[0][b], &q = v[1][b];
      put2(coh + (j + b) * n, m, n, p.rr, -p.ii, q.rr, -q.ii);
      put2(cov + (j + b) * n, m, n, p.ir, -p.ri, q.ir, -q.ri);
    }
}

template <typename A, GramOut kOut, int MT>
__global__ void __launch_bounds__(MT, sizeof(A) == 8 || MT == kWideGramThreads ? 2 : 3) gram_kernel(
    const float2* __restrict__ rslc, int nlines, int width, int n, const int32_t* __restrict__ idx,
    int64_t n_pc, const uint8_t* __restrict__ mask, int mask_stride, int az_win, int r_win,
    float2* __restrict__ coh, float2* __restrict__ cov, const int64_t* __restrict__ dcount, int64_t doff, int kc) {
  using C = typename cplx<A>::type;
  constexpr bool kWide = sizeof(A) == 8, kFull = kOut != kTriu;
  constexpr int V = 16 / sizeof(C);  // images per 16-byte word
  if (dcount) {  // points doff .. doff + n_pc - 1 of a count held on the device
    const int64_t c = *dcount - doff;
    n_pc = c < 0 ? 0 : (c < n_pc ? c : n_pc);
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int win = az_win * r_win;
  const int nb = (n + 3) >> 2, npad = 4 * nb;
  C* zc = reinterpret_cast<C*>(smem_raw);                             // FP32: 2 x kc x npad; FP64: kc x npad
  float2* raw = reinterpret_cast<float2*>(zc + (kWide ? 1 : 2) * kc * npad);  // FP64: kc x n, as fetched
  A* amp2 = reinterpret_cast<A*>(raw + (kWide ? kc * n + (kc * n & 1) : 0));  // npad
  A* rinv = amp2 + npad;                                              // FP64: npad
  int* s_pos = reinterpret_cast<int*>(amp2 + (kWide ? 2 : 1) * npad);  // win
  __shared__ int s_tmp[32];
  const int nblk = nb * (nb + 1) / 2;
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < (kWide ? 1 : 2) * kc * npad; e += nt) zc[e] = cmake<C>(0, 0);  // padding images stay 0
  // thread's staging walk over (row t, image c): nt elements ahead is (sdt, sdc)
  const int t_first = tid / n, c_first = tid - t_first * n;
  const int sdt = nt / n, sdc = nt - sdt * n;
  const int rounds = (nblk + nt - 1) / nt;
  __syncthreads();

  for (int64_t i = blockIdx.x; i < n_pc; i += gridDim.x) {
    int ra, rr;
    if (idx) { ra = idx[2 * i]; rr = idx[2 * i + 1]; }
    else { ra = (int)(i / width); rr = (int)(i % width); }
    if (ra < 0 || ra >= nlines || rr < 0 || rr >= width) {  // index outside the image: NaN row
      const float2 nan2 = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
      if (kFull) {
        for (int e = tid; e < n * n; e += nt) { coh[i * n * n + e] = nan2; cov[i * n * n + e] = nan2; }
      } else {
        for (int64_t e = tid; e < npairs; e += nt) coh[i * npairs + e] = nan2;
      }
      continue;
    }
    const uint8_t* m = mask + (mask_stride ? ((int64_t)ra * width + rr) : i) * win;
    const int S = collect_shps(m, az_win, r_win, ra, rr, nlines, width, s_pos, s_tmp);
    // fn(row t, image c) over this thread's elements of ns rows
    auto each = [&](int ns, auto fn) {
      int t = t_first, c = c_first;
      while (t < ns) {
        fn(t, c);
        t += sdt;
        c += sdc;
        if (c >= n) { c -= n; ++t; }
      }
    };
    auto place = [&](int t, int c) { return t * npad + (c & 3) / V * V * nb + (c >> 2) * V + (c & 3) % V; };
    auto fetch = [&](int s0, int buf) {
      each(min(kc, S - s0), [&](int t, int c) {
        const float2* src = rslc + (int64_t)s_pos[s0 + t] * n + c;
        if constexpr (kWide) copy8(raw + t * n + c, src);
        else copy8(reinterpret_cast<float2*>(zc) + buf * kc * npad + place(t, c), src);
      });
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (kWide) {
      if (S == 0)
        for (int c = tid; c < n; c += nt) amp2[c] = 0;
    }
    for (int round = 0; round < rounds; ++round) {
      const int blk = round * nt + tid;
      const bool active = blk < nblk;
      int bm = 0, bj = 0;
      if (active) {  // the diagonal blocks, then the rest row by row
        if (blk < nb) { bm = bj = blk; }
        else {
          int q = blk - nb;
          while (q >= nb - 1 - bm) { q -= nb - 1 - bm; ++bm; }
          bj = bm + 1 + q;
        }
      }
      GramAcc<A> acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = {};
      if (S > 0) fetch(0, 0);
      int buf = 0;
      for (int s0 = 0; s0 < S; s0 += kc) {
        const int ns = min(kc, S - s0);
        const C* row = zc;
        if constexpr (kWide) {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          each(ns, [&](int t, int c) {  // what this thread fetched
            const float2 z = raw[t * n + c];
            zc[place(t, c)] = cmake<C>((A)z.x, (A)z.y);
          });
          if (s0 + kc < S) fetch(s0 + kc, 0);
        } else {
          if (s0 + kc < S) {
            fetch(s0 + kc, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
          } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
          }
          row += buf * kc * npad;
          buf ^= 1;
        }
        __syncthreads();
        if constexpr (kWide) {
          if (round == 0) sum_squares(zc, npad, n, ns, s0 == 0, amp2, [&](int c) { return place(0, c); });
        }
        if (active) {
#pragma unroll 2
          for (int t = 0; t < ns; ++t, row += npad) {
            C zm[4], zj[4];
            load_block(row, nb, bm, zm);
            load_block(row, nb, bj, zj);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
              for (int b = 0; b < 4; ++b) acc[a][b].add(zm[a], zj[b]);
          }
        }
        __syncthreads();  // the rows are overwritten by the next pass
      }
      if (round == 0) {
        if constexpr (kWide) {
          for (int c = tid; c < n; c += nt) rinv[c] = (A)1 / sqrt(amp2[c]);
        } else if (blk < nb) {
#pragma unroll
          for (int a = 0; a < 4; ++a) amp2[4 * blk + a] = acc[a][a].re();
        }
        __syncthreads();
      }
      if constexpr (kOut == kRasterPairs) {
        if (active) {
          const int64_t o = i * n * n;
#pragma unroll
          for (int a = 0; a < 4; a += 2) {
            GramAcc<float> v[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                const A den = sqrt(amp2[4 * bm + a + r] * amp2[4 * bj + b]);
                const A re = acc[a + r][b].re(), im = acc[a + r][b].im();
                v[r][b] = {re / den, im / den, re / (A)S, im / (A)S};
              }
            write_rows(coh + o, cov + o, n, bm, bj, a, v);
          }
        }
      } else if (active) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int mm = 4 * bm + a, jj = 4 * bj + b;
            if (mm >= n || jj >= n || mm > jj) continue;
            const A re = acc[a][b].re(), im = acc[a][b].im();
            float2 g;
            if constexpr (kWide) {
              const A f = rinv[mm] * rinv[jj];
              g = normalised(re, im, f, amp2 + mm, amp2 + jj);
            } else {
              const A den = sqrt(amp2[mm] * amp2[jj]);
              g = make_float2(re / den, im / den);
            }
            if (kFull) {
              const float2 v = make_float2((float)(re / (A)S), (float)(im / (A)S));
              const int64_t o = (i * n + mm) * n + jj, ot = (i * n + jj) * n + mm;
              coh[o] = g;
              cov[o] = v;
              if (mm != jj) {
                coh[ot] = make_float2(g.x, -g.y);
                cov[ot] = make_float2(v.x, -v.y);
              }
            } else if (mm < jj) {
              coh[i * npairs + triu_index(mm, jj, n)] = g;
            }
          }
      }
    }
    __syncthreads();  // s_pos and amp2 are rewritten for the next point
  }
}

// FP64 up to kDmmaImages images on the FP64 tensor instruction (DMMA m16n8k8). It has the rate of
// the FP64 pipe, 64 FMA per clock and SM, but reads each operand from shared memory once per
// 16 x 8 block instead of once per 4 x 4. With k = 2 s + {re, im} as the contraction index,
// A[m][k] = z_m's component k:
//   Re = sum_k A[m][k] A[j][k],   Im = sum_k X[m][k] Y[j][k],  X = (im, re), Y = (re, -im),
// two products of real matrices with 2 S rows and no redundant sum, each added up in the order of
// gram_kernel's FMA chain. Every fragment is plain 8-byte reads of the staged rows (image
// lane / 4, k = lane % 4); Y is a sign on A's.
//
// The upper triangle is cut into 16 x 8 blocks, and the blocks into runs of at most SLOTS that
// span one or two block rows (plan_gram64); a run is one warp's accumulators, its A fragments are
// read once or twice per step and its other addresses are a base and a constant (nothing issues
// beside a DMMA, so every instruction counts: with a next-block rule per slot it took 5.9 ms
// below, on m8n8k4 7.9 ms). Four warps of 13 blocks hold 104 images in one pass over the SHPs,
// two such CTAs per SM, eight of 9 hold 128; smaller runs leave room for more warps (plan_gram64).
// N = 100, 11 x 21 window, 20,000 points: 5.2 ms against 6.4 (one CTA of 256 threads, samples
// widened at each use) and 5.5 with gram_kernel<double>; N = 64 1.9 against 3.3 and 2.8; N = 50,
// 35,627 points: 2.5 against 4.6. The exact sums |z|^2 and the
// rounding test of `normalised` are 0.4 ms of the 5.2: without them a few coherences in 10^8 round
// to the other float, which the EMI of a nearly singular point magnifies to milliradians.
constexpr int kMaxRuns = 8;
constexpr int kDmmaImages = 128;

// Run r: blocks (br1, bc1 ...) c1 of them, then (br2, bc2 ...) up to cnt.
struct GramRun {
  uint8_t br1, bc1, c1, br2, bc2, cnt;
};
struct GramPlan {
  int warps, runs, slots;  // slots: the longest run
  GramRun run[kMaxRuns];
};

__device__ __forceinline__ void dmma(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// CTAs per SM that the registers are cut to, of `warps` warps with `slots` blocks of accumulators each.
constexpr int gram64_ctas(int slots, int warps) {
  return warps == 4 ? (slots <= 4 ? 4 : slots <= 7 ? 3 : 2) : warps * slots <= 42 ? 2 : 1;
}

template <int SLOTS, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, gram64_ctas(SLOTS, WARPS)) gram64_kernel(
    const float2* __restrict__ rslc, int nlines, int width, int n, const int32_t* __restrict__ idx,
    int64_t n_pc, const uint8_t* __restrict__ mask, int mask_stride, int az_win, int r_win,
    float2* __restrict__ coh, const int64_t* __restrict__ dcount, int64_t doff, int kc,
    const __grid_constant__ GramPlan plan) {
  if (dcount) {
    const int64_t c = *dcount - doff;
    n_pc = c < 0 ? 0 : (c < n_pc ? c : n_pc);
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int win = az_win * r_win;
  const int nr = (n + 15) >> 4;
  const int npd = 16 * nr + 4;  // images of a staged row: = 4 mod 8, so that the two rows that a
                                // fragment read spans lie on different banks
  double2* zc = reinterpret_cast<double2*>(smem_raw);             // kc (a multiple of 4) x npd
  double* rinv = reinterpret_cast<double*>(zc + kc * npd);         // 16 nr: 1 / sqrt(sum |z|^2)
  double* amp2 = rinv + 16 * nr;                                   // 16 nr: sum |z|^2
  float2* raw = reinterpret_cast<float2*>(amp2 + 16 * nr);         // kc x n, as fetched
  int* s_pos = reinterpret_cast<int*>(raw + kc * n);               // win
  __shared__ int s_tmp[32];
  const int64_t npairs = (int64_t)n * (n - 1) / 2;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
  for (int e = tid; e < kc * npd; e += nt) zc[e] = make_double2(0.0, 0.0);  // padding images stay 0
  // thread's staging walk over (row t, image c): nt elements ahead is (sdt, sdc)
  const int t_first = tid / n, c_first = tid - t_first * n;
  const int sdt = nt / n, sdc = nt - sdt * n;
  const int comp = lane & 1;
  const double* zk = reinterpret_cast<const double*>(zc + ((lane >> 1) & 1) * npd + (lane >> 2));
  const int k4 = 4 * npd;  // doubles from k to k + 4: two staged rows
  const int row = lane >> 2, colp = 2 * (lane & 3);  // of accumulators 0 and 1; 2 and 3 are 8 rows on
  __syncthreads();

  for (int64_t i = blockIdx.x; i < n_pc; i += gridDim.x) {
    const int ra = idx[2 * i], rr = idx[2 * i + 1];
    if (ra < 0 || ra >= nlines || rr < 0 || rr >= width) {  // index outside the image: NaN row
      const float2 nan2 = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
      for (int64_t e = tid; e < npairs; e += nt) coh[i * npairs + e] = nan2;
      continue;
    }
    const uint8_t* m = mask + (mask_stride ? ((int64_t)ra * width + rr) : i) * win;
    const int S = collect_shps(m, az_win, r_win, ra, rr, nlines, width, s_pos, s_tmp);
    // rows s0 .. of the point's samples on their way to `raw`; a thread widens what it fetched
    auto fetch = [&](int s0) {
      const int ns = min(kc, S - s0);
      int t = t_first, c = c_first;
      while (t < ns) {
        copy8(raw + t * n + c, rslc + (int64_t)s_pos[s0 + t] * n + c);
        t += sdt;
        c += sdc;
        if (c >= n) { c -= n; ++t; }
      }
    };
    int w = wid;
    asm volatile("" : "+r"(w));  // the run is read for each point: kept over the loop it costs spills
    const GramRun run = plan.run[w];
    const int cnt = run.cnt, c1 = run.c1;
    const int a1 = 32 * run.br1, a2 = 32 * run.br2;
    const int b1 = 16 * run.bc1, b2 = 16 * ((int)run.bc2 - c1);
    double re[SLOTS][4], im[SLOTS][4];
#pragma unroll
    for (int q = 0; q < SLOTS; ++q)
#pragma unroll
      for (int h = 0; h < 4; ++h) re[q][h] = im[q][h] = 0.0;
    fetch(0);
    for (int s0 = 0; s0 < S; s0 += kc) {
      const int ns = min(kc, S - s0);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // the previous rows have been used
      {
        int t = t_first, c = c_first;
        while (t < ns) {
          const float2 z = raw[t * n + c];
          zc[t * npd + c] = make_double2((double)z.x, (double)z.y);
          t += sdt;
          c += sdc;
          if (c >= n) { c -= n; ++t; }
        }
      }
      for (int r = ns; r & 3; ++r)  // a fragment takes four rows
        for (int c2 = tid; c2 < n; c2 += nt) zc[r * npd + c2] = make_double2(0.0, 0.0);
      fetch(s0 + kc);
      __syncthreads();
      sum_squares(zc, npd, n, ns, s0 == 0, amp2, [](int c) { return c; });
      const double* z = zk;
      for (int t = 0; t < ns; t += 4, z += 2 * k4) {
        double a[4], x[4];  // rows lane / 4 + 8 (h % 2), k = lane % 4 + 4 (h / 2)
        auto load_a = [&](const double* p, const double* o) {
          a[0] = p[0];
          a[1] = p[16];
          a[2] = p[k4];
          a[3] = p[k4 + 16];
          x[0] = o[0];
          x[1] = o[16];
          x[2] = o[k4];
          x[3] = o[k4 + 16];
        };
        load_a(z + a1 + comp, z + a1 + (comp ^ 1));
        const double* p = z + b1 + comp;
#pragma unroll
        for (int q = 0; q < SLOTS; ++q) {
          if (q < cnt) {
            if (q == c1) {
              load_a(z + a2 + comp, z + a2 + (comp ^ 1));
              p = z + b2 + comp;
            }
            double b[2] = {p[16 * q], p[16 * q + k4]};
            dmma(re[q], a, b);
            b[0] = comp ? -b[0] : b[0];
            b[1] = comp ? -b[1] : b[1];
            dmma(im[q], x, b);
          }
        }
      }
    }
    for (int c = tid; c < n; c += nt) rinv[c] = 1.0 / sqrt(S > 0 ? amp2[c] : 0.0);
    if (S == 0)
      for (int c = tid; c < n; c += nt) amp2[c] = 0.0;
    __syncthreads();
    float2* out = coh + i * npairs;
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
      if (q < cnt) {
        const int br = q < c1 ? run.br1 : run.br2, bc = q < c1 ? run.bc1 + q : run.bc2 + q - c1;
        const int jj = 8 * bc + colp;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int mm = 16 * br + row + 8 * (h >> 1), j = jj + (h & 1);
          if (mm < j && j < n) {
            out[mm * n - ((mm * (mm + 1)) >> 1) - mm - 1 + j] =  // triu_index(mm, j, n)
                normalised(re[q][h], im[q][h], rinv[mm] * rinv[j], amp2 + mm, amp2 + j);
          }
        }
      }
    }
    __syncthreads();  // s_pos and rinv are rewritten for the next point
  }
}

// Runs of at most `cap` blocks for n images: each block row br has the blocks bc = 2 br .. nc - 1,
// cut into pieces of cap; what is left of each row is paired with another rest, longest with the
// longest that still fits. No heap: the plan is made inside a C entry point, at each call.
GramPlan cut_gram64(int n, int cap) {
  struct Piece { int br, bc, len; };
  const int nc = (n + 7) / 8, nr = (n + 15) / 16;
  GramPlan plan{};
  Piece rest[kDmmaImages / 16];  // longest first
  int left = 0;
  auto add = [&](Piece a, Piece b) {
    if (plan.runs < kMaxRuns)
      plan.run[plan.runs] = {(uint8_t)a.br, (uint8_t)a.bc, (uint8_t)a.len, (uint8_t)b.br, (uint8_t)b.bc,
                             (uint8_t)(a.len + b.len)};
    ++plan.runs;
    plan.slots = std::max(plan.slots, a.len + b.len);
  };
  for (int br = 0; br < nr; ++br) {
    int bc = 2 * br;
    for (; nc - bc >= cap; bc += cap) add({br, bc, cap}, {0, 0, 0});
    if (bc >= nc) continue;
    int at = left++;
    for (; at > 0 && rest[at - 1].len < nc - bc; --at) rest[at] = rest[at - 1];
    rest[at] = {br, bc, nc - bc};
  }
  for (int i = 0; i < left; ++i) {
    if (rest[i].len == 0) continue;  // taken
    int j = i + 1;
    while (j < left && (rest[j].len == 0 || rest[i].len + rest[j].len > cap)) ++j;
    add(rest[i], j < left ? rest[j] : Piece{0, 0, 0});
    if (j < left) rest[j].len = 0;
  }
  plan.warps = plan.runs;
  return plan;
}

// The cut for n images into at most `warps` runs of at most `most` blocks whose longest run is the
// shortest (runs = 0: there is none).
GramPlan fit_gram64(int n, int warps, int most) {
  const int nc = (n + 7) / 8, nr = (n + 15) / 16, blocks = nr * nc - nr * (nr - 1);
  for (int cap = (blocks + warps - 1) / warps; cap <= most; ++cap) {
    const GramPlan p = cut_gram64(n, cap);
    if (p.runs <= warps) return p;
  }
  return {};
}

// A CTA's shape: its warps and the accumulator blocks that each may hold. The first shape that the
// images fit is taken, in an order by warps resident per SM (16, 12 or 8, by registers) and by how
// evenly the blocks fill the runs. Times of 4,000 points, 11 x 21 window, in us, with four warps, with
// gram_kernel<double>, and as dispatched:
//   up to 72 images  four warps of up to 7    N = 64: 364, 499, 364 (six warps 424, eight 403)
//   up to 80         eight warps of 4         N = 76: 682, 507, 493
//   up to 96         six warps of 6 or 7      N = 84: 791, 759, 617;  N = 96: 846, 897, 689
//   up to 104        four warps of 13         N = 104: 945, 978, 945 (eight warps of 7: 1,023)
//   up to 128        eight warps of 7 to 9    N = 112: -, 1,242, 1,022;  N = 124: -, 1,366, 1,265
// From 129 to 144 images eight warps of 11 or 12 blocks lose as often as they win (4,000 points, N = 132
// 1,750 against 1,502 us with gram_kernel, N = 144 1,809 against 1,885); above, the accumulators need
// several passes over the SHPs (N = 150, 5,224 points of 166 SHPs: 6.4 against 5.2 ms).
// 57 to 60 images, padded to 64 here, fill 120 of 128 threads of gram_kernel: N = 60 327 against 361 us.
// 105 to 108, padded to 112, fill 378 of its 384: N = 105 992 against 1,018 us, but 900 points 269
// against 253 us: there with more than 16 points per SM.
// Few points, at most two per SM, end sooner with more warps each whatever the images (200 points,
// 11 x 21 window, N = 64 58 against 62 us, N = 104 98 against 108; with six per SM that lost: N = 64,
// 900 points 118 against 111). At most one per SM: eight warps always (148 points, N = 84 44 against 56 us
// with six, N = 96 50 against 60; but 296 points, N = 84 81 against 67).
// Up to 24 images one warp can hold all blocks of a point; it wastes no step on an idle warp, but a
// point takes longer, so it is taken where every SM has more than 32 points (11 x 21 window, 20,000
// points: N = 17 438 against 550 us, N = 24 448 against 567; 5,000 points 152 against 153 and 156
// against 155; 2,000 points of a 15 x 31 window, N = 24: 165 against 114).
constexpr int kOneWarpImages = 24;

struct GramShape {
  int warps, slots;
};
constexpr GramShape kManyPoints[] = {{4, 7}, {8, 4}, {6, 7}, {4, 13}, {8, 9}};
constexpr GramShape kTwoPerSm[] = {{8, 4}, {6, 7}, {8, 9}};
constexpr GramShape kOnePerSm[] = {{8, 9}};

// The plan, and in `shape` the CTA shape of the kernel that holds it.
GramPlan plan_gram64(int n, int64_t n_pc, int sms, GramShape& shape) {
  shape = {4, 4};
  if (n <= kOneWarpImages && n_pc > (int64_t)sms * 32) return cut_gram64(n, 4);
  GramPlan plan{};
  auto first = [&](const auto& shapes) {
    for (const GramShape& s : shapes) {
      plan = fit_gram64(n, s.warps, s.slots);
      if (plan.runs) {
        if (plan.runs > 4) shape = s;
        else shape = {4, plan.slots};
        return;
      }
    }
  };
  if (n_pc <= sms) first(kOnePerSm);
  else if (n_pc <= (int64_t)sms * 2) first(kTwoPerSm);
  else first(kManyPoints);
  return plan;
}

// Whether gram64_kernel takes n images.
bool dmma_images(int n, int64_t n_pc, int sms) {
  if (n > 56 && n <= 60) return false;
  if (n > 104 && n <= 108 && n_pc > (int64_t)sms * 16) return false;
  return n <= kDmmaImages;
}

// Arbitrary pair lists: one thread per (point, pair), serial over the window.
__global__ void gram_pairs_kernel(const float2* __restrict__ rslc, int nlines, int width, int n,
                                  const int32_t* __restrict__ idx, int64_t n_pc,
                                  const uint8_t* __restrict__ mask, int mask_stride, int az_win,
                                  int r_win, const int32_t* __restrict__ pairs, int npairs,
                                  float2* __restrict__ coh) {
  const int64_t total = n_pc * npairs;
  const int azh = az_win / 2, rh = r_win / 2, win = az_win * r_win;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / npairs;
    const int q = (int)(e - i * npairs);
    const int mm = pairs[2 * q], jj = pairs[2 * q + 1];
    const int ra = idx[2 * i], rr = idx[2 * i + 1];
    if (mm < 0 || mm >= n || jj < 0 || jj >= n || ra < 0 || ra >= nlines || rr < 0 || rr >= width) {
      coh[e] = make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
      continue;
    }
    const uint8_t* m = mask + (mask_stride ? ((int64_t)ra * width + rr) : i) * win;
    float nr = 0.f, ni = 0.f, am = 0.f, aj = 0.f;
    for (int k = 0; k < az_win; ++k)
      for (int l = 0; l < r_win; ++l) {
        const int sa = ra - azh + k, sr = rr - rh + l;
        if (m[k * r_win + l] && sa >= 0 && sa < nlines && sr >= 0 && sr < width) {
          const float2 zm = rslc[((int64_t)sa * width + sr) * n + mm];
          const float2 zj = rslc[((int64_t)sa * width + sr) * n + jj];
          am += zm.x * zm.x + zm.y * zm.y;
          aj += zj.x * zj.x + zj.y * zj.y;
          nr += zm.x * zj.x + zm.y * zj.y;
          ni += zm.y * zj.x - zm.x * zj.y;
        }
      }
    const float den = sqrtf(am * aj);
    coh[e] = make_float2(nr / den, ni / den);
  }
}

// Points of a launch: enough CTAs to fill the device several times over (their SHP counts, and
// so their times, differ), each walking its share.
template <class K>
unsigned gram_grid(K kernel, int threads, size_t smem, int64_t n_pc) {
  if (n_pc <= (int64_t)sm_count() * 8) return (unsigned)n_pc;  // whatever the occupancy
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess || occ < 1) occ = 1;
  return (unsigned)std::min<int64_t>(n_pc, (int64_t)sm_count() * occ * 8);
}

template <typename A, GramOut kOut, int MT>
int launch_gram_of(const float2* rslc, int nlines, int width, int n, const int32_t* idx, int64_t n_pc,
                   const uint8_t* mask, int mask_stride, int az_win, int r_win, float2* coh, float2* cov,
                   cudaStream_t s, const int64_t* dcount, int64_t doff) {
  using C = typename cplx<A>::type;
  constexpr bool kWide = sizeof(A) == 8;
  const int nb = (n + 3) / 4, nblk = nb * (nb + 1) / 2;
  // no more warps than the blocks fill; all but the last round run full
  const int threads = std::min(MT, (nblk + 31) / 32 * 32);
  const size_t row = (size_t)(kWide ? 1 : 2) * 4 * nb * sizeof(C);
  const int kc = chunk_rows(kWide ? 16 : 32, row);
  const size_t smem = kc * row + (kWide ? ((size_t)kc * n + 1) / 2 * 2 * sizeof(float2) : 0) + (kWide ? 2 : 1) * 4 * nb * sizeof(A) +
                      (size_t)az_win * r_win * sizeof(int);
  if (int rc = allow_smem(reinterpret_cast<const void*>(gram_kernel<A, kOut, MT>), smem)) return rc;
  KernelTimer kt(kWide ? "gram fp64" : "gram fp32", s);
  gram_kernel<A, kOut, MT><<<gram_grid(gram_kernel<A, kOut, MT>, threads, smem, n_pc), threads, smem, s>>>(
      rslc, nlines, width, n, idx, n_pc, mask, mask_stride, az_win, r_win, coh, cov, dcount, doff, kc);
  return check_launch("coherence gram");
}

// Two values to a store in the raster form: the transposed blocks' values go to a row each, 32 lines to an
// instruction, which takes most of the time of long stacks with few SHPs. 50 x 51 pixels, 3 x 3 window, N = 64
// 155 us one by one and 95 in pairs, N = 80 216 and 145; 15 x 31 window 323 and 309, 460 and 421. Below 24
// images the pairs' registers cost more than the stores (N = 20, 3 x 3: 20 and 22).
bool raster_pairs(int n, const float2* coh, const float2* cov) {
  return n >= 24 && !(n & 1) && !((reinterpret_cast<uintptr_t>(coh) | reinterpret_cast<uintptr_t>(cov)) & 15);
}

template <typename A, GramOut kOut>
int launch_gram(const float2* rslc, int nlines, int width, int n, const int32_t* idx, int64_t n_pc,
                const uint8_t* mask, int mask_stride, int az_win, int r_win, float2* coh, float2* cov,
                cudaStream_t s, const int64_t* dcount = nullptr, int64_t doff = 0) {
  const int nb = (n + 3) / 4, nblk = nb * (nb + 1) / 2;
  auto rounds = [&](int threads) { return (nblk + threads - 1) / threads; };
  const bool wide = rounds(kWideGramThreads) < rounds(kGramThreads);
  return wide ? launch_gram_of<A, kOut, kWideGramThreads>(rslc, nlines, width, n, idx, n_pc, mask, mask_stride, az_win,
                                                          r_win, coh, cov, s, dcount, doff)
              : launch_gram_of<A, kOut, kGramThreads>(rslc, nlines, width, n, idx, n_pc, mask, mask_stride, az_win,
                                                      r_win, coh, cov, s, dcount, doff);
}

int launch_gram64(const float2* rslc, int nlines, int width, int n, const int32_t* idx, int64_t n_pc,
                  const uint8_t* mask, int mask_stride, int az_win, int r_win, float2* coh, cudaStream_t s,
                  const int64_t* dcount = nullptr, int64_t doff = 0) {
  const int sms = sm_count();
  if (!dmma_images(n, n_pc, sms))
    return launch_gram<double, kTriu>(rslc, nlines, width, n, idx, n_pc, mask, mask_stride, az_win, r_win, coh,
                                      nullptr, s, dcount, doff);
  const int nr = (n + 15) / 16;
  GramShape shape;
  const GramPlan plan = plan_gram64(n, n_pc, sms, shape);
  const int threads = 32 * plan.warps;
  const int kc = plan.warps == 1 ? 8 : 16;  // one-warp CTAs stage fewer rows, so that more of them fit an SM
  const size_t smem = (size_t)kc * ((16 * nr + 4) * sizeof(double2) + n * sizeof(float2)) + 32 * nr * sizeof(double) +
                      (size_t)az_win * r_win * sizeof(int);
  auto go = [&](auto kernel) {
    if (int rc = allow_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    KernelTimer kt("gram fp64", s);
    kernel<<<gram_grid(kernel, threads, smem, n_pc), threads, smem, s>>>(
        rslc, nlines, width, n, idx, n_pc, mask, mask_stride, az_win, r_win, coh, dcount, doff, kc, plan);
    return check_launch("coherence gram");
  };
  if (shape.warps == 6) return go(gram64_kernel<7, 6>);
  if (shape.warps == 8)
    return plan.slots <= 4 ? go(gram64_kernel<4, 8>) : plan.slots <= 7 ? go(gram64_kernel<7, 8>) : go(gram64_kernel<9, 8>);
  return plan.slots <= 4 ? go(gram64_kernel<4, 4>) : plan.slots <= 7 ? go(gram64_kernel<7, 4>) : go(gram64_kernel<13, 4>);
}

}  // namespace

// Tensor-core Gram (coh_tc.cu); returns MR_ERR_UNSUPPORTED for shapes it does not take.
int gram_tc(const float2* rslc, int nlines, int width, int n, const int32_t* idx, int64_t n_pc,
            const uint8_t* mask, int mask_stride, int az_win, int r_win, float2* coh, int precision,
            cudaStream_t s);

}  // namespace mr

using namespace mr;

extern "C" int mr_emperical_co_pc(const mr_complex64* rslc, int nlines, int width, int nimages,
                                  const int32_t* idx, int64_t n_pc, const uint8_t* mask, int mask_stride,
                                  int az_win, int r_win, const int32_t* image_pairs, int n_pairs,
                                  mr_complex64* coh, int precision, mr_stream_t stream) {
  MR_REQUIRE(n_pc >= 0, "emperical_co_pc: negative n_pc");
  if (n_pc == 0) return MR_OK;
  MR_REQUIRE(rslc && idx && mask && coh, "emperical_co_pc: NULL pointer");
  MR_REQUIRE(nlines > 0 && width > 0 && nimages >= 2, "emperical_co_pc: bad stack shape");
  MR_REQUIRE(az_win > 0 && r_win > 0 && (az_win & 1) && (r_win & 1),
             "emperical_co_pc: window (%d, %d) must be odd", az_win, r_win);
  if (nimages > MR_MAX_NIMAGES) return fail(MR_ERR_UNSUPPORTED, "emperical_co_pc: nimages > %d", MR_MAX_NIMAGES);
  if ((int64_t)az_win * r_win > MR_MAX_WINDOW) return fail(MR_ERR_UNSUPPORTED, "emperical_co_pc: window too large");
  MR_REQUIRE(mask_stride == 0 || mask_stride == 1, "emperical_co_pc: mask_stride must be 0 or 1");
  MR_REQUIRE(n_pc >= 0, "emperical_co_pc: negative n_pc");
  if (n_pc == 0) return MR_OK;
  cudaStream_t s = as_stream(stream);
  const float2* z = reinterpret_cast<const float2*>(rslc);
  float2* out = reinterpret_cast<float2*>(coh);
  if (image_pairs) {
    MR_REQUIRE(n_pairs > 0, "emperical_co_pc: n_pairs must be > 0");
    int grid = (int)std::min<int64_t>((n_pc * n_pairs + 255) / 256, (int64_t)sm_count() * 32);
    gram_pairs_kernel<<<grid, 256, 0, s>>>(z, nlines, width, nimages, idx, n_pc, mask, mask_stride, az_win,
                                          r_win, image_pairs, n_pairs, out);
    return check_launch("coherence gram (pairs)");
  }
  switch (precision) {
    case MR_PREC_FP32:
      return launch_gram<float, kTriu>(z, nlines, width, nimages, idx, n_pc, mask, mask_stride, az_win, r_win,
                                       out, nullptr, s);
    case MR_PREC_FP64:
      return launch_gram64(z, nlines, width, nimages, idx, n_pc, mask, mask_stride, az_win, r_win, out, s);
    case MR_PREC_BF16:
    case MR_PREC_BF16X3:
      return gram_tc(z, nlines, width, nimages, idx, n_pc, mask, mask_stride, az_win, r_win, out, precision, s);
    default:
      return fail(MR_ERR_INVALID, "emperical_co_pc: unknown precision %d", precision);
  }
}

// Two single-date images to the interleaved 2-date layout of the Gram kernels.
__global__ void interleave2_kernel(const float2* __restrict__ a, const float2* __restrict__ b, int64_t npix,
                                   float4* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 x = a[i], y = b[i];
    out[i] = make_float4(x.x, x.y, y.x, y.y);
  }
}

extern "C" size_t mr_ad_intf_pc_workspace_bytes(int nlines, int width) {
  return std::max<size_t>(16, (size_t)nlines * width * 2 * sizeof(float2));
}

extern "C" int mr_ad_intf_pc(const mr_complex64* ref_rslc, const mr_complex64* sec_rslc, int nlines, int width,
                             const int32_t* idx, int64_t n_pc, const uint8_t* pc_is_shp, int az_win, int r_win,
                             mr_complex64* intf, int precision, void* workspace, size_t workspace_bytes,
                             mr_stream_t stream) {
  MR_REQUIRE(n_pc >= 0, "ad_intf_pc: negative n_pc");
  if (n_pc == 0) return MR_OK;
  MR_REQUIRE(ref_rslc && sec_rslc && idx && pc_is_shp && intf, "ad_intf_pc: NULL pointer");
  MR_REQUIRE(nlines > 0 && width > 0, "ad_intf_pc: bad image shape");
  MR_REQUIRE(precision == MR_PREC_FP32 || precision == MR_PREC_FP64, "ad_intf_pc: precision must be FP32 or FP64");
  const size_t need = mr_ad_intf_pc_workspace_bytes(nlines, width);
  if (!workspace || workspace_bytes < need)
    return fail(MR_ERR_WORKSPACE, "ad_intf_pc: workspace %zu < %zu bytes", workspace_bytes, need);
  MR_REQUIRE(((uintptr_t)workspace & 15) == 0, "ad_intf_pc: workspace not 16-byte aligned");
  const int64_t npix = (int64_t)nlines * width;
  const int grid = (int)std::min<int64_t>((npix + 255) / 256, (int64_t)sm_count() * 16);
  interleave2_kernel<<<grid, 256, 0, as_stream(stream)>>>(reinterpret_cast<const float2*>(ref_rslc),
                                                          reinterpret_cast<const float2*>(sec_rslc), npix,
                                                          static_cast<float4*>(workspace));
  if (int rc = check_launch("ad_intf_pc interleave")) return rc;
  // the one pair (0, 1) of the 2-date stack: the same kernel and arithmetic as pair (0, 1)
  // of emperical_co_pc on the full stack
  return mr_emperical_co_pc(static_cast<const mr_complex64*>(workspace), nlines, width, 2, idx, n_pc, pc_is_shp, 0,
                            az_win, r_win, nullptr, 1, intf, precision, stream);
}

namespace mr {
int gram_counted(const float2* rslc, int nlines, int width, int n, const int32_t* idx, int64_t n_max,
                 const int64_t* dcount, int64_t doff, const uint8_t* mask, int az_win, int r_win, float2* coh,
                 int precision, cudaStream_t s) {
  if (n_max <= 0) return MR_OK;
  if (precision == MR_PREC_FP32)
    return launch_gram<float, kTriu>(rslc, nlines, width, n, idx, n_max, mask, 1, az_win, r_win, coh, nullptr, s,
                                     dcount, doff);
  if (precision == MR_PREC_FP64)
    return launch_gram64(rslc, nlines, width, n, idx, n_max, mask, 1, az_win, r_win, coh, s, dcount, doff);
  return fail(MR_ERR_UNSUPPORTED, "device-counted coherence runs in FP32 or FP64");
}
}  // namespace mr

extern "C" int mr_emperical_co(const mr_complex64* rslc, int nlines, int width, int nimages,
                               const uint8_t* is_shp, int az_win, int r_win, mr_complex64* cov,
                               mr_complex64* coh, mr_stream_t stream) {
  MR_REQUIRE(rslc && is_shp && cov && coh, "emperical_co: NULL pointer");
  MR_REQUIRE(nlines > 0 && width > 0 && nimages >= 1, "emperical_co: bad stack shape");
  MR_REQUIRE(az_win > 0 && r_win > 0 && (az_win & 1) && (r_win & 1), "emperical_co: window must be odd");
  if (nimages > MR_MAX_NIMAGES) return fail(MR_ERR_UNSUPPORTED, "emperical_co: nimages > %d", MR_MAX_NIMAGES);
  if ((int64_t)az_win * r_win > MR_MAX_WINDOW) return fail(MR_ERR_UNSUPPORTED, "emperical_co: window too large");
  auto* c = reinterpret_cast<float2*>(coh);
  auto* v = reinterpret_cast<float2*>(cov);
  const auto launch = raster_pairs(nimages, c, v) ? launch_gram<float, kRasterPairs> : launch_gram<float, kRaster>;
  return launch(reinterpret_cast<const float2*>(rslc), nlines, width, nimages, nullptr, (int64_t)nlines * width, is_shp,
                1, az_win, r_win, c, v, as_stream(stream), nullptr, 0);
}
