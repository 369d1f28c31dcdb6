// PS-side statistics of the stack: amplitude, amplitude dispersion, calibrated amplitude.
//
// Replace moraine.calamp.rslc2amp (moraine/calamp.py:33-41), moraine.ps.amp_disp
// (moraine/ps.py:65-73) and moraine.calamp.calamp (moraine/calamp.py:63-71). All three are
// HBM-streaming passes over the same (nlines, width, nimages) complex64 stack the DS chain
// reads.
//
// |z| is the float32 rounding of the double square root of the exact double sum of squares,
// +inf when either part is infinite: bit-exact with np.abs on complex64 in the reference's
// Numba build (numpy's own hypotf can differ in the last bit). Means and standard
// deviations accumulate in double and the ratio rounds once to float32.
#include <algorithm>

#include "common.cuh"

namespace mr {
namespace {

__device__ __forceinline__ float abs_c64(float2 z) {
  if (isinf(z.x) || isinf(z.y)) return __int_as_float(0x7f800000);
  return (float)sqrt((double)z.x * z.x + (double)z.y * z.y);
}

__global__ void rslc2amp_kernel(const float2* __restrict__ z, int64_t n, float* __restrict__ amp) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    amp[i] = abs_c64(z[i]);
}

// The floats of abs_c64 without its FP64 root: x^2 + y^2 as an FP32 sum with its rounding errors, the
// approximate root corrected by its residual, together within 2^-41 of |z| (rsqrtf to 2 ulp). Where
// 2^-40 to either side would round to another float (2e-5 of the samples) the FP64 path decides; so it
// does for squares near the ends of the FP32 range, NaN and infinities.
__device__ __forceinline__ float abs_c64_fast(float2 z) {
  const float p = z.x * z.x, h = z.y * z.y;
  const float s = p + h;
  if (!(s > 1e-28f && s < 1e37f)) return abs_c64(z);
  const float big = fmaxf(p, h), small = fminf(p, h);
  const float lo = (small - (s - big)) + (fmaf(z.x, z.x, -p) + fmaf(z.y, z.y, -h));
  const float y = rsqrtf(s), r = s * y;
  const float e = fmaf(-r, r, s) + lo, off = s * 0x1p-39f, half = 0.5f * y;
  const float a = fmaf(e - off, half, r);
  return a == fmaf(e + off, half, r) ? a : abs_c64(z);
}

// kPx pixels per group of G lanes and step, lanes over a pixel's dates (contiguous, image axis
// innermost; NPL per lane). Sums of a - a_0 and (a - a_0)^2 in FP64, a_0 the pixel's first
// amplitude: the variance about the mean in one pass without cancellation on near-constant (PS)
// pixels, both sums of all kPx pixels reduced together. Bound by HBM and, below 32 dates a
// pixel, by the lane sums: 700 x 701 x 30 takes 70 us (with FP64 roots and two sums per
// pixel one after the other over 16 slots a lane: 383 us).
constexpr int kPx = 4;

template <int G, int NPL>
__global__ void __launch_bounds__(256) amp_disp_kernel(const float2* __restrict__ z, int64_t npix, int n,
                                                       float* __restrict__ out) {
  const int lane = threadIdx.x & (G - 1);
  const int64_t groups = (int64_t)gridDim.x * (256 / G);
  for (int64_t p0 = ((int64_t)blockIdx.x * (256 / G) + threadIdx.x / G) * kPx; p0 - kPx * (threadIdx.x % 32 / G) < npix;
       p0 += groups * kPx) {  // the test is the same for a whole warp
    float a[kPx][NPL], a0[kPx];
#pragma unroll
    for (int q = 0; q < kPx; ++q)
#pragma unroll
      for (int t = 0; t < NPL; ++t) {
        const int k = lane + G * t;
        a[q][t] = (k < n && p0 + q < npix) ? abs_c64_fast(z[(p0 + q) * n + k]) : 0.f;
      }
    double v[2 * kPx];
#pragma unroll
    for (int q = 0; q < kPx; ++q) {
      a0[q] = __shfl_sync(0xffffffffu, a[q][0], 0, G);
      v[2 * q] = v[2 * q + 1] = 0.0;
#pragma unroll
      for (int t = 0; t < NPL; ++t) {
        const double d = lane + G * t < n ? (double)a[q][t] - (double)a0[q] : 0.0;
        v[2 * q] += d;
        v[2 * q + 1] += d * d;
      }
    }
    // eight sums over G >= 8 lanes: each halving hands half of them to the other half of the lanes,
    // so that lane l ends with sum l / (G / 8) of the group
    int live = 2 * kPx;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      if (live > 1) {
        live >>= 1;
        const bool hi = lane & o;
#pragma unroll
        for (int e = 0; e < kPx; ++e)
          if (e < live) {
            const double keep = hi ? v[e + live] : v[e], give = hi ? v[e] : v[e + live];
            v[e] = keep + __shfl_xor_sync(0xffffffffu, give, o, G);
          }
      } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o, G);
      }
    }
    const int q = lane / (G / kPx);  // pixel of the sum that this lane holds
    const double sq = __shfl_xor_sync(0xffffffffu, v[0], G / 8, G);
    const float first = q == 0 ? a0[0] : q == 1 ? a0[1] : q == 2 ? a0[2] : a0[3];
    if (lane % (G / kPx) == 0 && p0 + q < npix) {
      const double m1 = v[0] / n, var = sq / n - m1 * m1;
      // one rounding: near-constant PS pixels keep their digits
      out[p0 + q] = (float)(sqrt(var < 0.0 ? 0.0 : var) / ((double)first + m1));
    }
  }
}

// Above 128 dates: one pixel per warp and step, eight dates per lane at a time. A pixel keeps a warp
// busy by itself there, and four at a time only leave fewer warps: 40 x 43 x 300 takes 19 us against 27
// with four (16 dates per lane unrolled), 350 x 353 x 512 227 against 479.
__global__ void __launch_bounds__(256) amp_disp_long_kernel(const float2* __restrict__ z, int64_t npix, int n,
                                                            float* __restrict__ out) {
  constexpr int kDates = 8;
  const int lane = threadIdx.x & 31;
  for (int64_t p = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); p < npix; p += (int64_t)gridDim.x * 8) {
    const float2* zp = z + p * n;
    float first = 0.f;
    double s1 = 0.0, s2 = 0.0;
#pragma unroll 1
    for (int k0 = 0; k0 < n; k0 += 32 * kDates) {
      float a[kDates];
#pragma unroll
      for (int t = 0; t < kDates; ++t) {
        const int k = k0 + lane + 32 * t;
        a[t] = k < n ? abs_c64_fast(zp[k]) : 0.f;
      }
      if (k0 == 0) first = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
      for (int t = 0; t < kDates; ++t) {
        const double d = k0 + lane + 32 * t < n ? (double)a[t] - (double)first : 0.0;
        s1 += d;
        s2 += d * d;
      }
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) {
      const double m1 = s1 / n, var = s2 / n - m1 * m1;
      out[p] = (float)(sqrt(var < 0.0 ? 0.0 : var) / ((double)first + m1));
    }
  }
}

template <int G, int NPL>
void launch_amp_disp(const float2* z, int64_t npix, int n, float* out, cudaStream_t s) {
  const int64_t blocks = (npix + (256 / G) * kPx - 1) / ((256 / G) * kPx);
  amp_disp_kernel<G, NPL><<<(unsigned)std::min<int64_t>(blocks, (int64_t)sm_count() * 64), 256, 0, s>>>(z, npix, n,
                                                                                                      out);
}

// calamp: per-block (sum, count) of the non-NaN amplitudes in double, then one block adds
// the partials in block order, then every sample is divided by the mean.
constexpr int kCalBlocks = 1024;

__global__ void calamp_partial_kernel(const float* __restrict__ amp, int64_t n, double2* __restrict__ part) {
  __shared__ double ss[8], sc[8];
  double s = 0, c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = amp[i];
    if (v == v) { s += v; c += 1; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { ss[w] = s; sc[w] = c; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ts = 0, tc = 0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { ts += ss[q]; tc += sc[q]; }
    part[blockIdx.x] = make_double2(ts, tc);
  }
}

__global__ void calamp_apply_kernel(const float* __restrict__ amp, int64_t n, const double2* __restrict__ part,
                                    int nparts, float* __restrict__ out) {
  __shared__ float mean;
  if (threadIdx.x == 0) {
    double s = 0, c = 0;
    for (int q = 0; q < nparts; ++q) { s += part[q].x; c += part[q].y; }
    mean = (float)(s / c);
  }
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = amp[i] / mean;
}

int grid_of(int64_t n, int per_block) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + per_block - 1) / per_block, (int64_t)sm_count() * 16));
}

}  // namespace
}  // namespace mr

using namespace mr;

extern "C" int mr_rslc2amp(const mr_complex64* rslc, int64_t n, float* amp, mr_stream_t stream) {
  MR_REQUIRE(n >= 0, "rslc2amp: negative size");
  if (n == 0) return MR_OK;
  MR_REQUIRE(rslc && amp, "rslc2amp: NULL pointer");
  rslc2amp_kernel<<<grid_of(n, 256), 256, 0, as_stream(stream)>>>(reinterpret_cast<const float2*>(rslc), n, amp);
  return check_launch("rslc2amp");
}

extern "C" int mr_amp_disp(const mr_complex64* rslc, int64_t npix, int nimages, float* amp_disp, mr_stream_t stream) {
  MR_REQUIRE(npix >= 0 && nimages >= 1, "amp_disp: bad stack shape");
  if (nimages > MR_MAX_NIMAGES) return fail(MR_ERR_UNSUPPORTED, "amp_disp: nimages %d > %d", nimages, MR_MAX_NIMAGES);
  if (npix == 0) return MR_OK;
  MR_REQUIRE(rslc && amp_disp, "amp_disp: NULL pointer");
  const auto* z = reinterpret_cast<const float2*>(rslc);
  cudaStream_t s = as_stream(stream);
  // as many lanes per pixel as it has dates, up to a warp
  if (nimages <= 8) launch_amp_disp<8, 1>(z, npix, nimages, amp_disp, s);
  else if (nimages <= 16) launch_amp_disp<16, 1>(z, npix, nimages, amp_disp, s);
  else if (nimages <= 32) launch_amp_disp<32, 1>(z, npix, nimages, amp_disp, s);
  else if (nimages <= 64) launch_amp_disp<32, 2>(z, npix, nimages, amp_disp, s);
  else if (nimages <= 128) launch_amp_disp<32, 4>(z, npix, nimages, amp_disp, s);
  else amp_disp_long_kernel<<<(unsigned)std::min<int64_t>((npix + 7) / 8, (int64_t)sm_count() * 64), 256, 0, s>>>(
      z, npix, nimages, amp_disp);
  return check_launch("amp_disp");
}

extern "C" size_t mr_calamp_workspace_bytes(void) { return kCalBlocks * sizeof(double2); }

extern "C" int mr_calamp(const float* amp, int64_t n, float* out, void* workspace, size_t workspace_bytes,
                         mr_stream_t stream) {
  MR_REQUIRE(n >= 0, "calamp: negative size");
  if (n == 0) return MR_OK;
  MR_REQUIRE(amp && out, "calamp: NULL pointer");
  if (!workspace || workspace_bytes < mr_calamp_workspace_bytes())
    return fail(MR_ERR_WORKSPACE, "calamp: workspace %zu < %zu bytes", workspace_bytes, mr_calamp_workspace_bytes());
  MR_REQUIRE(((uintptr_t)workspace & 15) == 0, "calamp: workspace not 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  auto* part = static_cast<double2*>(workspace);
  const int nb = (int)std::min<int64_t>(kCalBlocks, std::max<int64_t>(1, (n + 255) / 256));
  calamp_partial_kernel<<<nb, 256, 0, s>>>(amp, n, part);
  calamp_apply_kernel<<<grid_of(n, 256), 256, 0, s>>>(amp, n, part, nb, out);
  return check_launch("calamp", 2);
}
