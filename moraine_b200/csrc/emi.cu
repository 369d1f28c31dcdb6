// EMI phase linking on the GPU: host entry points.
//
// Reference behaviour followed (kanglcn/moraine):
//   moraine/pl.py:34-41, 56-64  Gamma = uncompress(coh); M = inv(|Gamma|) o Gamma;
//                               (lambda, v) = eigh(M)[0]  (algebraically smallest);
//                               ph = v conj(v[ref]) / |v conj(v[ref])|; quality = lambda
//   moraine/tnet.py:123-130     N from the number of pairs (all pairs m < j)
//   moraine/pl.py:112-120       temporal coherence of the result (fused epilogue)
//
// |Gamma| is frequently indefinite when a point has fewer SHPs than images, so M is then
// indefinite too and its smallest eigenvalue is large and negative. The algorithm is
// therefore valid for any Hermitian M:
//   1. inv(|Gamma|) by Gauss-Jordan elimination with partial pivoting;
//   2. M = inv(|Gamma|) o Gamma;
//   3. Householder reduction M = Q T Q^H, T Hermitian tridiagonal, then a diagonal unitary
//      scaling T = D R D^H with R real symmetric tridiagonal;
//   4. lambda_min(R) by Sturm-count multisection, a group of lanes per point;
//   5. its eigenvector y by two inverse iterations on R - lambda I (pivoted tridiagonal LU);
//   6. v = Q D y.
// The kernels are in emi_fast.cu: in the arithmetic asked for up to 128 images, in FP64 above.
#include <algorithm>
#include <atomic>

#include "common.cuh"

namespace mr {
namespace emi {

// emi_fast.cu
extern std::atomic<int64_t> g_sub_batch_cap;
size_t fast_workspace_bytes(int64_t n_pc, int n);
int fast_run(const float2* coh, int64_t n_pc, int n, int ref, int precision, float cond_max, float2* ph,
             float* quality, float* tcoh, uint8_t* route, void* workspace, cudaStream_t s,
             const int64_t* dcount = nullptr, int64_t doff = 0);

}  // namespace emi
}  // namespace mr

using namespace mr;
using namespace mr::emi;

extern "C" int mr_set_emi_sub_batch(int64_t max_points) {
  if (max_points < 0) return fail(MR_ERR_INVALID, "set_emi_sub_batch: max_points %lld < 0", (long long)max_points);
  mr::emi::g_sub_batch_cap.store(max_points);
  return MR_OK;
}

extern "C" size_t mr_emi_workspace_bytes(int64_t n_pc, int nimages) {
  if (n_pc <= 0 || nimages <= 0) return 16;
  return fast_workspace_bytes(n_pc, nimages);
}

namespace {

int emi_entry(const mr_complex64* coh, int64_t n_pc, int nimages, int ref, int precision, double cond_max,
              mr_complex64* ph, float* emi_quality, float* t_coh, uint8_t* route, void* workspace,
              size_t workspace_bytes, mr_stream_t stream) {
  MR_REQUIRE(nimages >= 2, "emi: nimages must be >= 2 (got %d)", nimages);
  if (nimages > MR_MAX_NIMAGES) return fail(MR_ERR_UNSUPPORTED, "emi: nimages %d > %d", nimages, MR_MAX_NIMAGES);
  MR_REQUIRE(ref >= 0 && ref < nimages, "emi: ref %d out of range [0, %d)", ref, nimages);
  MR_REQUIRE(n_pc >= 0, "emi: negative n_pc");
  MR_REQUIRE(precision == MR_PREC_FP32 || precision == MR_PREC_FP64 || precision == MR_PREC_MIXED ||
                 precision == MR_PREC_REFINE,
             "emi: precision must be FP32, FP64, MIXED or REFINE");
  MR_REQUIRE(cond_max > 0, "emi: cond_max (or the refinement tolerance) must be positive");
  if (n_pc == 0) return MR_OK;
  MR_REQUIRE(coh && ph && emi_quality, "emi: NULL pointer");
  const size_t need = mr_emi_workspace_bytes(n_pc, nimages);
  if (!workspace || workspace_bytes < need)
    return fail(MR_ERR_WORKSPACE, "emi: workspace %zu < %zu bytes", workspace_bytes, need);
  MR_REQUIRE(((uintptr_t)workspace & 15) == 0, "emi: workspace not 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  auto* c = reinterpret_cast<const float2*>(coh);
  auto* p = reinterpret_cast<float2*>(ph);
  return fast_run(c, n_pc, nimages, ref, nimages > 128 ? (int)MR_PREC_FP64 : precision,
                  (float)std::min(cond_max, 3.0e38), p, emi_quality, t_coh, route, workspace, s);
}

}  // namespace

extern "C" int mr_emi(const mr_complex64* coh, int64_t n_pc, int nimages, int ref, int precision,
                      mr_complex64* ph, float* emi_quality, float* t_coh, void* workspace, size_t workspace_bytes,
                      mr_stream_t stream) {
  return emi_entry(coh, n_pc, nimages, ref, precision,
                   precision == MR_PREC_REFINE ? MR_EMI_REFINE_TOL : MR_EMI_COND_MAX, ph, emi_quality, t_coh,
                   nullptr, workspace, workspace_bytes, stream);
}

extern "C" int mr_emi_refined(const mr_complex64* coh, int64_t n_pc, int nimages, int ref, double tol,
                              mr_complex64* ph, float* emi_quality, float* t_coh, uint8_t* route, void* workspace,
                              size_t workspace_bytes, mr_stream_t stream) {
  return emi_entry(coh, n_pc, nimages, ref, MR_PREC_REFINE, tol, ph, emi_quality, t_coh, route, workspace,
                   workspace_bytes, stream);
}

extern "C" int mr_emi_routed(const mr_complex64* coh, int64_t n_pc, int nimages, int ref, double cond_max,
                             mr_complex64* ph, float* emi_quality, float* t_coh, uint8_t* route, void* workspace,
                             size_t workspace_bytes, mr_stream_t stream) {
  return emi_entry(coh, n_pc, nimages, ref, MR_PREC_MIXED, cond_max, ph, emi_quality, t_coh, route, workspace,
                   workspace_bytes, stream);
}

namespace mr {
int emi_counted(const float2* coh, int64_t n_max, const int64_t* dcount, int64_t doff, int n, int precision,
                float2* ph, float* quality, float* tcoh, void* workspace, size_t workspace_bytes, cudaStream_t s) {
  if (n_max <= 0) return MR_OK;
  if (n < 2 || n > 128) return fail(MR_ERR_UNSUPPORTED, "emi: device-counted points need nimages <= 128");
  if (precision != MR_PREC_FP32 && precision != MR_PREC_FP64 && precision != MR_PREC_REFINE)
    return fail(MR_ERR_UNSUPPORTED, "emi: device-counted points run in FP32, FP64 or refined");
  if (!workspace || workspace_bytes < mr_emi_workspace_bytes(n_max, n))
    return fail(MR_ERR_WORKSPACE, "emi: workspace too small");
  const float tol = precision == MR_PREC_REFINE ? (float)MR_EMI_REFINE_TOL : 0.f;  // the refinement's bound
  return emi::fast_run(coh, n_max, n, 0, precision, tol, ph, quality, tcoh, nullptr, workspace, s, dcount, doff);
}
}  // namespace mr
