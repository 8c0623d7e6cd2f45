// Launchers of the parameter-gradient kernels: every compiled (type, kernel size) combination.
#include "wt2d_corr.cuh"
#include "wt2d_corr_host.h"

namespace wt {

namespace {

template <typename T, int K, bool BASE>
cudaError_t launch_level(const CorrStage& st, const CorrArgs& a, const void* x, const void* gy, cudaStream_t stream) {
  auto kern = wt2d_corr_kernel<T, K, BASE>;
  static bool done[kMaxDevices] = {false};
  const cudaError_t e = allow_full_smem(kern, done);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)(st.nsplit * st.p.ngroups), st.p.nthreads, (size_t)st.p.smem_bytes, stream>>>(st.p, a, static_cast<const T*>(x), static_cast<const T*>(gy));
  return cudaGetLastError();
}

template <int K>
cudaError_t launch_k(const CorrStage& st, const CorrArgs& a, int dtype, const void* x, const void* gy, cudaStream_t stream) {
  if (st.deep) {
    auto kern = wt2d_corr_deep_kernel<K>;
    static bool done[kMaxDevices] = {false};
    const cudaError_t e = allow_full_smem(kern, done);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(st.nsplit * st.p.ngroups), st.p.nthreads, (size_t)st.p.smem_bytes, stream>>>(st.p, a, static_cast<const float*>(x), static_cast<const float*>(gy));
    return cudaGetLastError();
  }
  if (!st.p.has_base) return launch_level<float, K, false>(st, a, x, gy, stream);
  switch (dtype) {
    case 0: return launch_level<float, K, true>(st, a, x, gy, stream);
    case 1: return launch_level<__nv_bfloat16, K, true>(st, a, x, gy, stream);
    default: return launch_level<__half, K, true>(st, a, x, gy, stream);
  }
}

}  // namespace

cudaError_t launch_corr(const CorrStage& st, const CorrArgs& a, int dtype, const void* x, const void* gy, cudaStream_t stream) {
  switch (st.p.K) {
    case 3: return launch_k<3>(st, a, dtype, x, gy, stream);
    case 5: return launch_k<5>(st, a, dtype, x, gy, stream);
    case 7: return launch_k<7>(st, a, dtype, x, gy, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace wt
