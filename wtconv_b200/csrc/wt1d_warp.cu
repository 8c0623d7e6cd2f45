// Launchers of the register-resident 1-D kernels: every compiled (dtype, K, L) combination.
#include "wt1d_warp.cuh"

namespace wt {

namespace {

template <typename T, int K, int L, int SPT>
cudaError_t launch_spt(Warp1dArgs a, cudaStream_t stream) {
  a.nseg = cdiv(a.N, warp1d_segment(K, L, SPT));
  a.nwarps = (long long)a.B * a.C * a.nseg;
  if (a.nwarps >= (1LL << 31)) return cudaErrorNotSupported;     // 32-bit warp index in the kernel
  const long long want = (a.nwarps + kWarp1dWarps - 1) / kWarp1dWarps;
  const long long resident = 148 * (SPT == 32 ? 2 : (K <= 5 && L <= 3 ? 4 : 3));   // persistent: see the kernel's launch bounds
  auto kern = wt1d_warp_kernel<T, K, L, SPT>;
  static bool done[kMaxDevices] = {false};
  const cudaError_t e = allow_full_smem(kern, done);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)(want < resident ? want : resident), kWarp1dWarps * 32, warp1d_smem_bytes<T, K, L, SPT>(), stream>>>(a);
  return cudaGetLastError();
}

// Samples per thread: 32 halve the shuffles, the neighbour-only lanes and the per-item work per sample, but a
// warp then spans about 960 samples; with fewer than eight such warps per SM (or rows shorter than half
// a warp) 16 samples keep more of the chip busy.
template <typename T, int K, int L>
cudaError_t launch_one(const Warp1dArgs& a, cudaStream_t stream) {
  if constexpr (L == 5) return launch_spt<T, K, L, 32>(a, stream);
  else {
    const long long warps = (long long)a.B * a.C * cdiv(a.N, warp1d_segment(K, L, 32));
    if (a.N >= 480 && warps >= 148 * 8) return launch_spt<T, K, L, 32>(a, stream);
    return launch_spt<T, K, L, 16>(a, stream);
  }
}

template <typename T, int K, int L>
cudaError_t launch_one(Wgrad1dArgs a, cudaStream_t stream) {
  constexpr int SPT = L == 5 ? 32 : 16;                  // the sums take (1 + 2L) * K registers: short runs where they suffice
  constexpr size_t smem = warp1d_wgrad_smem<T, SPT>();
  a.nseg = cdiv(a.N, warp1d_segment(K, L, SPT));
  a.items = (long long)a.B * a.nseg;
  // two waves of the resident CTAs (two per SM), shared by the channels; every CTA keeps at least
  // one item per warp
  const long long most = (a.items + kWarp1dWarps - 1) / kWarp1dWarps;
  long long split = imax(1, 592 / a.C);
  if (split > most) split = most;
  a.nsplit = (int)split;
  auto kern = wt1d_wgrad_kernel<T, K, L, SPT>;
  static bool done[kMaxDevices] = {false};
  const cudaError_t e = allow_full_smem(kern, done);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)(a.C * split), kWarp1dWarps * 32, smem, stream>>>(a);
  return cudaGetLastError();
}

template <typename T, int K, typename Args>
cudaError_t launch_levels(const Args& a, int L, cudaStream_t st) {
  switch (L) {
    case 0: return launch_one<T, K, 0>(a, st);
    case 1: return launch_one<T, K, 1>(a, st);
    case 2: return launch_one<T, K, 2>(a, st);
    case 3: return launch_one<T, K, 3>(a, st);
    case 4: return launch_one<T, K, 4>(a, st);
    case 5: return launch_one<T, K, 5>(a, st);
    default: return cudaErrorNotSupported;
  }
}

template <typename T, typename Args>
cudaError_t launch_sizes(const Args& a, int K, int L, cudaStream_t st) {
  switch (K) {
    case 1: return launch_levels<T, 1>(a, L, st);
    case 3: return launch_levels<T, 3>(a, L, st);
    case 5: return launch_levels<T, 5>(a, L, st);
    case 7: return launch_levels<T, 7>(a, L, st);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace

cudaError_t launch_wt1d_warp(const Warp1dArgs& a, int K, int L, int dtype, cudaStream_t stream) {
  switch (dtype) {
    case 0: return launch_sizes<float>(a, K, L, stream);
    case 1: return launch_sizes<__nv_bfloat16>(a, K, L, stream);
    default: return launch_sizes<__half>(a, K, L, stream);
  }
}

cudaError_t launch_wt1d_wgrad(const Wgrad1dArgs& a, int K, int L, int dtype, cudaStream_t stream) {
  switch (dtype) {
    case 0: return launch_sizes<float>(a, K, L, stream);
    case 1: return launch_sizes<__nv_bfloat16>(a, K, L, stream);
    default: return launch_sizes<__half>(a, K, L, stream);
  }
}

}  // namespace wt
