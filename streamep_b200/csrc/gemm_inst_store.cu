// Instances of the grouped GEMM with the plain store epilogue over row tiles (preact recompute).
#include "gemm_kernel.cuh"

namespace sep {

template <int BN, int CG>
static cudaError_t launch_width(const GemmParams& p, const LaunchMaps& m, int n, cudaStream_t s) {
  if (p.b_mn_major) return launch_instance<BN, false, true, kEpiStore, false, CG>(p, m, PushParams{}, n, s);
  return launch_instance<BN, false, false, kEpiStore, false, CG>(p, m, PushParams{}, n, s);
}

cudaError_t launch_store(const GemmParams& p, const LaunchMaps& m, const PushParams* push, int n, cudaStream_t s, bool& handled) {
  handled = p.mode == kVarlenM && !p.a_mn_major && push == nullptr;
  if (!handled) return cudaSuccess;
  if (p.block_n == 128) return launch_width<128, 1>(p, m, n, s);
  return p.pair_ctas ? launch_width<256, 2>(p, m, n, s) : launch_width<256, 1>(p, m, n, s);
}

}  // namespace sep
