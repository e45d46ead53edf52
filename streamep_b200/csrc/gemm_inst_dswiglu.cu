// Instances of the grouped GEMM with the dSwiGLU epilogue (kernel Y_bwd), with and without a fused push.
#include "gemm_kernel.cuh"

namespace sep {

template <int BN, int CG>
static cudaError_t launch_width(const GemmParams& p, const LaunchMaps& m, const PushParams* push, int n, cudaStream_t s) {
  if (push != nullptr) return launch_instance<BN, false, true, kEpiDswiglu, true, CG>(p, m, *push, n, s);
  return launch_instance<BN, false, true, kEpiDswiglu, false, CG>(p, m, PushParams{}, n, s);
}

cudaError_t launch_dswiglu(const GemmParams& p, const LaunchMaps& m, const PushParams* push, int n, cudaStream_t s, bool& handled) {
  handled = p.mode == kVarlenM && !p.a_mn_major && p.b_mn_major;
  if (!handled) return cudaSuccess;
  if (p.block_n == 128) return launch_width<128, 1>(p, m, push, n, s);
  return p.pair_ctas ? launch_width<256, 2>(p, m, push, n, s) : launch_width<256, 1>(p, m, push, n, s);
}

}  // namespace sep
