// Instances of the grouped GEMM over the rows of each expert (weight gradients dW1 and dW2).
#include "gemm_kernel.cuh"

namespace sep {

cudaError_t launch_store_varlen_k(const GemmParams& p, const LaunchMaps& m, const PushParams* push, int n, cudaStream_t s, bool& handled) {
  handled = p.mode == kVarlenK && p.a_mn_major && p.b_mn_major && push == nullptr;
  if (!handled) return cudaSuccess;
  if (p.block_n == 128) return launch_instance<128, true, true, kEpiStore, false, 1>(p, m, PushParams{}, n, s);
  return p.pair_ctas ? launch_instance<256, true, true, kEpiStore, false, 2>(p, m, PushParams{}, n, s)
                     : launch_instance<256, true, true, kEpiStore, false, 1>(p, m, PushParams{}, n, s);
}

}  // namespace sep
