// Instances of the grouped GEMM with the store epilogues over row tiles: preact recompute (bf16) and router logits (fp32).
#include "gemm_kernel.cuh"

namespace sep {

template <int BN, int CG>
static cudaError_t launch_width(const GemmParams& p, const LaunchMaps& m, int n, cudaStream_t s) {
  if (p.b_mn_major) return launch_instance<BN, false, true, kEpiStore, false, CG>(p, m, PushParams{}, n, s);
  return launch_instance<BN, false, false, kEpiStore, false, CG>(p, m, PushParams{}, n, s);
}

cudaError_t launch_store(const GemmParams& p, const LaunchMaps& m, const PushParams* push, int n, cudaStream_t s, bool& handled) {
  handled = p.mode == kVarlenM && !p.a_mn_major && push == nullptr && (p.epilogue == kEpiStore || (!p.b_mn_major && !p.pair_ctas));
  if (!handled) return cudaSuccess;
  if (p.epilogue == kEpiStoreF32) {
    return p.block_n == 128 ? launch_instance<128, false, false, kEpiStoreF32, false, 1>(p, m, PushParams{}, n, s)
                            : launch_instance<256, false, false, kEpiStoreF32, false, 1>(p, m, PushParams{}, n, s);
  }
  if (p.block_n == 128) return launch_width<128, 1>(p, m, n, s);
  return p.pair_ctas ? launch_width<256, 2>(p, m, n, s) : launch_width<256, 1>(p, m, n, s);
}

}  // namespace sep
