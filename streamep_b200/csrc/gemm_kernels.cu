// Launch of the grouped GEMM (the template is in gemm_kernel.cuh, its instances in gemm_inst_*.cu) and the
// allocation-free entry point of kernel Y.
#include <cstdio>
#include <mutex>

#include "gemm_kernel.cuh"
#include "no_alloc.h"

namespace sep {

bool launch_grouped_gemm(const GemmParams& p, const void* tmap_a, const void* tmap_b, const void* tmap_o0,
                         const void* tmap_o1, const PushParams* fused_push, int num_ctas, cudaStream_t stream,
                         cudaError_t* setup_error, const void* maps2) {
  LaunchMaps m;
  m.a = *static_cast<const CUtensorMap*>(tmap_a);
  m.b = *static_cast<const CUtensorMap*>(tmap_b);
  m.o0 = tmap_o0 != nullptr ? *static_cast<const CUtensorMap*>(tmap_o0) : m.a;
  m.o1 = tmap_o1 != nullptr ? *static_cast<const CUtensorMap*>(tmap_o1) : m.a;
  if (maps2 != nullptr) m.second = *static_cast<const SecondMaps*>(maps2);
  else { m.second.a = m.a; m.second.b = m.b; m.second.o = m.o0; }
  bool handled = false;
  cudaError_t err = cudaSuccess;
  if (p.mode == kVarlenK) err = launch_store_varlen_k(p, m, fused_push, num_ctas, stream, handled);
  else if (p.epilogue == kEpiSwiglu) err = launch_swiglu(p, m, fused_push, num_ctas, stream, handled);
  else if (p.epilogue == kEpiDswiglu) err = launch_dswiglu(p, m, fused_push, num_ctas, stream, handled);
  else if (p.epilogue == kEpiScatter) err = launch_scatter(p, m, fused_push, num_ctas, stream, handled);
  else err = launch_store(p, m, fused_push, num_ctas, stream, handled);
  if (setup_error != nullptr) *setup_error = err;
  return handled;
}

}  // namespace sep

// =============================================================================================
// Allocation-free entry point (declared and documented in no_alloc.h).
// =============================================================================================
namespace {

// Scratch of the no-alloc entry point: per-M-tile "N stripes finished" counters, followed by the status block the
// kernel's bounded waits report into.  In host code this name is only a handle for cudaGetSymbolAddress; the
// device address is resolved once per device.
constexpr int kNoAllocStatusInts = 64;    // 256 bytes: keeps the status block on its own 256-byte line
static __device__ __align__(256) int g_noalloc_scratch[kNoAllocMaxTiles + kNoAllocStatusInts];
static_assert(sizeof(sep::StatusBlock) <= kNoAllocStatusInts * sizeof(int), "status block must fit its slot");

int* g_noalloc_scratch_ptr[sep::kMaxDevices] = {};
std::mutex g_noalloc_setup_mutex;
thread_local char g_noalloc_error[256] = "";

int noalloc_fail(int code, const char* what, cudaError_t e = cudaSuccess) {
  if (e != cudaSuccess) snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s: %s", what, cudaGetErrorString(e));
  else snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", what);
  return code;
}

using NoAllocEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                     const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

bool noalloc_tmap(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t b0, uint32_t b1) {
  static std::atomic<NoAllocEncodeFn> encode_fn{nullptr};
  NoAllocEncodeFn encode = encode_fn.load(std::memory_order_acquire);
  if (encode == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || fn == nullptr)
      return false;
    encode = reinterpret_cast<NoAllocEncodeFn>(fn);
    encode_fn.store(encode, std::memory_order_release);
  }
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {d0 * 2, d0 * d1 * 2};
  cuuint32_t box[3] = {b0, b1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Device address of the scratch array on the current device (resolved under a lock on first use).
int* noalloc_scratch(int dev, cudaError_t* e) {
  std::lock_guard<std::mutex> g(g_noalloc_setup_mutex);
  if (g_noalloc_scratch_ptr[dev] == nullptr) {
    int* ptr = nullptr;
    *e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_scratch);
    if (*e != cudaSuccess || ptr == nullptr) return nullptr;
    g_noalloc_scratch_ptr[dev] = ptr;
  }
  return g_noalloc_scratch_ptr[dev];
}

}  // namespace

extern "C" const char* streamep_noalloc_last_error(void) { return g_noalloc_error; }

extern "C" int streamep_noalloc_device_status(int* code, int* where) {
  using namespace sep;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaGetDevice", e);
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(-2, "device ordinal out of range");
  int* scratch = noalloc_scratch(dev, &e);
  if (scratch == nullptr) return noalloc_fail(-3, "cudaGetSymbolAddress(scratch)", e);
  StatusBlock h;
  e = cudaMemcpy(&h, scratch + kNoAllocMaxTiles, sizeof(h), cudaMemcpyDeviceToHost);   // waits for earlier work
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaMemcpy(status)", e);
  if (code != nullptr) *code = h.code;
  if (where != nullptr) *where = h.where;
  return 0;
}

extern "C" int streamep_gemm_y_scatter_noalloc(const void* postact, const void* w2, const int* tile_id_to_expert,
                                               const float* pool_topk_weight, const int* pool_recv_token, void* o,
                                               int* k_local_remaining, long long* y_done_per_token, int total_tiles,
                                               int hidden, int ffn, int num_local_experts, long long seq, void* stream_v) {
  using namespace sep;
  g_noalloc_error[0] = 0;
  if (total_tiles < 0) return noalloc_fail(-2, "total_tiles must not be negative");
  if (total_tiles > kNoAllocMaxTiles)
    return noalloc_fail(-1, "total_tiles exceeds kNoAllocMaxTiles (32768): split the call or use the regular entry point");
  if (total_tiles == 0) return 0;
  if (!postact || !w2 || !tile_id_to_expert || !pool_topk_weight || !pool_recv_token || !o || !k_local_remaining || !y_done_per_token)
    return noalloc_fail(-2, "null pointer argument");
  if (hidden <= 0 || ffn <= 0 || hidden % 8 != 0 || ffn % 8 != 0 || num_local_experts <= 0)
    return noalloc_fail(-2, "hidden and ffn must be positive multiples of 8, num_local_experts positive");
  if (reinterpret_cast<uintptr_t>(postact) % 16 != 0 || reinterpret_cast<uintptr_t>(w2) % 16 != 0 || reinterpret_cast<uintptr_t>(o) % 16 != 0)
    return noalloc_fail(-2, "postact, w2 and o must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaGetDevice", e);
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(-2, "device ordinal out of range");
  // One-time set-up for this device (with it current): the device address behind the symbol.
  int* scratch = noalloc_scratch(dev, &e);
  if (scratch == nullptr) return noalloc_fail(-3, "cudaGetSymbolAddress(scratch)", e);

  const int block_n = (hidden % 256 == 0) ? 256 : ((hidden % 128 == 0) ? 128 : (hidden > 128 ? 256 : 128));
  const long long rows = static_cast<long long>(total_tiles) * BM;
  LaunchMaps maps;
  if (!noalloc_tmap(&maps.a, postact, ffn, rows, 1, 64, BM) || !noalloc_tmap(&maps.b, w2, ffn, hidden, num_local_experts, 64, block_n))
    return noalloc_fail(-3, "cuTensorMapEncodeTiled failed");
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaDeviceGetAttribute", e);

  // Nothing was enqueued so far.  The array keeps the previous call's counts and status: clear the part this call
  // uses (stream-ordered, so it cannot overtake an earlier call on the same stream).
  e = cudaMemsetAsync(scratch, 0, sizeof(int) * static_cast<size_t>(total_tiles), stream);
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaMemsetAsync(scratch)", e);
  e = cudaMemsetAsync(scratch + kNoAllocMaxTiles, 0, sizeof(int) * kNoAllocStatusInts, stream);
  if (e != cudaSuccess) return noalloc_fail(-3, "cudaMemsetAsync(status)", e);

  GemmParams p{};
  p.mode = kVarlenM; p.epilogue = kEpiScatter; p.block_n = block_n;
  p.N = hidden; p.K = ffn; p.num_experts = num_local_experts; p.total_rows = static_cast<int>(rows);
  p.num_m_tiles = total_tiles; p.num_n_tiles = (hidden + block_n - 1) / block_n;
  p.tile_id_to_expert = tile_id_to_expert;
  p.row_weight = pool_topk_weight; p.row_token = pool_recv_token;
  p.scatter_local = o;
  p.tile_stripes_done = scratch; p.k_remaining = k_local_remaining; p.done_per_token = y_done_per_token; p.seq = seq;
  p.num_ranks = 1; p.rank = 0;
  p.status = reinterpret_cast<StatusBlock*>(scratch + kNoAllocMaxTiles);   // read back by streamep_noalloc_device_status
  p.wait_budget_ns = 2000000000ull;
  const long long total = static_cast<long long>(p.num_m_tiles) * p.num_n_tiles;
  const int ctas = static_cast<int>(total < sms ? total : sms);
  maps.o0 = maps.o1 = maps.second.o = maps.second.a = maps.a;
  maps.second.b = maps.b;
  bool handled = false;
  e = launch_scatter(p, maps, nullptr, ctas, stream, handled);
  if (e != cudaSuccess) return noalloc_fail(-3, "kernel set-up (shared-memory attribute)", e);
  e = cudaGetLastError();
  if (e != cudaSuccess) return noalloc_fail(-3, "kernel launch", e);
  return 0;
}
