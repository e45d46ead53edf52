// Dispatch of one rank on its own: every (token, k) pair stays on this GPU, so nothing is exchanged and the layer needs
// only a stable counting sort of its pairs by expert and one copy of each token row per pair.
//
// The pool layout is the one of the general dispatch (expert-major, every expert padded to whole 128-row tiles, (token, k)
// order inside an expert).  The general path costs a count exchange, a single-block layout synthesis, a materialise
// launch and row pushes by extra warps of the GEMM kernels (8192 tokens, top-6, hidden 2048: 41 us of metadata, and the
// pushes lengthened GEMM-A by 67 us and GEMM-Y_bwd by 78 us).  Here:
//
//   local_count_kernel   pairs per (block of tokens, expert)
//   local_place_kernel   offsets, slots and per-slot arrays; then the block copies its tokens' rows into the pool, each
//                        row read once and stored once per pair; idle warps zero the layer's output meanwhile
//   local_rows_kernel    backward: gradient rows into their pool along the stored slots
//
// All three are bound by the pool's writes to HBM (2 x pairs x hidden bytes).  Small calls (<= kFusedPairs pairs) skip
// the count launch: every block counts all pairs itself, which costs a few microseconds less than a launch.
#include "comm_common.cuh"

namespace sep {

constexpr int kLocalThreads = 512;
constexpr int kLocalWarps = kLocalThreads / 32;
constexpr int kFusedPairs = 8192;         // up to 16 pairs per thread to count
constexpr int kMaxBlockPairs = 4096;      // pairs one block ranks (slots kept in shared memory)
constexpr int kCountCells = 19 << 10;     // blocks x experts whose counts every block reads: ~76 KB from L2

static int local_sms() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    cached[dev] = n;
  }
  return cached[dev];
}

LocalGrid local_grid(int num_tokens, int num_topk, int num_experts) {
  LocalGrid g;
  const long long pairs = static_cast<long long>(num_tokens) * num_topk;
  g.fused_count = pairs <= kFusedPairs;
  // Two blocks per SM copy rows at full rate.  Fewer when the count matrix would get large, more when a block would have
  // more pairs than it can rank.
  long long blocks = 2 * local_sms();
  if (!g.fused_count && blocks * num_experts > kCountCells) blocks = kCountCells / num_experts;
  if (blocks > num_tokens) blocks = num_tokens;
  if (blocks < 1) blocks = 1;
  const long long need = (pairs + kMaxBlockPairs - 64 - 1) / (kMaxBlockPairs - 64);
  if (blocks < need) blocks = need;
  g.tokens_per_block = static_cast<int>((num_tokens + blocks - 1) / blocks);
  if (g.tokens_per_block < 1) g.tokens_per_block = 1;
  g.blocks = (num_tokens + g.tokens_per_block - 1) / g.tokens_per_block;
  if (g.blocks < 1) g.blocks = 1;
  g.count_ints = g.fused_count ? 0 : static_cast<size_t>(g.blocks) * num_experts;
  return g;
}

__global__ void __launch_bounds__(kLocalThreads) local_count_kernel(const long long* topk_idx, int num_tokens, int num_topk, int num_experts,
                                                                    int tokens_per_block, int* counts) {
  extern __shared__ int s_hist[];
  grid_release();
  for (int e = threadIdx.x; e < num_experts; e += kLocalThreads) s_hist[e] = 0;
  __syncthreads();
  const int t0 = blockIdx.x * tokens_per_block, t1 = min(t0 + tokens_per_block, num_tokens);
  const long long* idx = topk_idx + static_cast<size_t>(t0) * num_topk;
  for (int i = threadIdx.x; i < (t1 - t0) * num_topk; i += kLocalThreads) {
    const long long e = idx[i];
    if (e >= 0 && e < num_experts) atomicAdd(&s_hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < num_experts; e += kLocalThreads) counts[static_cast<size_t>(e) * gridDim.x + blockIdx.x] = s_hist[e];
}

__device__ __forceinline__ void zero_slice(void* ptr, size_t bytes, size_t part, size_t parts) {
  const size_t vecs = bytes / 16;
  for (size_t i = part; i < vecs; i += parts) reinterpret_cast<uint4*>(ptr)[i] = make_uint4(0, 0, 0, 0);
  if (part < (bytes & 15) / 4) reinterpret_cast<int*>(ptr)[vecs * 4 + part] = 0;
}

// The pairs are sorted in 6-19 us during which HBM has little to do.  A call bound by reading the weights (fewer pairs than
// kPrefetchRowsPerPair weight rows each) uses them to bring the first columns of every weight row of the experts it hits
// into the L2, where the GEMM behind this kernel starts reading; as much as HBM can deliver meanwhile, well below the L2's
// 126 MB.  Together with the padding rows that inference does not zero: 96 tokens on 32 experts, hidden 7168, 499 -> 486 us.
constexpr size_t kPrefetchBytes = 40u << 20;
constexpr int kPrefetchRowsPerPair = 4;

__device__ __forceinline__ void prefetch_weights(const LocalPlaceParams& p, const int* s_total, int tid) {
  int hit = 0;
  for (int e = 0; e < p.num_experts; ++e) hit += s_total[e] > 0;
  if (hit == 0) return;
  const size_t row_bytes = static_cast<size_t>(p.hidden) * 2;
  const size_t share = kPrefetchBytes / (static_cast<size_t>(hit) * p.prefetch_rows) / 128 * 128;
  const uint32_t bytes = static_cast<uint32_t>(share < row_bytes ? share : row_bytes);
  if (bytes == 0) return;
  for (int i = blockIdx.x * kLocalThreads + tid; i < p.num_experts * p.prefetch_rows; i += gridDim.x * kLocalThreads)
    if (s_total[i / p.prefetch_rows] > 0) bulk_prefetch_l2(static_cast<const char*>(p.prefetch) + static_cast<size_t>(i) * row_bytes, bytes);
}

// Zeroes the pool rows between an expert's length and the next multiple of 64 (the weight-gradient GEMM multiplies whole
// 64-row blocks).
__device__ __forceinline__ void zero_padding_rows(char* pool, int first_slot, int len, int vecs, int tid, int threads) {
  const int rows = (len + 63) / 64 * 64 - len;
  char* base = pool + static_cast<size_t>(first_slot + len) * vecs * 16;
  for (int i = tid; i < rows * vecs; i += threads) reinterpret_cast<uint4*>(base)[i] = make_uint4(0, 0, 0, 0);
}

template <bool FUSED_COUNT>
__global__ void __launch_bounds__(kLocalThreads, 2) local_place_kernel(const LocalPlaceParams p) {
  extern __shared__ int s_dyn[];
  int* s_total = s_dyn;                       // [E] pairs of each expert
  int* s_run = s_dyn + p.num_experts;         // [E] next slot of each expert for this block's pairs
  int* s_tiles = s_dyn + 2 * p.num_experts;   // [E + 1] first tile of each expert
  int* s_slot = s_tiles + p.num_experts + 1;  // [pairs of this block]
  __shared__ int s_ok, s_pairs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int E = p.num_experts, K = p.num_topk;
  const bool has_tokens = static_cast<int>(blockIdx.x) < p.token_blocks;
  const int t0 = min(static_cast<int>(blockIdx.x) * p.tokens_per_block, p.num_tokens), t1 = min(t0 + p.tokens_per_block, p.num_tokens);
  const int n = has_tokens ? (t1 - t0) * K : 0;
  const long long* idx = p.topk_idx + static_cast<size_t>(t0) * K;
  if (!FUSED_COUNT) grid_wait();
  grid_release();

  // 1. pairs of every expert: in all, and in the blocks before this one
  if (FUSED_COUNT) {
    for (int e = tid; e < E; e += kLocalThreads) { s_total[e] = 0; s_run[e] = 0; }
    __syncthreads();
    const int all = p.num_tokens * K, before = t0 * K;
    for (int i = tid; i < all; i += kLocalThreads) {
      const long long e = p.topk_idx[i];
      if (e >= 0 && e < E) {
        atomicAdd(&s_total[e], 1);
        if (i < before) atomicAdd(&s_run[e], 1);
      }
    }
  } else {
    for (int e = warp; e < E; e += kLocalWarps) {
      int total = 0, before = 0;
      const int* c = p.counts + static_cast<size_t>(e) * p.token_blocks;
      for (int b = lane; b < p.token_blocks; b += 32) {
        const int v = c[b];
        total += v;
        if (b < static_cast<int>(blockIdx.x)) before += v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        total += __shfl_xor_sync(0xffffffffu, total, o);
        before += __shfl_xor_sync(0xffffffffu, before, o);
      }
      if (lane == 0) { s_total[e] = total; s_run[e] = before; }
    }
  }
  __syncthreads();
  if (FUSED_COUNT && p.prefetch != nullptr) prefetch_weights(p, s_total, tid);
  // 2. first tile of every expert
  if (warp == 0) {
    int carry = 0, pairs = 0;
    for (int base = 0; base < E; base += 32) {
      const int e = base + lane;
      const int tiles = e < E ? (s_total[e] + kTileM - 1) / kTileM : 0;
      int x = tiles, y = (tiles + 1) / 2;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) { x += a; y += b; }
      }
      if (e < E) s_tiles[e] = carry + x - tiles;
      carry += __shfl_sync(0xffffffffu, x, 31);
      pairs += __shfl_sync(0xffffffffu, y, 31);
    }
    if (lane == 0) { s_tiles[E] = carry; s_pairs = pairs; s_ok = carry <= p.tiles_cap; }
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  if (!ok) {     // (capacity mode) the layout does not fit: this dispatch runs as an empty one and the host hears about it
    if (blockIdx.x == 0 && tid == 0) {
      report_note(p.status, kStatusOverflow, kKernelMetadata, 1, 0, p.region_id, p.tiles_cap, s_tiles[E]);
      if (p.host_overflow != nullptr) {
        p.host_overflow->needed_tiles = s_tiles[E];
        p.host_overflow->needed_recv = p.num_tokens;
        p.host_overflow->epoch = p.epoch;
        __threadfence_system();
        p.host_overflow->count = p.host_overflow->count + 1;
      }
    }
    __syncthreads();
    for (int e = tid; e <= E; e += kLocalThreads) { if (e < E) s_total[e] = 0; s_tiles[e] = 0; }
    if (tid == 0) s_pairs = 0;
    __syncthreads();
  }
  // 3. slots of this block's pairs, in (token, k) order inside an expert; the other warps zero the output meanwhile
  if (warp == 0) {
    if (!ok) { for (int i = lane; i < n; i += 32) s_slot[i] = -1; }
    else {
      for (int e = lane; e < E; e += 32) s_run[e] += s_tiles[e] * kTileM;
      __syncwarp();
      for (int base0 = 0; base0 < n; base0 += 256) {       // eight steps' expert ids in flight
        int ev[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = base0 + j * 32 + lane;
          const long long e = i < n ? idx[i] : -1;
          ev[j] = (e >= 0 && e < E) ? static_cast<int>(e) : -1;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = base0 + j * 32 + lane;
          if (base0 + j * 32 >= n) break;
          const unsigned peers = __match_any_sync(0xffffffffu, ev[j] >= 0 ? ev[j] : -1 - lane);
          int slot = -1;
          if (ev[j] >= 0) slot = s_run[ev[j]] + __popc(peers & ((1u << lane) - 1u));
          __syncwarp();
          if (ev[j] >= 0 && (__ffs(peers) - 1) == lane) s_run[ev[j]] += __popc(peers);
          __syncwarp();
          if (i < n) s_slot[i] = slot;
        }
      }
    }
  } else {
    const size_t part = static_cast<size_t>(blockIdx.x) * (kLocalThreads - 32) + tid - 32;
    zero_slice(p.zero, p.zero_bytes, part, static_cast<size_t>(gridDim.x) * (kLocalThreads - 32));
  }
  __syncthreads();
  // 4. what the GEMM kernels read: per-slot arrays, padding slots, tiles, sizes
  const int vecs = p.hidden / 8;
  for (int i = tid; i < n; i += kLocalThreads) {
    const int slot = s_slot[i], pair = t0 * K + i;
    p.pair_slot[pair] = slot;
    if (slot >= 0) {
      p.row_token[slot] = pair / K;
      p.row_pair[slot] = pair;
      p.row_weight[slot] = p.topk_weights[pair];
    }
  }
  for (int e = blockIdx.x; e < E; e += gridDim.x) {
    const int first = s_tiles[e] * kTileM, len = s_total[e], end = s_tiles[e + 1] * kTileM;
    for (int s = first + len + tid; s < end; s += kLocalThreads) { p.row_token[s] = -1; p.row_pair[s] = -1; p.row_weight[s] = 0.f; }
    if (p.zero_padding) zero_padding_rows(static_cast<char*>(p.pool), first, len, vecs, tid, kLocalThreads);
  }
  const int live = s_tiles[E];
  for (int t = blockIdx.x * kLocalThreads + tid; t < live; t += gridDim.x * kLocalThreads) {
    int lo = 0, hi = E - 1;                      // the last expert whose first tile is not after t (and that has tiles)
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (s_tiles[mid] <= t) lo = mid; else hi = mid - 1;
    }
    p.tile_id_to_expert[t] = lo;
    const int j = t - s_tiles[lo];
    if ((j & 1) == 0) {
      int before = 0;
      for (int e = 0; e < lo; ++e) before += (s_tiles[e + 1] - s_tiles[e] + 1) / 2;
      p.pair_tiles[before + j / 2] = t * 2 + (t + 1 < s_tiles[lo + 1] ? 1 : 0);
    }
  }
  if (blockIdx.x == 0) {
    for (int e = tid; e < E; e += kLocalThreads) { p.expert_frequency[e] = s_total[e]; p.expert_pool_block_offset[e] = s_tiles[e]; }
    if (tid == 0) {
      p.expert_pool_block_offset[E] = live;
      p.sizes[0] = live; p.sizes[1] = p.num_tokens; p.sizes[2] = ok ? 0 : 1; p.sizes[3] = s_pairs;
      p.sizes[4] = 0; p.sizes[5] = 0;
    }
  }
  // 5. the rows: a warp takes a piece of one token's row, reads it once and stores it once per pair
  const char* x = static_cast<const char*>(p.x);
  const size_t row_bytes = static_cast<size_t>(p.hidden) * 2;
  const int pieces = (vecs + 255) / 256;
  for (int item = warp; item < (t1 - t0) * pieces && has_tokens; item += kLocalWarps) {
    const int t = item / pieces, v0 = (item - t * pieces) * 256;
    const int slot = lane < K ? s_slot[t * K + lane] : -1;
    copy_row_piece<8>(x + (t0 + t) * row_bytes, static_cast<char*>(p.pool),
                      p.x_saved != nullptr ? static_cast<char*>(p.x_saved) + (t0 + t) * row_bytes : nullptr, v0, vecs, K, slot, lane);
  }
}

cudaError_t launch_local_place(const LocalPlaceParams& q, const LocalGrid& g, cudaStream_t stream) {
  LocalPlaceParams p = q;
  p.tokens_per_block = g.tokens_per_block;
  p.token_blocks = g.blocks;
  if (!g.fused_count)
    local_count_kernel<<<g.blocks, kLocalThreads, sizeof(int) * p.num_experts, stream>>>(p.topk_idx, p.num_tokens, p.num_topk, p.num_experts,
                                                                                      g.tokens_per_block, p.counts);
  const size_t smem = sizeof(int) * (3 * static_cast<size_t>(p.num_experts) + 1 + static_cast<size_t>(g.tokens_per_block) * p.num_topk);
  if (g.fused_count) {
    if (static_cast<long long>(p.num_tokens) * p.num_topk * kPrefetchRowsPerPair > static_cast<long long>(p.num_experts) * p.prefetch_rows)
      p.prefetch = nullptr;
    const int blocks = p.prefetch != nullptr && g.blocks < local_sms() ? local_sms() : g.blocks;    // (blocks without tokens help)
    local_place_kernel<true><<<blocks, kLocalThreads, smem, stream>>>(p);
  }
  else {
    cudaLaunchAttribute early;          // sets up while the counts are being made
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(g.blocks)); cfg.blockDim = dim3(kLocalThreads);
    cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = &early; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, local_place_kernel<false>, p);
  }
  return cudaGetLastError();
}

// Rows of up to two matrices into their pools along the stored slots, the pools' padding rows, and two zero fills.
__global__ void __launch_bounds__(256, 4) local_rows_kernel(const LocalRowsParams p) {
  grid_release();
  const int tid = threadIdx.x, lane = tid & 31;
  const int K = p.num_topk, vecs = p.hidden / 8;
  const size_t row_bytes = static_cast<size_t>(p.hidden) * 2;
  const size_t gid = static_cast<size_t>(blockIdx.x) * blockDim.x + tid, gsz = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (int m = 0; m < 2; ++m) {
    if (p.zero[m] != nullptr) zero_slice(p.zero[m], p.zero_bytes[m], gid, gsz);
    if (p.pool[m] == nullptr) continue;
    for (int e = blockIdx.x; e < p.num_experts; e += gridDim.x)
      zero_padding_rows(static_cast<char*>(p.pool[m]), p.expert_pool_block_offset[e] * kTileM, p.expert_frequency[e], vecs, tid, blockDim.x);
    const int pieces = (vecs + 255) / 256;
    const int items = p.num_tokens * pieces;
    for (int item = static_cast<int>(gid >> 5); item < items; item += static_cast<int>(gsz >> 5)) {
      const int t = item / pieces, v0 = (item - t * pieces) * 256;
      const int slot = lane < K ? p.pair_slot[static_cast<size_t>(t) * K + lane] : -1;
      copy_row_piece<8>(static_cast<const char*>(p.rows[m]) + t * row_bytes, static_cast<char*>(p.pool[m]), nullptr, v0, vecs, K, slot, lane);
    }
  }
}

void launch_local_rows(const LocalRowsParams& p, cudaStream_t stream) {
  const long long warps = static_cast<long long>(p.num_tokens) * ((p.hidden / 8 + 255) / 256);
  long long blocks = (warps + 7) / 8;
  if (blocks > 8 * local_sms()) blocks = 8 * local_sms();
  if (blocks < 1) blocks = 1;
  local_rows_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(p);
}

}  // namespace sep
