// Router: logits = x @ w_gate^T, softmax, top-k, renormalise, rank bitmap.
// The reference has no router; its harnesses build routing with torch ops
// (stream_ep/stream_moe/profile_pipeline.py:102-139).
#include <atomic>
#include <cuda.h>

#include "api.h"
#include "ptx.cuh"

namespace sep {

constexpr int kRouterMaxExpertsPerLane = 16;   // up to 512 experts
constexpr int kRouterMaxSplits = 8;            // CTAs of a cluster that share the hidden dimension of a token tile

// One warp finishes one token from its fp32 logits (shared memory): softmax over all experts, top-k by repeated arg-max
// (ties -> lowest expert id), renormalise, rank bitmap.  EPL = experts per lane.  Probabilities are not negative, so their
// bit patterns order like the values and the arg-max is two warp reductions of the hardware (value, then lowest id)
// instead of ten shuffles: the finishing part of the router took 10 us for 8192 tokens x 64 experts with shuffles.
template <int EPL, class Row>
__device__ __forceinline__ void route_token(const RouterParams& p, Row row, int t, int lane) {
  const int E = p.num_experts, K = p.num_topk;
  const int e_local = E / p.num_ranks;
  float logit[EPL];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int e = j * 32 + lane;
    logit[j] = (e < E) ? row(e) : -INFINITY;
    mx = fmaxf(mx, logit[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int e = j * 32 + lane;
    logit[j] = (e < E) ? __expf(logit[j] - mx) : 0.f;
    sum += logit[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
  unsigned key[EPL];            // probability bits + 1 (0: taken, or no such expert)
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int e = j * 32 + lane;
    const float prob = logit[j] * inv;
    if (p.probs != nullptr && e < E) p.probs[static_cast<size_t>(t) * E + e] = prob;
    key[j] = e < E ? __float_as_uint(prob) + 1u : 0u;
  }
  float wsum = 0.f, my_w = 0.f;
  int my_e = -1;
  unsigned rank_mask = 0;
  for (int k = 0; k < K; ++k) {
    unsigned best = 0;
#pragma unroll
    for (int j = 0; j < EPL; ++j) best = max(best, key[j]);
    const unsigned top = __reduce_max_sync(0xffffffffu, best);
    unsigned mine = 0x7fffffffu;
#pragma unroll
    for (int j = EPL - 1; j >= 0; --j)
      if (key[j] == top) mine = j * 32 + lane;
    const int best_e = static_cast<int>(__reduce_min_sync(0xffffffffu, mine));
#pragma unroll
    for (int j = 0; j < EPL; ++j)
      if (j * 32 + lane == best_e) key[j] = 0;
    const float v = __uint_as_float(top - 1u);
    if (lane == k) { my_w = v; my_e = best_e; }
    wsum += v;
    rank_mask |= 1u << (best_e / e_local);
  }
  if (lane < K) {
    p.topk_idx[static_cast<size_t>(t) * K + lane] = my_e;
    p.topk_weights[static_cast<size_t>(t) * K + lane] = p.renormalize ? my_w / wsum : my_w;
  }
  if (lane < p.num_ranks && p.is_token_in_rank != nullptr)
    p.is_token_in_rank[static_cast<size_t>(t) * p.num_ranks + lane] = (rank_mask >> lane) & 1u;
}

// ---------------------------------------------------------------------------------------------
// Tensor-core router, one launch.  A unit of `p.tile_tokens` tokens belongs to a cluster of `splits` CTAs; each multiplies
// its share of the hidden dimension, W_gate (experts, 128 per accumulator) times the tokens (the narrow UMMA
// dimension, 16..128), both K-major through TMA, and leaves its partial logits in shared memory; then every CTA of the
// cluster finishes its share of the tokens, adding the partial sums over distributed shared memory.
//
// What bounds it: reading x once (HBM) for long calls, and latency for short ones; the products are nothing.  With W_gate
// as the wide operand the token tile is free: 8192 tokens make 128 CTAs of 64 tokens, and a decoding step of 64
// tokens with 256 experts uses 32 CTAs where one CTA used to walk the whole hidden dimension (42 us).
// ---------------------------------------------------------------------------------------------
constexpr int kRouterBK = 64;
constexpr int kRouterThreads = 512;
constexpr int kRouterMaxStages = 8;
constexpr int kRouterMaxSmem = 224 * 1024;

// logits of a tile: rows of e_pad floats (odd, so that the 32 experts a warp writes for one token and the rows of
// consecutive tokens fall into different banks)
__host__ __device__ constexpr int router_e_pad(int experts) { return (experts + 127) / 128 * 128 + 1; }

template <int EPL>
__global__ void __launch_bounds__(kRouterThreads, 1)
router_mma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const RouterParams p, const RouterTile g,
                  StatusBlock* status, unsigned long long budget) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kRouterMaxStages], empty_bar[kRouterMaxStages], done_bar;
  __shared__ uint32_t s_tmem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = static_cast<int>(blockIdx.x) % g.splits, tile = static_cast<int>(blockIdx.x) / g.splits;
  const int n = g.tile_tokens, nb = g.blocks;
  const int k_blocks = (p.hidden + kRouterBK - 1) / kRouterBK;
  const int kb0 = k_blocks * split / g.splits, kb1 = k_blocks * (split + 1) / g.splits;
  const int stage_bytes = nb * 128 * 128 + n * 128;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
    for (int s = 0; s < g.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc<1>(&s_tmem, g.tmem_cols); tmem_relinquish<1>(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = s_tmem;
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0; int issued = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, budget, status)) { ok = false; break; }
        unsigned char* s = smem + stage * stage_bytes;
        mbar_arrive_expect_tx(&full_bar[stage], stage_bytes);
        for (int b = 0; b < nb; ++b) tma_load_3d(s + b * 128 * 128, &map_w, &full_bar[stage], kb * kRouterBK, b * 128, 0);
        tma_load_3d(s + nb * 128 * 128, &map_x, &full_bar[stage], kb * kRouterBK, tile * n, 0);
        ++issued;
        if (++stage == g.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) {
        report_failure(status, kStatusTimeoutPipeline, kKernelGemm, 0, 0, tile, split, 0);
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {}          // copies in flight land before the CTA leaves (bounded)
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_bf16(128, 0, 0, 0) | (static_cast<uint32_t>(n >> 3) << 17);
    int stage = 0; uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, budget, status))) { ok = false; break; }
      tc_fence_after_sync();
      if (elect_one()) {
        const uint32_t a = smem_u32(smem + stage * stage_bytes), b = a + nb * 128 * 128;
        for (int m = 0; m < nb; ++m)
#pragma unroll
          for (int j = 0; j < kRouterBK / 16; ++j)
            umma_bf16_ss<1>(tmem + m * n, umma_smem_desc(a + m * 128 * 128 + j * 32, 16, 1024), umma_smem_desc(b + j * 32, 16, 1024), idesc,
                            (kb > kb0 || j > 0) ? 1u : 0u);
        umma_commit<1>(&empty_bar[stage]);
        if (kb == kb1 - 1) umma_commit<1>(&done_bar);
      }
      __syncwarp();
      if (++stage == g.stages) { stage = 0; phase ^= 1; }
    }
    if (!ok) report_failure(status, kStatusTimeoutPipeline, kKernelGemm, 1, 0, tile, split, 0);
  }
  __syncwarp();
  const int e_pad = router_e_pad(p.num_experts);
  float* logits = reinterpret_cast<float*>(smem);              // the operand ring is free once the products are done
  const bool have = kb1 > kb0;
  if (have && !mbar_wait(&done_bar, 0, budget, status)) ok = false;
  ok = __syncthreads_and(ok ? 1 : 0) != 0;
  if (ok) {
    tc_fence_after_sync();
    // TMEM lane = expert within its block of 128, column = token: a warp reads the 32 experts of its quarter
    const int quarter = warp & 3;
    for (int job = warp >> 2; job < nb * (n / 16); job += kRouterThreads / 128) {
      const int b = job / (n / 16), c = job - b * (n / 16);
      uint32_t r[16];
      if (have) {
        tmem_ld_32x16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + b * n + c * 16, r);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) logits[(c * 16 + i) * e_pad + b * 128 + quarter * 32 + lane] = __uint_as_float(r[i]);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (g.splits > 1) cluster_sync();
  if (ok) {
    for (int tt = split + warp * g.splits; tt < n; tt += g.splits * (kRouterThreads / 32)) {
      const int t = tile * n + tt;
      if (t >= p.num_tokens) break;
      if (g.splits == 1) {
        route_token<EPL>(p, [&](int e) { return logits[tt * e_pad + e]; }, t, lane);
      } else {
        route_token<EPL>(p, [&](int e) {
          float v[kRouterMaxSplits];
#pragma unroll
          for (int s = 0; s < kRouterMaxSplits; ++s) v[s] = s < g.splits ? ld_cluster_f32(cluster_map(&logits[tt * e_pad + e], s)) : 0.f;
          float sum = 0.f;
#pragma unroll
          for (int s = 0; s < kRouterMaxSplits; ++s) sum += v[s];
          return sum;
        }, t, lane);
      }
    }
  }
  if (g.splits > 1) cluster_sync();       // the peers have read this CTA's logits
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc<1>(tmem, g.tmem_cols); }
}

RouterTile router_tile(const RouterParams& p, int sms) {
  RouterTile g{};
  g.blocks = (p.num_experts + 127) / 128;
  const int k_blocks = (p.hidden + kRouterBK - 1) / kRouterBK;
  const int most = p.num_experts > 256 ? 64 : 128;             // (the tile's logits have to fit shared memory)
  // Wide token tiles re-read W_gate least; the hidden dimension is split to fill the GPU, and only then do tiles shrink.
  g.tile_tokens = p.num_tokens > 64 * sms ? most : 64;
  for (;;) {
    const int tiles = (p.num_tokens + g.tile_tokens - 1) / g.tile_tokens;
    g.splits = 1;
    while (g.splits < kRouterMaxSplits && tiles * g.splits * 2 <= sms && k_blocks >= 4 * g.splits) g.splits *= 2;
    if (tiles * g.splits * 2 > sms || g.tile_tokens == 16) break;
    g.tile_tokens /= 2;
  }
  const int stage = g.blocks * 128 * 128 + g.tile_tokens * 128;
  const int logits = g.tile_tokens * router_e_pad(p.num_experts) * 4;
  g.stages = (kRouterMaxSmem - 1024) / stage;
  if (g.stages > kRouterMaxStages) g.stages = kRouterMaxStages;
  g.smem_bytes = (g.stages * stage > logits ? g.stages * stage : logits) + 1024;
  g.tmem_cols = 32;
  while (g.tmem_cols < g.blocks * g.tile_tokens) g.tmem_cols *= 2;
  return g;
}

template <int EPL>
static cudaError_t launch_router_width(const RouterParams& p, const RouterTile& g, const CUtensorMap& map_w, const CUtensorMap& map_x,
                                       StatusBlock* status, unsigned long long budget, cudaStream_t stream) {
  auto kernel = router_mma_kernel<EPL>;
  static std::atomic<bool> configured[64];      // the shared-memory limit is an attribute of the function on a device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRouterMaxSmem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((p.num_tokens + g.tile_tokens - 1) / g.tile_tokens * g.splits));
  cfg.blockDim = dim3(kRouterThreads);
  cfg.dynamicSmemBytes = g.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = g.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, p, g, status, budget);
}

cudaError_t launch_router_mma(const RouterParams& p, const void* map_w, const void* map_x, int sms, StatusBlock* status,
                              unsigned long long wait_budget_ns, cudaStream_t stream) {
  const RouterTile g = router_tile(p, sms);
  const CUtensorMap &mw = *static_cast<const CUtensorMap*>(map_w), &mx = *static_cast<const CUtensorMap*>(map_x);
  if (p.num_experts <= 32) return launch_router_width<1>(p, g, mw, mx, status, wait_budget_ns, stream);
  if (p.num_experts <= 64) return launch_router_width<2>(p, g, mw, mx, status, wait_budget_ns, stream);
  if (p.num_experts <= 128) return launch_router_width<4>(p, g, mw, mx, status, wait_budget_ns, stream);
  if (p.num_experts <= 256) return launch_router_width<8>(p, g, mw, mx, status, wait_budget_ns, stream);
  return launch_router_width<kRouterMaxExpertsPerLane>(p, g, mw, mx, status, wait_budget_ns, stream);
}

// ---------------------------------------------------------------------------------------------
// SIMT router (Runtime.set_router_on_tensor_cores(False)): an fp32 GEMM on the CUDA cores.
// ---------------------------------------------------------------------------------------------
constexpr int kRouterKChunk = 64;              // hidden elements per shared-memory step (128 bytes of a row)
constexpr int kRouterLd = kRouterKChunk + 4;   // padded row: float4 reads of 8 consecutive rows hit 32 different banks

// One CTA routes TOK tokens with TOK * 4 threads.  Logits: a register-tiled fp32 GEMM, (TOK / 4) x 16 threads
// with 4 tokens x JE experts each, so one pass covers 16 * JE experts (16 / 32 / 64; wider expert counts loop).
// Operands are fetched 128 contiguous bytes per row (8 lanes per row), converted to fp32 and kept row-major in
// shared memory; the global loads of the next two chunks are in flight while the current one is multiplied.
// Few experts make the kernel latency-bound, so those instances use 32 tokens per CTA (twice the CTAs); 64
// experts per pass are FMA-bound and use 64 tokens for operand reuse.  Then each warp finishes 8 tokens:
// softmax over all experts, top-k by repeated arg-max, renormalise, rank bitmap.
template <int JE, int TOK>
__global__ void __launch_bounds__(TOK * 4) router_kernel(const RouterParams p) {
  constexpr int THREADS = TOK * 4;
  constexpr int NE = 16 * JE;                                      // experts per pass
  constexpr int EPL = JE == 4 ? kRouterMaxExpertsPerLane : 1;      // experts per lane in the softmax / top-k part
  constexpr int XV = TOK * 8 / THREADS;                            // 16-byte loads of x per thread and chunk (2)
  constexpr int WV = (NE * 8 + THREADS - 1) / THREADS;             // ... of the gate weights (1 or 2)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* xs = reinterpret_cast<float*>(smem_raw);                 // [TOK tokens][kRouterLd]
  float* ws = xs + TOK * kRouterLd;                               // [NE experts][kRouterLd]
  float* logits = ws + NE * kRouterLd;                            // [TOK tokens][e_pad]
  const int E = p.num_experts, H = p.hidden;
  const int e_pad = (E + NE - 1) / NE * NE + 1;                   // +1: rows start in different banks
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = tid >> 4, tx = tid & 15;
  const __nv_bfloat16* xg = static_cast<const __nv_bfloat16*>(p.x);
  const __nv_bfloat16* wg = static_cast<const __nv_bfloat16*>(p.w_gate);
  const int t0 = blockIdx.x * TOK;

  for (int e0 = 0; e0 < E; e0 += NE) {
    float acc[4][JE];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < JE; ++j) acc[i][j] = 0.f;
    uint4 xv0[XV], wv0[WV], xv1[XV], wv1[WV];
    auto fetch = [&](int k0, uint4 (&xv)[XV], uint4 (&wv)[WV]) {
#pragma unroll
      for (int i = 0; i < XV; ++i) {
        const int idx = tid + THREADS * i, row = idx >> 3, kk = k0 + (idx & 7) * 8;
        xv[i] = (t0 + row < p.num_tokens && kk < H) ? ld_nc_v4(xg + static_cast<size_t>(t0 + row) * H + kk)
                                                    : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < WV; ++i) {
        const int idx = tid + THREADS * i, row = idx >> 3, kk = k0 + (idx & 7) * 8;
        wv[i] = (row < NE && e0 + row < E && kk < H)
                    ? __ldg(reinterpret_cast<const uint4*>(wg + static_cast<size_t>(e0 + row) * H + kk))
                    : make_uint4(0, 0, 0, 0);
      }
    };
    auto stash1 = [&](float* dst, const uint4& v, int idx) {
      const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
      float4* o = reinterpret_cast<float4*>(dst + (idx >> 3) * kRouterLd + (idx & 7) * 8);
      o[0] = make_float4(a.x, a.y, b.x, b.y);
      o[1] = make_float4(c.x, c.y, d.x, d.y);
    };
    // one chunk: registers -> shared memory, refill the registers two chunks ahead, multiply
    auto chunk = [&](int k_next, uint4 (&xv)[XV], uint4 (&wv)[WV]) {
      __syncthreads();   // the previous chunk's tiles are no longer read
#pragma unroll
      for (int i = 0; i < XV; ++i) stash1(xs, xv[i], tid + THREADS * i);
#pragma unroll
      for (int i = 0; i < WV; ++i)
        if (tid + THREADS * i < NE * 8) stash1(ws, wv[i], tid + THREADS * i);
      __syncthreads();
      if (k_next < H) fetch(k_next, xv, wv);                       // in flight during this and the next multiply
#pragma unroll 4
      for (int k = 0; k < kRouterKChunk; k += 4) {
        float4 a[4], b[JE];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(xs + (ty * 4 + i) * kRouterLd + k);
#pragma unroll
        for (int j = 0; j < JE; ++j) b[j] = *reinterpret_cast<const float4*>(ws + (j * 16 + tx) * kRouterLd + k);   // lanes on consecutive rows: no bank conflict
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < JE; ++j) {
            acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
            acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
            acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
            acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
          }
      }
    };
    fetch(0, xv0, wv0);
    if (kRouterKChunk < H) fetch(kRouterKChunk, xv1, wv1);
    for (int k0 = 0; k0 < H; k0 += 2 * kRouterKChunk) {
      chunk(k0 + 2 * kRouterKChunk, xv0, wv0);
      if (k0 + kRouterKChunk >= H) break;
      chunk(k0 + 3 * kRouterKChunk, xv1, wv1);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < JE; ++j) logits[(ty * 4 + i) * e_pad + e0 + j * 16 + tx] = acc[i][j];
  }
  __syncthreads();

  for (int tt = warp; tt < TOK; tt += THREADS / 32) {
    const int t = t0 + tt;
    if (t >= p.num_tokens) break;
    route_token<EPL>(p, [&](int e) { return logits[tt * e_pad + e]; }, t, lane);
  }
}

template <int JE, int TOK>
static void launch_router_je(const RouterParams& p, cudaStream_t stream) {
  constexpr int NE = 16 * JE;
  const int e_pad = (p.num_experts + NE - 1) / NE * NE + 1;
  const size_t smem = sizeof(float) * (static_cast<size_t>(TOK + NE) * kRouterLd + static_cast<size_t>(TOK) * e_pad);
  const int grid = (p.num_tokens + TOK - 1) / TOK;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(router_kernel<JE, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  router_kernel<JE, TOK><<<grid, TOK * 4, smem, stream>>>(p);
}

void launch_router(const RouterParams& p, cudaStream_t stream) {
  if (p.num_experts <= 16) launch_router_je<1, 32>(p, stream);
  else if (p.num_experts <= 32) launch_router_je<2, 32>(p, stream);
  else launch_router_je<4, 64>(p, stream);
}

}  // namespace sep
