// The kernel template of the library's GEMMs (instances: gemm_inst_*.cu, launch: gemm_kernels.cu).
//
// Persistent grouped GEMM for sm_100a: TMA-fed shared-memory pipeline, tcgen05.mma with fp32
// accumulators in tensor memory (two accumulator buffers so the epilogue of tile i overlaps the
// main loop of tile i+1), and fused epilogues read back with tcgen05.ld.
//
// One kernel template covers every GEMM-shaped op of the MoE layer:
//   kernel A      pool[rows,H]   x W1[e]^T  -> SwiGLU on adjacent column pairs (+ optional preact)
//   kernel Y      postact[rows,I] x W2[e]^T -> x topk weight -> bf16x2 red.add scatter (local o, or the
//                                              source rank's output over NVLink = fused combine)
//   kernel Y_bwd  dL_do[rows,H]  x W2[e]    -> dswiglu, dL/dweight, zero padding rows
//   kernel A_bwd  dswiglu[rows,2I] x W1[e]  -> red.add scatter (local, or fused combine_grads)
//   dW1 / dW2     A[rows,M]^T x B[rows,N] per expert with true-length K masking
//   preact recompute = kernel A with the plain store epilogue
// Two widths of a work unit: CG = 1, one CTA per 128-row tile; CG = 2, a cluster of two CTAs per pair of row tiles of one
// expert (tcgen05 cta_group::2): each CTA loads its own 128 rows of A and HALF of the B tile, so a k-block costs
// an SM 32 KB of operands instead of 48 KB for the same 128 x 256 x 64 products.  The operand feed is what bounds these
// kernels (the MMA thread waited 19-26 % of its time for it with CG = 1), and the smaller stage also allows 6 stages
// instead of 4.
//
// The kernel optionally carries extra "push" warps that ship token rows into peers' pools while the
// tensor-core warps consume tiles as they complete (dispatch fused with the GEMM).
//
// Reference counterparts: stream_ep/stream_moe/kernel_a.py, kernel_y.py, kernel_y_bwd.py,
// kernel_a_bwd.py, tile_scheduler.py, epi_ops.py and the quack.gemm calls at
// stream_ep/stream_moe/stream_moe.py:993-1004,1111-1142 (all Hopper WGMMA through CuTeDSL there).
#pragma once

#include <atomic>
#include <type_traits>
#include <cuda.h>

#include "comm_common.cuh"

namespace sep {

constexpr int BM = 128;          // rows per tile == pool tile_m
constexpr int BK = 64;           // bf16 elements per k-block: one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int kGemmWarps = 10;   // 0: TMA producer, 1: MMA issuer + TMEM owner, 2..9: epilogue
// The kernels that consume tiles as a dispatch completes them (A and Y_bwd) carry one more warp whose lane 0 polls
// the tile gates AHEAD of the TMA producer.  A gate poll is an acquire load at system scope, microseconds long
// while NVLink traffic is landing; done by the producer itself it stalls the operand pipeline once per tile.
constexpr bool has_gate_warp(int epi) { return epi == kEpiSwiglu || epi == kEpiDswiglu; }
// The weight-gradient kernels (VarlenK, both operands MN-major) carry one whose lane 0 schedules: it claims the next unit, reads
// its expert's rows and queues the result for the other roles of both CTAs.  Operands arrive at the rate at which L2 delivers
// them, so time that the producer spends on anything else is never made up for: a claim (an atomic, a copy to the other CTA, two
// loads), and each store with release semantics, which waits for the copies in flight.  The other roles therefore report to
// the scheduler with plain stores (of units with products, see s_q).  Before and after, with the wider stores below, thousand SM cycles of
// the MMA loop and us of a launch on its own: 32 experts of 512 rows, hidden 3072, ffn 768 425 -> 314, 268 -> 219 us; of 1250 rows, hidden
// 7168, ffn 2048 4170 -> 3725, 2850 -> 2720; 12 of 440, hidden 1000, ffn 520 48 -> 38, 42 -> 37; 4 of 4096, hidden and ffn 4096 1532 -> 1523,
// 1156 -> 1160.  Long units beside narrow outputs lose: 8 of 6144, hidden 2048, ffn 1408 783 -> 791, 603 -> 613 us, hidden 4096 1564 -> 1580;
// all pairs then wait alike for operands (322 -> 364 thousand cycles), where claims had set them apart.  The kernels over row tiles,
// whose order is static, lose by such a queue (Y of 32008 rows 171 -> 187).
constexpr int base_warps(int epi, bool schedules) { return kGemmWarps + (schedules || has_gate_warp(epi) ? 1 : 0); }
// extra warps of the fused variants; the dSwiGLU epilogue keeps two preact segments in registers, so it gets fewer
// (Y_bwd: 16 warps x 128 registers, A: 20 warps x 96 registers fill the register file)
constexpr int push_warps(int epi) { return epi == kEpiDswiglu ? 5 : 9; }
constexpr int kMaxDevices = 64;  // per-device host-side tables (kernel attributes, no-alloc scratch address)
constexpr int kTileQueue = 8;    // tiles the scheduler may be ahead of the epilogue
// A claimed tile is work that no idle CTA can take any more, so the scheduler claims late: when the producer has this many
// k-blocks of the tile before left to issue, about the time that a claim takes until its first operands can be requested.  Thousand
// cycles more than at 10 with 2, 5, 20 and 40: 32 experts of 512 rows 39, 4, 0, 0; of 1250 rows 265, 35, 1, 2; 8 of 6144 18, 4, 0, 1.
constexpr int kClaimAhead = 10;
constexpr int kEpiWarps = 8;     // two threads per accumulator row: each takes half of the tile's columns

template <int BN, int CG> struct GemmCfg {
  static constexpr int kBN = BN / CG;                         // columns of B this CTA loads
  static constexpr int kABytes = BM * BK * 2;                 // 16 KB
  static constexpr int kBBytes = kBN * BK * 2;                // 16 / 32 KB
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = (kBN == 256) ? 4 : 6;
  static constexpr int kTmemCols = 2 * BN;                    // two accumulator buffers
  static constexpr int kBarrierBytes = 256;
  static constexpr int kEpiStageBytes = 4096;                 // per epilogue warp: 32 rows x 128 bytes
  static constexpr int kSmemBytes = kStages * kStageBytes + 8 * kEpiStageBytes + kBarrierBytes + 1024;  // + alignment slack
};

// Columns of the output tile that starts at `n0` which are multiplied: the last tile of a width that is no multiple of BN
// runs narrower MMAs (UMMA N is a multiple of 32 in the pair form) instead of multiplying columns nobody stores.
template <int BN>
__device__ __forceinline__ int tile_cols(int n, int n0) { return min(BN, (n - n0 + 31) / 32 * 32); }

struct SecondMaps { CUtensorMap a, b, o; };   // operands and output of the second VarlenK problem

// What the scheduler queues: a linear tile index (past the last tile: the end) and what decode_tile found for it.
struct __align__(16) TileEntry { int lin, m_tile, n_tile, expert, row0, k_blocks, k_tail, prob; };

struct TileCoord {
  int prob;        // VarlenK: 0 / 1 = first / second problem of the launch
  int m_tile, n_tile, expert;
  int row0;        // first row of A (VarlenM: m_tile * BM; VarlenK: first pool row of the expert)
  bool rows_valid; // false: the second CTA of a pair whose expert (or output) has an odd number of row tiles
  int k_blocks;    // number of BK blocks to accumulate
  int k_tail;      // VarlenK: valid rows in the last block (0 = full)
};

// Tile order.  Consecutive linear indices (= CTAs working at the same time) walk a band of kBandM row tiles
// column by column: a wave of 148 tiles then shares kBandM A tiles and ~148/kBandM B tiles instead of one A
// tile and 148 B tiles, which keeps weight traffic out of HBM when one expert's weights exceed the L2.
// Bands follow the pool order (expert-major), i.e. the order in which dispatch completes tiles.  GemmParams::band asks for
// higher ones (see tile_band in runtime.cpp).
constexpr int kBandM = 8;

__device__ __forceinline__ void band_decode(int band_m, int lin, int num_m, int num_n, int& m_tile, int& n_tile) {
  const int band = lin / (band_m * num_n);
  const int rem = lin - band * (band_m * num_n);
  const int m0 = band * band_m;
  const int gm = min(band_m, num_m - m0);
  n_tile = rem / gm;
  m_tile = m0 + (rem - n_tile * gm);
}

// `num_m`: live number of M units, i.e. row tiles (CG = 1) or pairs of row tiles (CG = 2); may come from device memory.
// Ignored for VarlenK.  `half` = rank of this CTA in its pair (0 with CG = 1).  The kernels over row tiles decode in every role,
// straight into the coordinates: by way of a TileEntry the six instances with a fused push spilled 8 to 20 bytes a thread
// instead of 0 to 12.
template <int CG>
__device__ __forceinline__ TileCoord decode_tile(const GemmParams& p, int lin, int num_m, int half) {
  TileCoord t;
  t.prob = 0;
  t.rows_valid = true;
  if (p.mode == kVarlenM) {
    band_decode(p.band > 0 ? p.band / CG : kBandM / CG, lin, num_m, p.num_n_tiles, t.m_tile, t.n_tile);
    if (CG == 2) {
      const int pair = p.pair_tiles[t.m_tile];       // first tile * 2 + (1 if the pair has a second tile)
      t.m_tile = pair >> 1;
      if (half != 0) { if (pair & 1) ++t.m_tile; else t.rows_valid = false; }   // no second tile: its loads repeat the first
    }
    t.expert = p.tile_id_to_expert[t.m_tile];
    t.row0 = t.m_tile * BM;
    t.k_blocks = (p.K + BK - 1) / BK;
    t.k_tail = 0;
  } else {
    int nm = p.num_m_tiles, nn = p.num_n_tiles, m_out = p.M_out;
    const int first = p.num_experts * nm * nn;
    if (lin >= first) { t.prob = 1; lin -= first; nm = p.num_m_tiles2; nn = p.num_n_tiles2; m_out = p.M_out2; }
    const int per_e = nm * nn;
    t.expert = lin / per_e;
    band_decode(p.band > 0 ? p.band / CG : kBandM / CG, lin - t.expert * per_e, nm, nn, t.m_tile, t.n_tile);
    if (CG == 2) { t.m_tile = t.m_tile * 2 + half; t.rows_valid = t.m_tile * BM < m_out; }
    t.row0 = p.expert_pool_block_offset[t.expert] * BM;
    const int len = p.expert_frequency[t.expert];
    t.k_blocks = (len + BK - 1) / BK;
    t.k_tail = len % BK;
  }
  return t;
}

// A queued VarlenK unit (decoded for the pair's first CTA) as it looks to CTA `half` of the pair.
template <int CG>
__device__ __forceinline__ TileCoord unit_coord(const GemmParams& p, const TileEntry& e, int half) {
  TileCoord t;
  t.prob = e.prob; t.n_tile = e.n_tile; t.expert = e.expert; t.row0 = e.row0; t.k_blocks = e.k_blocks; t.k_tail = e.k_tail;
  t.m_tile = e.m_tile + half;
  t.rows_valid = CG == 1 || t.m_tile * BM < (e.prob ? p.M_out2 : p.M_out);
  return t;
}

__device__ __forceinline__ void st_global_v4(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" :: "l"(p), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ int atom_add_acq_rel_gpu(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// OR of `pred` over the 256 epilogue threads (named barrier 1, as epi_bar_sync): every thread gets the same answer.
__device__ __forceinline__ bool epi_vote_any(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(static_cast<uint32_t>(pred)) : "memory");
  return r != 0;
}

template <int BN, bool A_MN, bool B_MN, int EPI, bool PUSH, int CG>
__global__ void __launch_bounds__((base_warps(EPI, A_MN) + (PUSH ? push_warps(EPI) : 0)) * 32, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_o0, const __grid_constant__ CUtensorMap tmap_o1,
                    const GemmParams p, const PushParams pp, const __grid_constant__ SecondMaps maps2) {
  using Cfg = GemmCfg<BN, CG>;
  extern __shared__ unsigned char smem_dyn[];
  // 128-byte swizzle atoms are 1024 bytes: align the operand ring accordingly.
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* stage_base = smem;
  unsigned char* epi_stage = smem + Cfg::kStages * Cfg::kStageBytes;      // 8 x 4 KB, 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_stage + 8 * Cfg::kEpiStageBytes);
  uint64_t* full_bar = bars;                               // [kStages]
  uint64_t* empty_bar = bars + Cfg::kStages;               // [kStages]
  uint64_t* tmem_full = bars + 2 * Cfg::kStages;           // [2]
  uint64_t* tmem_empty = bars + 2 * Cfg::kStages + 2;      // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * Cfg::kStages + 4);
  int* s_flag = reinterpret_cast<int*>(tmem_slot + 1);     // epilogue broadcast word
  __shared__ PushTargets s_tg;
  __shared__ int s_push_ok;
  __shared__ int s_gates_open;   // how many of this CTA's tiles have an open gate (-1: the gate warp gave up)
  __shared__ int s_tiles_done;   // tiles whose epilogue finished (read by the time stamps only)
  __shared__ uint64_t s_push_bar[32][2];   // push-only CTAs: two bulk-load barriers per warp
  // The scheduler's queue.  It overwrites an entry once every role that reads it has reported so.  A unit with products: producers
  // and MMA warp report with plain stores, since the epilogue, whose report is a release, comes after the copies and products
  // that were issued from what they read.  A unit without any (an expert without rows) makes no role wait for another, so each
  // reports with a release, on a path of its own (chosen at each report, 32 experts of 512 rows took 319 thousand cycles for 314);
  // a later plain store by the same thread to the same counter still carries it.
  __shared__ TileEntry s_q[kTileQueue];
  __shared__ int s_q_head, s_q_tail;       // ... how many tiles were queued, how many the epilogue has finished
  __shared__ int s_q_read, s_q_prod;       // ... how many entries the MMA warp has read, how many the producer is (nearly) done with
  __shared__ int s_q_tail_peer, s_q_read_peer;   // (CG = 2, first CTA of a pair) the peer's epilogue / producer
  __shared__ char* s_remote_out[kMaxRanks];
  __shared__ float* s_remote_dw[kMaxRanks];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half_of_pair = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;   // the pair's first CTA issues its MMAs
  const bool leader = half_of_pair == 0;
  const int unit = static_cast<int>(blockIdx.x) / CG, num_units = static_cast<int>(gridDim.x) / CG;
  // Tile feed.  Static: CTA b takes tiles b, b + stride, ...  Dynamic (VarlenK with a counter): tiles are claimed.  VarlenK units are
  // queued by the scheduler warp of the first CTA, in shared memory of both CTAs; otherwise every role decodes on its own.
  constexpr bool queued = A_MN;
  const bool dyn = p.mode == kVarlenK && p.tile_counter != nullptr;
  const unsigned long long budget = p.wait_budget_ns;
  // Fused push, two ways of sharing the GPU.  Mixed (push_ctas == 0): every CTA multiplies and its extra warps push.
  // Dedicated (push_ctas > 0): the last push_ctas CTAs only push, with all their warps, and the others only multiply.
  // Remote stores that wait for NVLink credit back up in an SM's load/store path, where the epilogue warps of
  // the same SM queue behind them: with the push on SMs of its own the GEMM runs at its stand-alone rate.
  const int num_push_ctas = PUSH ? min((max(pp.push_ctas, 0) + CG - 1) / CG, num_units - 1) : 0;   // in units
  const int lin_stride = num_units - num_push_ctas;
  const bool is_push_cta = PUSH && unit >= lin_stride;
  const int first_lin = is_push_cta ? 0x7fffffff : unit;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    for (int s = 0; s < Cfg::kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], kEpiWarps * CG); }
    mbar_fence_init();
    if (blockIdx.x == 0 && p.started_flag != nullptr) atomicAdd(p.started_flag, 1);
    if (PUSH) s_push_ok = 1;
    s_gates_open = 0;
    s_tiles_done = 0;
    s_q_head = 0; s_q_tail = 0; s_q_read = 0; s_q_prod = 0; s_q_tail_peer = 0; s_q_read_peer = 0;
    if (p.timing != nullptr) {
      long long* tm = p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols;
      tm[0] = static_cast<long long>(globaltimer_ns());
      tm[1] = 0; tm[2] = 0; tm[3] = 0; tm[4] = 0; tm[5] = 0; tm[7] = 0; tm[8] = 0; tm[9] = 0; tm[10] = 0;
    }
  }
  if (warp == 1) {
    tmem_alloc<CG>(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish<CG>();
  }
  // The barriers and the TMEM were set up while the kernel before this one drained (single-rank layer): the nine kernels of
  // a small training pass (1777 tokens, hidden 1000) 216 -> 198 us, a decoding step of 16 tokens 56.8 -> 52.7 us.  What
  // follows reads what that kernel wrote.
  grid_wait();
  grid_release();
  // Capacity mode keeps the live tile count in device memory (written by the metadata kernel earlier in the stream).
  const int num_m = (p.mode == kVarlenM && p.num_m_tiles_dev != nullptr) ? min(*p.num_m_tiles_dev, p.num_m_tiles) : p.num_m_tiles;
  const int total_tiles = p.mode == kVarlenM ? num_m * p.num_n_tiles
                                             : p.num_experts * (p.num_m_tiles * p.num_n_tiles + p.num_m_tiles2 * p.num_n_tiles2);
  if (PUSH) {
    if ((pp.flags & 1) && !pp.static_targets && blockIdx.x == 0 && warp == base_warps(EPI, A_MN) && lane < pp.num_ranks)
      publish_record(pp.own, pp.peer_base, pp.ctl, pp.kind, pp.epoch, pp.rank, lane);
  }
  if ((EPI == kEpiScatter || EPI == kEpiDswiglu) && warp == 2 && lane < p.num_ranks) {
    // Resolve buffers that every rank allocated at its own arena offset from the published records.
    if (p.remote_out.enabled) {
      if (p.remote_out.is_static) {
        s_remote_out[lane] = static_cast<char*>(p.peer_base[lane]) + p.remote_out.offset;
      } else {
        const unsigned long long* rec = fetch_record(p.peer_base[p.rank], p.ctl, p.remote_out.kind, p.remote_out.epoch,
                                                     lane, budget, p.status, kKernelGemm, p.rank);
        s_remote_out[lane] = rec ? static_cast<char*>(p.peer_base[lane]) + rec[p.remote_out.field] : nullptr;
      }
    }
    if (p.remote_dw.enabled) {
      if (p.remote_dw.is_static) {
        s_remote_dw[lane] = reinterpret_cast<float*>(static_cast<char*>(p.peer_base[lane]) + p.remote_dw.offset);
      } else {
        const unsigned long long* rec = fetch_record(p.peer_base[p.rank], p.ctl, p.remote_dw.kind, p.remote_dw.epoch,
                                                     lane, budget, p.status, kKernelGemm, p.rank);
        s_remote_dw[lane] = rec ? reinterpret_cast<float*>(static_cast<char*>(p.peer_base[lane]) + rec[p.remote_dw.field]) : nullptr;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (CG == 2) cluster_sync();      // the peer's barriers are initialised before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (is_push_cta) {
    // ------------------------------------------------------------------ push-only CTA: every warp ships rows
    if (pp.flags & 2) {
      if (warp == 0 && lane < pp.num_ranks) {
        const unsigned long long* rec = pp.static_targets
            ? reinterpret_cast<const unsigned long long*>(&pp.own)
            : fetch_record(pp.peer_base[pp.rank], pp.ctl, pp.kind, pp.epoch, lane,
                           pp.wait_budget_ns, pp.status, kKernelDispatch, pp.rank);
        if (rec == nullptr) s_push_ok = 0;
        else resolve_push_targets(s_tg, lane, pp.peer_base[lane], rec);
      }
      // The operand ring of the GEMM is unused here: every warp takes two 4 KB slots of it for bulk copies
      // (global -> shared -> owner's pool through the copy engine, see push_chunk).
      PushRing ring{};
      ring.bar = s_push_bar[warp];
      ring.ok = true;
      if (pp.bulk_push && (warp + 1) * 2 * static_cast<int>(kPushPieceBytes) <= Cfg::kStages * Cfg::kStageBytes) {
        ring.smem = smem_u32(stage_base) + warp * 2 * kPushPieceBytes;
        if (lane == 0) { mbar_init(&ring.bar[0], 1); mbar_init(&ring.bar[1], 1); mbar_fence_init(); }
      }
      __syncthreads();
      if (s_push_ok) {
        const int num_send = *pp.num_send;
        const int num_chunks = push_num_chunks(pp, num_send);
        if (p.timing != nullptr && threadIdx.x == 0)
          p.timing[static_cast<size_t>(blockIdx.x) * kTimingCols + 4] = static_cast<long long>(globaltimer_ns());
        for (;;) {
          int chunk = 0;
          if (lane == 0) chunk = ring.ok ? atomicAdd(pp.work_counter, 1) : 0x7fffffff;
          chunk = __shfl_sync(0xffffffffu, chunk, 0);
          if (chunk >= num_chunks) break;
          int p0, p1;
          push_chunk_range(pp, num_send, chunk, p0, p1);
          push_chunk(pp, s_tg, p0, p1, lane, &ring, pp.split_local ? 2 : 0);
        }
        if (p.timing != nullptr && lane == 0)
          atomicMax(reinterpret_cast<unsigned long long*>(p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols + 5), globaltimer_ns());
      }
    }
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0; int issued = 0; bool ok = true; int my_tile = 0;
      for (int it = 0; ok; ++it) {
        TileCoord t;
        int lin;
        if constexpr (queued) {
          if (!spin_until([&] { return (leader ? ld_acquire_cta_shared(&s_q_head) : ld_acquire_cluster_shared(&s_q_head)) > it; }, budget, p.status)) { ok = false; break; }
          const TileEntry e = s_q[it % kTileQueue];
          lin = e.lin;
          t = unit_coord<CG>(p, e, half_of_pair);
          if (lin >= total_tiles) break;
          if (t.k_blocks == 0) {      // nothing to load (see s_q: only this report has to order the read of the entry)
            if (CG == 2 && !leader) st_release_cluster(cluster_map(&s_q_read_peer, 0), it + 1);
            else st_release_cta_shared(&s_q_prod, it + 1);
            continue;
          }
          if (CG == 2 && !leader) st_cluster(cluster_map(&s_q_read_peer, 0), it + 1);
        } else {
          lin = first_lin + it * lin_stride;
          if (lin >= total_tiles || lin < 0) break;
          t = decode_tile<CG>(p, lin, num_m, half_of_pair);
        }
        const int n0 = t.n_tile * BN;
        const int b0 = n0 + half_of_pair * (tile_cols<BN>(t.prob ? p.N2 : p.N, n0) / CG);   // first column of B this CTA loads
        const CUtensorMap* ta = t.prob ? &maps2.a : &tmap_a;
        const CUtensorMap* tb = t.prob ? &maps2.b : &tmap_b;
        if (p.mode == kVarlenM && p.arrival_count != nullptr) {
          const unsigned long long gate_t0 = p.timing != nullptr ? globaltimer_ns() : 0ull;
          bool open;
          if constexpr (has_gate_warp(EPI)) {
            // the gate warp polls the counters ahead of this thread and publishes how far it got
            open = spin_until([&] { const int g = ld_acquire_cta_shared(&s_gates_open); return g < 0 || g > my_tile; }, budget, p.status) &&
                   ld_acquire_cta_shared(&s_gates_open) > my_tile;
          } else {
            const int target = p.arrival_target[t.m_tile];
            const int* cnt = p.arrival_count + t.m_tile;
            const bool local_only = p.num_ranks == 1;
            open = spin_until([&] { return (local_only ? ld_acquire_gpu(cnt) : ld_acquire_sys(cnt)) == target; }, budget, p.status);
            if (!open) report_failure(p.status, kStatusTimeoutTileGate, kKernelGemm, 0, p.rank, t.m_tile, target, ld_acquire_sys(cnt));
          }
          if (!open) { ok = false; break; }
          fence_proxy_async();   // rows were written through the generic proxy (possibly by a peer GPU)
          if (p.timing != nullptr) {
            long long* tm = p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols;
            tm[1] += static_cast<long long>(globaltimer_ns() - gate_t0);   // time the operand pipeline stood still for gates
            tm[7] += 1;
          }
          ++my_tile;
        }
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (queued && leader && kb == max(t.k_blocks - kClaimAhead, 0)) st_volatile_shared(&s_q_prod, it + 1);
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, budget, p.status)) {
            report_failure(p.status, kStatusTimeoutPipeline, kKernelGemm, 0, p.rank, lin, kb, stage);
            ok = false; break;
          }
          unsigned char* sa = stage_base + stage * Cfg::kStageBytes;
          unsigned char* sb = sa + Cfg::kABytes;
          // CG = 2: both CTAs' bytes are counted on the first CTA's barrier, which that CTA arms for the sum.  (Bytes of
          // the second CTA may arrive before the barrier is armed: its phase cannot complete without the arrival.)
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], CG * Cfg::kStageBytes);
          const uint32_t pair_bar = CG == 2 ? cluster_map(&full_bar[stage], 0) : 0;
          auto load = [&](unsigned char* dst, const CUtensorMap* map, int x, int y, int z) {
            if constexpr (CG == 2) tma_load_3d_pair(dst, map, pair_bar, x, y, z);
            else tma_load_3d(dst, map, &full_bar[stage], x, y, z);
          };
          const int k0 = kb * BK;
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) load(sa + j * (BK * 128), ta, t.m_tile * BM + j * 64, t.row0 + k0, 0);
          } else {
            load(sa, ta, k0, t.row0, 0);
          }
          if (B_MN) {
            const int kz = (p.mode == kVarlenM) ? k0 : t.row0 + k0;
            const int ez = (p.mode == kVarlenM) ? t.expert : 0;
#pragma unroll
            for (int j = 0; j < Cfg::kBN / 64; ++j) load(sb + j * (BK * 128), tb, b0 + j * 64, kz, ez);
          } else {
            load(sb, tb, k0, b0, t.expert);
          }
          ++issued;
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // Drain: every copy this thread issued must have landed before the CTA may exit.
        if (CG == 2) {          // the copies of a pair are counted in one place for both CTAs: let them land (bounded)
          const unsigned long long t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 2000000ull) {}
          issued = 0;
        }
        const int pending = issued < Cfg::kStages ? issued : Cfg::kStages;
        for (int i = 0; i < pending; ++i) {
          int s = stage - 1 - i; uint32_t ph = phase;
          if (s < 0) { s += Cfg::kStages; ph ^= 1; }
          const unsigned long long t0 = globaltimer_ns();
          while (!mbar_try_wait(&full_bar[s], ph) && globaltimer_ns() - t0 < 2000000ull) {}
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (one per unit)
    constexpr uint32_t idesc0 = umma_idesc_bf16(BM * CG, 0, A_MN ? 1 : 0, B_MN ? 1 : 0);
    if (leader) {
    int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
    // With time stamps on the loop also counts where this warp's time goes (SM cycles, see GemmParams::timing).  The
    // loop is compiled twice: even a predicated-off clock read between "operands have landed" and the MMA issue
    // cost 2 % of the whole step.
    long long cyc_operands = 0, cyc_accumulator = 0;
    const long long cyc_begin = p.timing != nullptr ? clock64() : 0;
    auto tile_loop = [&](auto timed) {
    constexpr bool stamp = decltype(timed)::value;
    for (int it = 0; ok; ++it) {
      TileCoord t;
      if constexpr (queued) {
        if (!__all_sync(0xffffffffu, spin_until([&] { return ld_acquire_cta_shared(&s_q_head) > it; }, budget, p.status))) { ok = false; break; }
        const TileEntry e = s_q[it % kTileQueue];
        if (e.lin >= total_tiles) break;
        __syncwarp();
        if (e.k_blocks == 0) {        // an expert without rows: the epilogue writes zeros on its own
          if (lane == 0) st_release_cta_shared(&s_q_read, it + 1);
          continue;
        }
        if (lane == 0) st_volatile_shared(&s_q_read, it + 1);
        t = unit_coord<CG>(p, e, 0);
      } else {
        const int lin = first_lin + it * lin_stride;
        if (lin >= total_tiles || lin < 0) break;
        t = decode_tile<CG>(p, lin, num_m, 0);
      }
      const uint32_t idesc = idesc0 | (static_cast<uint32_t>(tile_cols<BN>(t.prob ? p.N2 : p.N, t.n_tile * BN) >> 3) << 17);
      // all 32 lanes wait; the outcome is made warp-uniform so that no lane leaves ahead of elect_one / __syncwarp
      long long c_acc = 0;
      if constexpr (stamp) c_acc = clock64();
      if (!__all_sync(0xffffffffu, mbar_wait<CG == 2>(&tmem_empty[acc], acc_phase ^ 1, budget, p.status))) { ok = false; break; }
      if constexpr (stamp) cyc_accumulator += clock64() - c_acc;
      tc_fence_after_sync();
      const uint32_t tmem_d = tmem_base + acc * BN;
      for (int kb = 0; kb < t.k_blocks; ++kb) {
        long long c_ops = 0;
        if constexpr (stamp) c_ops = clock64();
        if (!__all_sync(0xffffffffu, mbar_wait<CG == 2>(&full_bar[stage], phase, budget, p.status))) { ok = false; break; }
        if constexpr (stamp) cyc_operands += clock64() - c_ops;
        unsigned char* sa = stage_base + stage * Cfg::kStageBytes;
        unsigned char* sb = sa + Cfg::kABytes;
        if (CG == 1 && p.mode == kVarlenK && t.k_tail != 0 && kb == t.k_blocks - 1) {
          // Rows past the expert's true length hold other data: zero them in both operands
          // (MN-major boxes keep one 128-byte row per k index, so whole rows are cleared).  CG = 2 launches come with
          // operands whose rows up to the next multiple of BK are zero already.
          const int first = t.k_tail;
          constexpr int kBoxes = BM / 64 + Cfg::kBN / 64;
          for (int i = lane; i < kBoxes * (BK - first) * 8; i += 32) {
            const int box = i / ((BK - first) * 8);
            const int r = i - box * ((BK - first) * 8);
            *reinterpret_cast<uint4*>(sa + box * (BK * 128) + (first + r / 8) * 128 + (r % 8) * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
        tc_fence_after_sync();
        if (elect_one()) {
          const uint32_t a_addr = smem_u32(sa), b_addr = smem_u32(sb);
#pragma unroll
          for (int j = 0; j < BK / UMMA_K; ++j) {
            const uint64_t da = A_MN ? umma_smem_desc(a_addr + j * (UMMA_K * 128), BK * 128, 1024)
                                     : umma_smem_desc(a_addr + j * (UMMA_K * 2), 16, 1024);
            const uint64_t db = B_MN ? umma_smem_desc(b_addr + j * (UMMA_K * 128), BK * 128, 1024)
                                     : umma_smem_desc(b_addr + j * (UMMA_K * 2), 16, 1024);
            umma_bf16_ss<CG>(tmem_d, da, db, idesc, (kb > 0 || j > 0) ? 1u : 0u);
          }
          umma_commit<CG>(&empty_bar[stage]);                       // frees the smem stage when the MMAs retire
          if (kb == t.k_blocks - 1) umma_commit<CG>(&tmem_full[acc]);  // accumulator complete
        }
        __syncwarp();
        if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
      }
      acc ^= 1; if (acc == 0) acc_phase ^= 1;
    }
    };
    if (p.timing != nullptr) tile_loop(std::true_type{}); else tile_loop(std::false_type{});
    if (p.timing != nullptr && lane == 0) {
      long long* tm = p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols;
      tm[8] = clock64() - cyc_begin; tm[9] = cyc_operands; tm[10] = cyc_accumulator;
    }
    if (!ok) report_failure(p.status, kStatusTimeoutPipeline, kKernelGemm, 1, p.rank, 0, 0, 0);
    }
  } else if (warp < kGemmWarps) {
    // ------------------------------------------------------------------ epilogue (8 warps: a warp reads the 32 TMEM
    // lanes of its quarter; warps 2..5 take the left half of the tile's columns, warps 6..9 the right half).
    // Results go through a per-warp 4 KB swizzled staging tile so that global memory only ever sees
    // full contiguous row segments: TMA stores for dense outputs, warp-coalesced red.add / st for scatters.
    const int quarter = warp & 3;                 // TMEM lanes this warp may read
    const int row = quarter * 32 + lane;
    const int epi_tid = (warp - 2) * 32 + lane;
    const int half = (warp - 2) >> 2;
    constexpr int kChunksPerHalf = BN / 64;
    const uint32_t stg = smem_u32(epi_stage + (warp - 2) * Cfg::kEpiStageBytes);
    int acc = 0; uint32_t acc_phase = 0;
    for (int it = 0;; ++it) {
      int lin;
      TileCoord t;
      if constexpr (queued) {
        // every epilogue thread reads the queue itself; the give-up decision is taken together (see below)
        const bool got = spin_until([&] { return (leader ? ld_acquire_cta_shared(&s_q_head) : ld_acquire_cluster_shared(&s_q_head)) > it; },
                                    budget, p.status);
        if (epi_vote_any(!got)) break;
        const TileEntry e = s_q[it % kTileQueue];
        lin = e.lin;
        if (lin >= total_tiles) break;
        t = unit_coord<CG>(p, e, half_of_pair);
      } else {
        lin = first_lin + it * lin_stride;
        if (lin >= total_tiles || lin < 0) break;
        t = decode_tile<CG>(p, lin, num_m, half_of_pair);
      }
      const CUtensorMap* to0 = t.prob ? &maps2.o : &tmap_o0;
      // output width of this tile's problem (0: this CTA's half of the pair has no rows)
      const int prob_n = !t.rows_valid ? 0 : t.prob ? p.N2 : p.N;
      const bool empty = (t.k_blocks == 0);
      // Everything that does not need the accumulator is fetched while the tensor cores still work on this tile.
      const int n0 = t.n_tile * BN;
      const int warp_row0 = (p.mode == kVarlenM ? t.row0 : t.m_tile * BM) + quarter * 32;   // TMA y coordinate
      const int zc = (p.mode == kVarlenK) ? t.expert : 0;
      const long long grow = static_cast<long long>(p.mode == kVarlenM ? t.row0 : t.m_tile * BM) + row;
      const int c_begin = half * kChunksPerHalf;
      int tok = 0; float w = 1.f;
      if (EPI == kEpiScatter || EPI == kEpiDswiglu) {
        tok = t.rows_valid ? p.row_token[grow] : -1;
        if (p.row_weight != nullptr && tok >= 0) w = p.row_weight[grow];
      }
      // scatter to other ranks too: where this row goes and how (0 skip, 1 bf16x2 red.add, 2 plain store)
      char* dst_row = nullptr; int op = 0;
      if (EPI == kEpiScatter && p.remote_out.enabled && tok >= 0) {
        const int2 src = p.row_src[grow];
        if (src.x == p.rank) {
          dst_row = static_cast<char*>(p.scatter_local) + static_cast<long long>(src.y) * p.N * 2; op = 1;
        } else {   // the source rank's per-(token, k) row: written once, reduced there in fp32
          dst_row = s_remote_out[src.x] + (static_cast<long long>(src.y) * p.num_topk + p.row_k_slot[grow]) * p.N * 2; op = 2;
        }
      }
      // dSwiGLU reads preact[row, 2n .. 2n+64) per chunk.  A thread-per-row read would touch 32 different lines
      // per instruction, which the load/store unit handles one line at a time; instead 8 lanes fetch one
      // row's 128 bytes (4 full lines per instruction) and the rows are handed to their threads through the
      // staging tile.  pqc = the next chunk in that fetch layout, pq = this thread's row segment.
      uint4 pq[8], pqc[8];
      const char* pre_base = nullptr;
      if (EPI == kEpiDswiglu) {
        pre_base = reinterpret_cast<const char*>(static_cast<const __nv_bfloat16*>(p.preact) +
                                                 static_cast<long long>(warp_row0 + (lane >> 3)) * p.ld_preact) + (lane & 7) * 16;
        const int nf = n0 + c_begin * 32;
        if (nf < prob_n) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            pqc[i] = (2 * nf + (lane & 7) * 8 < 2 * p.N)
                         ? ld_nc_v4(pre_base + static_cast<long long>(i) * 4 * p.ld_preact * 2 + static_cast<long long>(nf) * 4)
                         : make_uint4(0, 0, 0, 0);
        }
      }
      if (!empty) {
        const bool got = mbar_wait(&tmem_full[acc], acc_phase, budget, p.status);
        if (!got) report_failure(p.status, kStatusTimeoutPipeline, kKernelGemm, 2, p.rank, lin, acc, 0);
        // The give-up decision is taken by all 256 epilogue threads together: a thread that saw the accumulator
        // must not go on to the stripe barriers (or to a warp-wide tcgen05.ld) while another one leaves the loop.
        if (epi_vote_any(!got)) break;
        tc_fence_after_sync();
      }
      const uint32_t taddr = tmem_base + acc * BN + (static_cast<uint32_t>(quarter * 32) << 16);
      // The accumulator goes back as soon as this warp has read its last columns (one arrival per warp, on the barrier of the
      // CTA that issues the MMAs), not after they were stored.  With a short reduction the epilogue bounds a tile, and an
      // arrival that releases at cluster scope held every warp until its reductions had been performed.  Y at 32008 rows, hidden 3072, ffn 768: 172 -> 149 us; Y_bwd at
      // 49152 rows, hidden 2048, ffn 1408: 316 -> 267 us.
      const int c_last = min(c_begin + kChunksPerHalf, (prob_n - n0 + 31) / 32) - 1;
      bool given_back = empty;
      auto give_back = [&] {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (CG == 2) mbar_arrive_cluster(cluster_map(&tmem_empty[acc], 0));
          else mbar_arrive(&tmem_empty[acc]);
        }
        given_back = true;
      };
      int row_tok[EPI == kEpiScatter ? 8 : 1];     // tokens of the rows this lane stores (scatter into this GPU only)
      if (EPI == kEpiScatter) {
#pragma unroll
        for (int i = 0; i < (EPI == kEpiScatter ? 8 : 1); ++i) row_tok[i] = __shfl_sync(0xffffffffu, tok, i * 4 + (lane >> 3));
      }
      float dw_acc = 0.f;
#pragma unroll 1
      for (int c = c_begin; c < c_begin + kChunksPerHalf; ++c) {
        const int n = n0 + c * 32;
        if (n >= prob_n) break;
        if (EPI == kEpiDswiglu) {
          // hand this chunk's preact rows to their threads, then request the next chunk (software pipeline)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            st_shared_v4(stg + stage_off<128>(i * 4 + (lane >> 3), lane & 7), pqc[i].x, pqc[i].y, pqc[i].z, pqc[i].w);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) pq[j] = ld_shared_v4(stg + stage_off<128>(lane, j));
          __syncwarp();
          const int nn = n + 32;
          if (c + 1 < c_begin + kChunksPerHalf && nn < p.N) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              pqc[i] = (2 * nn + (lane & 7) * 8 < 2 * p.N)
                           ? ld_nc_v4(pre_base + static_cast<long long>(i) * 4 * p.ld_preact * 2 + static_cast<long long>(nn) * 4)
                           : make_uint4(0, 0, 0, 0);
          }
        }
        uint32_t r[EPI == kEpiDswiglu ? 1 : 32];   // the dSwiGLU epilogue reads the accumulator 16 columns at a time
        if (EPI != kEpiDswiglu) {
          if (!empty) {
            tmem_ld_32x32(taddr + c * 32, reinterpret_cast<uint32_t(&)[32]>(r)); tmem_ld_wait();
            if (c == c_last) give_back();
          } else {
#pragma unroll
            for (int i = 0; i < (EPI == kEpiDswiglu ? 1 : 32); ++i) r[i] = 0;
          }
        }
        // Two chunks side by side leave as one store of 128-byte rows: half the rows for the TMA unit of stores of 32 columns each,
        // two of which fitted the staging tile (weight gradients of 32 x 512, 32 x 1250 and 8 x 6144 rows: 4, 30 and 3 thousand cycles less).
        if (EPI == kEpiStore) {
          if (((c - c_begin) & 1) == 0) {
            if (lane == 0) bulk_wait_read();
            __syncwarp();
          }
        } else if (EPI == kEpiSwiglu) {
          // The staging tile is reused by every chunk: the previous chunk's bulk store must have read it.
          // Waiting here, after the accumulator fetch, instead of right after the store was issued lets the
          // read overlap the TMEM load.
          if (lane == 0) bulk_wait_read();
          __syncwarp();
        }
        if (EPI == kEpiStore) {
          const int hpos = (c - c_begin) & 1;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            st_shared_v4(stg + stage_off<128>(lane, hpos * 4 + q),
                         pack_bf16x2(__uint_as_float(r[q * 8 + 0]), __uint_as_float(r[q * 8 + 1])),
                         pack_bf16x2(__uint_as_float(r[q * 8 + 2]), __uint_as_float(r[q * 8 + 3])),
                         pack_bf16x2(__uint_as_float(r[q * 8 + 4]), __uint_as_float(r[q * 8 + 5])),
                         pack_bf16x2(__uint_as_float(r[q * 8 + 6]), __uint_as_float(r[q * 8 + 7])));
          if (hpos == 1 || n + 32 >= prob_n || c + 1 == c_begin + kChunksPerHalf) {    // (columns past the last are clipped)
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) { tma_store_3d(to0, epi_stage + (warp - 2) * Cfg::kEpiStageBytes, n - hpos * 32, warp_row0, zc); bulk_commit(); }
          }
        } else if (EPI == kEpiSwiglu) {
          // columns (2i, 2i+1) = (gate_i, up_i); preact tile at +0 (64-byte rows), postact tile at +2048 (32-byte rows)
          if (p.out1 != nullptr) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              st_shared_v4(stg + stage_off<64>(lane, q),
                           pack_bf16x2(__uint_as_float(r[q * 8 + 0]), __uint_as_float(r[q * 8 + 1])),
                           pack_bf16x2(__uint_as_float(r[q * 8 + 2]), __uint_as_float(r[q * 8 + 3])),
                           pack_bf16x2(__uint_as_float(r[q * 8 + 4]), __uint_as_float(r[q * 8 + 5])),
                           pack_bf16x2(__uint_as_float(r[q * 8 + 6]), __uint_as_float(r[q * 8 + 7])));
          }
          float a[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float g = __uint_as_float(r[2 * i]), u = __uint_as_float(r[2 * i + 1]);
            a[i] = g * fast_sigmoid(g) * u;
          }
#pragma unroll
          for (int q = 0; q < 2; ++q)
            st_shared_v4(stg + 2048 + stage_off<32>(lane, q), pack_bf16x2(a[q * 8 + 0], a[q * 8 + 1]),
                         pack_bf16x2(a[q * 8 + 2], a[q * 8 + 3]), pack_bf16x2(a[q * 8 + 4], a[q * 8 + 5]),
                         pack_bf16x2(a[q * 8 + 6], a[q * 8 + 7]));
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            unsigned char* sb = epi_stage + (warp - 2) * Cfg::kEpiStageBytes;
            if (p.out1 != nullptr) tma_store_3d(&tmap_o1, sb, n, warp_row0, 0);
            tma_store_3d(&tmap_o0, sb + 2048, n / 2, warp_row0, 0);
            bulk_commit();
          }
        } else if (EPI == kEpiScatter) {
          // Stage two 32-column chunks side by side (128 bytes per row), then let 8 lanes handle one row so
          // that every global access - local red.add or store into a peer's landing row over NVLink - is a
          // full, contiguous 128-byte line of the destination row.
          const int hpos = (c - c_begin) & 1;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            st_shared_v4(stg + stage_off<128>(lane, hpos * 4 + q),
                         pack_bf16x2(w * __uint_as_float(r[q * 8 + 0]), w * __uint_as_float(r[q * 8 + 1])),
                         pack_bf16x2(w * __uint_as_float(r[q * 8 + 2]), w * __uint_as_float(r[q * 8 + 3])),
                         pack_bf16x2(w * __uint_as_float(r[q * 8 + 4]), w * __uint_as_float(r[q * 8 + 5])),
                         pack_bf16x2(w * __uint_as_float(r[q * 8 + 6]), w * __uint_as_float(r[q * 8 + 7])));
          const bool flush = hpos == 1 || n + 32 >= p.N || c + 1 == c_begin + kChunksPerHalf;
          if (flush) {
            __syncwarp();
            const int nbase = n - hpos * 32;
            uint4 vs[8];      // shared-memory reads first: volatile asm keeps program order, see the dSwiGLU branch
#pragma unroll
            for (int i = 0; i < 8; ++i) vs[i] = ld_shared_v4(stg + stage_off<128>(i * 4 + (lane >> 3), lane & 7));
            const int piece = lane & 7, col = nbase + piece * 8;
            const bool mine = piece < (hpos + 1) * 4 && col < p.N;
            if (!p.remote_out.enabled) {
              char* base = static_cast<char*>(p.scatter_local) + static_cast<long long>(col) * 2;
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (mine && row_tok[i] >= 0)
                  red_add_bf16x2_v4(base + static_cast<long long>(row_tok[i]) * p.N * 2, vs[i].x, vs[i].y, vs[i].z, vs[i].w);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int rr = i * 4 + (lane >> 3);
                const uint4 v = vs[i];
                char* ptr = reinterpret_cast<char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst_row), rr));
                const int o = __shfl_sync(0xffffffffu, op, rr);
                if (o != 0 && mine) {
                  if (o == 1) red_add_bf16x2_v4(ptr + static_cast<long long>(col) * 2, v.x, v.y, v.z, v.w);
                  else st_na_v4(ptr + static_cast<long long>(col) * 2, v);
                }
              }
            }
            __syncwarp();
          }
        } else {   // kEpiDswiglu: r = g[row, n..n+32) = dL/d(postact) before the topk weight
          uint32_t o_pw[16];
          unsigned char* sb = epi_stage + (warp - 2) * Cfg::kEpiStageBytes;
          uint32_t rh[16];
#pragma unroll
          for (int q = 0; q < 4; ++q) {       // 8 output columns per step; N is a multiple of 8
            if ((q & 1) == 0) {
              // One 16-column half at a time, fetched where it is used: fetching both halves up front, or the
              // first half before the preact hand-over, costs registers (spills at the 168-register cap of a
              // 10-warp CTA) and measured 7-12 % slower.
              if (!empty) {
                tmem_ld_32x16(taddr + c * 32 + q * 8, rh); tmem_ld_wait();
                if (q == 2 && c == c_last) give_back();
              }
              else {
#pragma unroll
                for (int i = 0; i < 16; ++i) rh[i] = 0;
              }
            }
            uint32_t o_in[8];
            if (tok >= 0 && n + q * 8 < p.N) {
              const uint4 p0 = pq[q * 2], p1 = pq[q * 2 + 1];
              const uint32_t pv[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
              float post[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float2 gu = unpack_bf16x2(pv[i]);          // (gate, up)
                const float g = __uint_as_float(rh[(q & 1) * 8 + i]);
                const float sig = fast_sigmoid(gu.x);
                const float silu = gu.x * sig;
                post[i] = silu * gu.y;
                dw_acc = fmaf(post[i], g, dw_acc);
                const float wg = w * g;
                const float dsilu = sig + fmaf(-sig, silu, silu);   // d silu / d gate = sig + silu * (1 - sig)
                o_in[i] = pack_bf16x2(wg * gu.y * dsilu, wg * silu);
              }
#pragma unroll
              for (int i = 0; i < 4; ++i) o_pw[q * 4 + i] = pack_bf16x2(w * post[2 * i], w * post[2 * i + 1]);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) o_in[i] = 0;
#pragma unroll
              for (int i = 0; i < 4; ++i) o_pw[q * 4 + i] = 0;
            }
            st_shared_v4(stg + stage_off<128>(lane, 2 * q), o_in[0], o_in[1], o_in[2], o_in[3]);
            st_shared_v4(stg + stage_off<128>(lane, 2 * q + 1), o_in[4], o_in[5], o_in[6], o_in[7]);
          }
          // Both outputs leave through the staging tile with plain coalesced stores (8 resp. 4 lanes per
          // 128- resp. 64-byte row segment).  No proxy fence here on purpose: a fence would wait for the
          // preact loads of the next chunk that are still in flight.
          __syncwarp();
          {
            char* din_base = reinterpret_cast<char*>(static_cast<__nv_bfloat16*>(p.out0) + static_cast<long long>(warp_row0) * p.ld0 + 2 * n);
            // all shared-memory reads first, then all global stores: the helpers are volatile asm, which the
            // compiler keeps in program order, so an interleaved loop would wait for every read in turn
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = ld_shared_v4(stg + stage_off<128>(i * 4 + (lane >> 3), lane & 7));
            if (2 * n + (lane & 7) * 8 < 2 * p.N) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                st_global_v4(din_base + static_cast<long long>(i * 4 + (lane >> 3)) * p.ld0 * 2 + (lane & 7) * 16,
                             v[i].x, v[i].y, v[i].z, v[i].w);
            }
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q)
            st_shared_v4(stg + stage_off<64>(lane, q), o_pw[q * 4 + 0], o_pw[q * 4 + 1], o_pw[q * 4 + 2], o_pw[q * 4 + 3]);
          __syncwarp();
          {
            char* pw_base = reinterpret_cast<char*>(static_cast<__nv_bfloat16*>(p.out1) + static_cast<long long>(warp_row0) * p.ld1 + n);
            uint4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = ld_shared_v4(stg + stage_off<64>(i * 8 + (lane >> 2), lane & 3));
            if (n + (lane & 3) * 8 < p.N) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                st_global_v4(pw_base + static_cast<long long>(i * 8 + (lane >> 2)) * p.ld1 * 2 + (lane & 3) * 16,
                             v[i].x, v[i].y, v[i].z, v[i].w);
            }
          }
          __syncwarp();
        }
      }
      if (!given_back) give_back();       // (no column of this tile is this warp's)
      if (!empty) { acc ^= 1; if (acc == 0) acc_phase ^= 1; }
      if (p.timing != nullptr && epi_tid == 0) *reinterpret_cast<volatile int*>(&s_tiles_done) += 1;
      if constexpr (queued) {      // this queue entry may be reused once every epilogue thread is done with the tile
        epi_bar_sync();
        if (epi_tid == 0) {
          if (CG == 2 && !leader) st_release_cluster(cluster_map(&s_q_tail_peer, 0), it + 1);
          else st_release_cta_shared(&s_q_tail, it + 1);
        }
      }
      if (!t.rows_valid) continue;
      if (EPI == kEpiDswiglu) {
        if (tok >= 0 && p.dl_dweight != nullptr) red_add_f32(p.dl_dweight + (p.row_pair != nullptr ? p.row_pair[grow] : grow), dw_acc);
      }
      if ((EPI == kEpiScatter && !p.remote_out.enabled && p.tile_stripes_done != nullptr) ||
          (EPI == kEpiDswiglu && p.remote_dw.enabled)) {
        // Per-M-tile completion: the CTA that finishes the last N stripe of a tile does the
        // per-row bookkeeping once every stripe's writes are visible.
        __threadfence();
        epi_bar_sync();
        if (epi_tid == 0) *s_flag = (atom_add_acq_rel_gpu(p.tile_stripes_done + t.m_tile, 1) == p.num_n_tiles - 1);
        epi_bar_sync();
        const bool last = (*s_flag != 0);
        epi_bar_sync();
        if (last && tok >= 0 && half == 0) {
          if (EPI == kEpiScatter) {
            if (atom_add_acq_rel_gpu(p.k_remaining + tok, -1) == 1) {
              // The stand-alone combine of another GPU acquires this stamp at system scope and then reads the
              // row: the release must be at system scope too (device scope is enough with one rank).
              if (p.num_ranks > 1) { fence_acq_rel_sys(); st_release_sys(p.done_per_token + tok, p.seq); }
              else st_release_gpu(p.done_per_token + tok, p.seq);
            }
          } else {
            const int2 src = p.row_src[grow];
            const float v = *reinterpret_cast<volatile float*>(p.dl_dweight + grow);
            s_remote_dw[src.x][static_cast<long long>(src.y) * p.num_topk + p.row_k_slot[grow]] = v;
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();     // every bulk store this warp issued has been performed
    if (p.tail.enabled) __threadfence_system();
  } else if (warp == kGemmWarps) {
    if constexpr (queued) {
      // ------------------------------------------------------------------ scheduler: tiles into the queue of both CTAs
      if (leader && lane == 0) {
        for (int it = 0;; ++it) {
          // A free entry: every role of both CTAs is done with what it held.  And not too early (kClaimAhead).
          const bool ok = spin_until([&] {
            if (it > ld_acquire_cta_shared(&s_q_prod)) { __nanosleep(128); return false; }      // (seldom: polls take issue slots)
            return it - ld_acquire_cta_shared(&s_q_read) < kTileQueue && it - ld_acquire_cta_shared(&s_q_tail) < kTileQueue &&
                   (CG == 1 || (it - ld_acquire_cluster_shared(&s_q_read_peer) < kTileQueue && it - ld_acquire_cluster_shared(&s_q_tail_peer) < kTileQueue));
          }, budget, p.status);
          int lin = total_tiles;
          if (!ok) report_failure(p.status, kStatusTimeoutPipeline, kKernelGemm, 4, p.rank, it, 0, 0);
          else lin = dyn ? atomicAdd(p.tile_counter, 1) : first_lin + it * lin_stride;
          const bool end = lin >= total_tiles || lin < 0;
          TileEntry e{};
          e.lin = end ? total_tiles : lin;
          if (!end) {
            const TileCoord t = decode_tile<CG>(p, lin, num_m, 0);
            e = TileEntry{lin, t.m_tile, t.n_tile, t.expert, t.row0, t.k_blocks, t.k_tail, t.prob};
          }
          TileEntry* q = &s_q[it % kTileQueue];
          *q = e;
          st_release_cta_shared(&s_q_head, it + 1);
          if (CG == 2) {
            const uint32_t peer = cluster_map(q, 1);
            st_cluster_v4(peer, e.lin, e.m_tile, e.n_tile, e.expert);
            st_cluster_v4(peer + 16, e.row0, e.k_blocks, e.k_tail, e.prob);
            st_release_cluster(cluster_map(&s_q_head, 1), it + 1);
          }
          if (end) break;
        }
      }
    } else if (has_gate_warp(EPI) && lane == 0 && p.mode == kVarlenM && p.arrival_count != nullptr) {
      // ------------------------------------------------------------------ gate warp: polls tile gates ahead of the producer
      const bool local_only = p.num_ranks == 1;   // every writer of the counters is on this GPU: device scope is enough
      int n = 0;
      for (int lin = first_lin; lin < total_tiles; lin += lin_stride) {
        const TileCoord t = decode_tile<CG>(p, lin, num_m, half_of_pair);
        const int target = p.arrival_target[t.m_tile];
        const int* cnt = p.arrival_count + t.m_tile;
        if (!spin_until([&] { return (local_only ? ld_acquire_gpu(cnt) : ld_acquire_sys(cnt)) == target; }, budget, p.status)) {
          report_failure(p.status, kStatusTimeoutTileGate, kKernelGemm, 0, p.rank, t.m_tile, target, ld_acquire_sys(cnt));
          st_release_cta_shared(&s_gates_open, -1);
          break;
        }
        if (p.timing != nullptr) {
          long long* tm = p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols;
          const long long now = static_cast<long long>(globaltimer_ns());
          if (n == 0) tm[2] = now;
        }
        st_release_cta_shared(&s_gates_open, ++n);
      }
    }
  } else if (PUSH) {
    // ------------------------------------------------------------------ dispatch push warps (mixed mode)
    // (with push-only CTAs in the grid these warps either stay idle or, split_local, ship the pairs that stay on
    // this rank: local copies drain fast and do not back up the load/store path)
    const bool local_walker = num_push_ctas > 0 && pp.split_local && pp.work_counter_local != nullptr;
    if ((pp.flags & 2) && (num_push_ctas == 0 || local_walker)) {
      const int pw = warp - base_warps(EPI, A_MN);
      if (pw == 0 && lane < pp.num_ranks) {
        const unsigned long long* rec = pp.static_targets
            ? reinterpret_cast<const unsigned long long*>(&pp.own)
            : fetch_record(pp.peer_base[pp.rank], pp.ctl, pp.kind, pp.epoch, lane,
                           pp.wait_budget_ns, pp.status, kKernelDispatch, pp.rank);
        if (rec == nullptr) s_push_ok = 0;
        else resolve_push_targets(s_tg, lane, pp.peer_base[lane], rec);
      }
      asm volatile("bar.sync 2, %0;" :: "r"(push_warps(EPI) * 32) : "memory");
      if (s_push_ok && (pp.active_push_warps <= 0 || pw < pp.active_push_warps)) {
        const int num_send = *pp.num_send;
        const int num_chunks = push_num_chunks(pp, num_send);
        if (p.timing != nullptr && pw == 0 && lane == 0)
          p.timing[static_cast<size_t>(blockIdx.x) * kTimingCols + 4] = static_cast<long long>(globaltimer_ns());
        for (;;) {
          int chunk = 0;
          if (lane == 0) chunk = atomicAdd(local_walker ? pp.work_counter_local : pp.work_counter, 1);
          chunk = __shfl_sync(0xffffffffu, chunk, 0);
          if (chunk >= num_chunks) break;
          int p0, p1;
          push_chunk_range(pp, num_send, chunk, p0, p1);
          push_chunk(pp, s_tg, p0, p1, lane, nullptr, local_walker ? 1 : 0);
        }
        if (p.timing != nullptr && lane == 0) {
          long long* tm = p.timing + static_cast<size_t>(blockIdx.x) * kTimingCols;
          const unsigned long long now = globaltimer_ns();
          if (atomicMax(reinterpret_cast<unsigned long long*>(tm + 5), now) < now)   // this warp is the CTA's last one so far
            tm[3] = *reinterpret_cast<volatile int*>(&s_tiles_done);
        }
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (CG == 2) cluster_sync();     // neither CTA of a pair leaves (or frees its TMEM) while the other may still reach it
  if (p.timing != nullptr && threadIdx.x == 0)
    p.timing[static_cast<size_t>(blockIdx.x) * kTimingCols + 6] = static_cast<long long>(globaltimer_ns());
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<CG>(tmem_base, Cfg::kTmemCols);
  }
  if (dyn && threadIdx.x == 0) {     // the last CTA puts the claim counter back to zero for the next launch
    __threadfence();
    if (atomicAdd(p.tile_counter + 1, 1) == static_cast<int>(gridDim.x) - 1) { p.tile_counter[0] = 0; p.tile_counter[1] = 0; }
  }
  if (threadIdx.x == 0) {
    int* done_ctr = p.tail.enabled ? p.tail.ctas_done : (PUSH ? pp.blocks_done : nullptr);
    if (done_ctr != nullptr) {
      __threadfence();
      const int old = atomicAdd(done_ctr, 1);
      if (old == static_cast<int>(gridDim.x) - 1) {
        *done_ctr = 0;
        if (PUSH) { *pp.work_counter = 0; if (pp.work_counter_local != nullptr) *pp.work_counter_local = 0; }
        if (p.tail.enabled) {
          // Every CTA's remote reductions were fenced at system scope before it counted itself.
          __threadfence_system();
          for (int r = 0; r < p.num_ranks; ++r)
            flags_signal(p.peer_base, p.ctl, p.tail.kind, p.tail.epoch, p.rank, r);
          if (p.tail.wait)
            for (int r = 0; r < p.num_ranks; ++r)
              if (!flags_wait(p.peer_base[p.rank], p.ctl, p.tail.kind, p.tail.epoch, r,
                              p.wait_budget_ns, p.status, kKernelGemm, p.rank, kStatusTimeoutTail))
                break;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Host side of one instance
// ---------------------------------------------------------------------------------------------
struct LaunchMaps { CUtensorMap a, b, o0, o1; SecondMaps second; };

template <int BN, bool A_MN, bool B_MN, int EPI, bool PUSH, int CG>
cudaError_t launch_instance(const GemmParams& p, const LaunchMaps& m, const PushParams& pp, int num_ctas, cudaStream_t stream) {
  auto kernel = grouped_gemm_kernel<BN, A_MN, B_MN, EPI, PUSH, CG>;
  // The shared-memory limit is an attribute of the function ON A DEVICE: raise it once per device.
  static std::atomic<bool> configured[kMaxDevices];
  const int smem = GemmCfg<BN, CG>::kSmemBytes;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  if (!configured[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((num_ctas + CG - 1) / CG * CG));
  cfg.blockDim = dim3((base_warps(EPI, A_MN) + (PUSH ? push_warps(EPI) : 0)) * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (CG > 1) {
    cudaLaunchAttribute& a = attr[cfg.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = CG; a.val.clusterDim.y = 1; a.val.clusterDim.z = 1;
  }
  if (p.early_start) {
    cudaLaunchAttribute& a = attr[cfg.numAttrs++];
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, m.a, m.b, m.o0, m.o1, p, pp, m.second);
}

// The launchers of one epilogue each (gemm_inst_*.cu, compiled in parallel): `handled` = an instance for this combination
// of tile width, CTA pairing, operand layouts and fused push exists.
cudaError_t launch_swiglu(const GemmParams&, const LaunchMaps&, const PushParams*, int, cudaStream_t, bool& handled);
cudaError_t launch_dswiglu(const GemmParams&, const LaunchMaps&, const PushParams*, int, cudaStream_t, bool& handled);
cudaError_t launch_scatter(const GemmParams&, const LaunchMaps&, const PushParams*, int, cudaStream_t, bool& handled);
cudaError_t launch_store(const GemmParams&, const LaunchMaps&, const PushParams*, int, cudaStream_t, bool& handled);
cudaError_t launch_store_varlen_k(const GemmParams&, const LaunchMaps&, const PushParams*, int, cudaStream_t, bool& handled);

}  // namespace sep
