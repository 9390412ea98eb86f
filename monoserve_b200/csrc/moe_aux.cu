// Routing, planning, packing and combining kernels of one MoE layer.  These
// are HBM/latency-bound integer and byte kernels built on warp primitives; no
// tensor cores.  Their results are defined exactly (see detmath.cuh) so that a
// CPU oracle can be compared bit for bit:
//
//   router_logits   logits[t][e] = sum_h x[t][h] * Wr[e][h]   fp32, fixed order
//   router_topk     softmax / sigmoid(+bias), K rounds of arg-max with the
//                   lowest index winning ties, renormalisation, scale
//                   (csrc/fabric/tiles/aux.cuh:326-417), plus the stable rank of
//                   every (token, pick) pair inside its 32-token chunk
//   plan            per-expert counts, exclusive prefix sums (aux.cuh:423-450),
//                   per-chunk bases, and the grouped-GEMM tile lists chosen
//                   through the layer's (region, slot) table (aux.cuh:453-616)
//   pack            expert-sorted activation rows and pair lists
//                   (aux.cuh:648-684).  The reference orders an expert's rows by
//                   atomic arrival; here the order is fixed: token ascending,
//                   then pick ascending.
//   combine         x[t] = bf16(x2[t] + sum_k w[t][k] * y[pos(t,k)]) in pick
//                   order, optionally followed by the next RMSNorm
//                   (aux.cuh:137-188; the reference sums with fp32 atomics).
#include <cuda_bf16.h>

#include "detmath.cuh"
#include "kernels.h"
#include "peer_sync.cuh"
#include "ptx.cuh"
#include "row_blocks.h"
#include "rowwise.cuh"

namespace mf {

// ------------------------------------------------------------ router logits
// A warp per R tokens x C experts (rowwise.cuh), four expert groups side by side in a block.  The tile is the largest that
// still gives most schedulers a warp: its products per load grow with it, but a decode batch has few of them.
template <int R, int C>
__global__ void __launch_bounds__(128) router_logits_kernel(const bf16* __restrict__ x, const bf16* __restrict__ wr,
                                                            float* __restrict__ logits, int T, int H, int E) {
  chain_release();
  chain_wait();
  const int warp = threadIdx.x >> 5, quads = (E + 4 * C - 1) / (4 * C);
  const int t0 = static_cast<int>(blockIdx.x) / quads * R, e0 = (static_cast<int>(blockIdx.x) % quads * 4 + warp) * C;
  if (t0 < T && e0 < E) router_block<R, C, false>(x, wr, logits, H, E, t0, min(T, t0 + R), e0, min(E, e0 + C));
}

// Many tokens: 16 warps of 4 tokens x 8 experts share 16 tokens x 32 experts, whose columns come 256 at a time through four
// stages of shared memory (each warp loading its own: bound by the latency of those loads, 8192 x 128 x 2048 in 180 us against 145).
constexpr int kStagedTokens = 16, kStagedExperts = 32, kStagedRows = kStagedTokens + kStagedExperts, kStagedDepth = 4;
constexpr int kStagedBytes = kStagedDepth * kStagedRows * 512;

__global__ void __launch_bounds__(512) router_logits_staged_kernel(const bf16* __restrict__ x, const bf16* __restrict__ wr,
                                                                   float* __restrict__ out, int T, int H, int E) {
  extern __shared__ __align__(16) uint8_t staged[];
  chain_release();
  chain_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nj = H / 256, blocks_e = (E + kStagedExperts - 1) / kStagedExperts;
  const int t0 = static_cast<int>(blockIdx.x) / blocks_e * kStagedTokens, e0 = static_cast<int>(blockIdx.x) % blocks_e * kStagedExperts;
  constexpr int kCopies = kStagedRows * 32 / 512;   // 16-byte pieces of a stage per thread: a row per warp and round
  const bf16* from[kCopies];
#pragma unroll
  for (int i = 0; i < kCopies; ++i) {
    const int row = warp + 16 * i;                   // tokens, then experts; those past the end repeat the last
    from[i] = (row < kStagedTokens ? x + static_cast<size_t>(min(t0 + row, T - 1)) * H
                                   : wr + static_cast<size_t>(min(e0 + row - kStagedTokens, E - 1)) * H) + 8 * lane;
  }
  auto stage = [&](int j) {
    if (j < nj) {
#pragma unroll
      for (int i = 0; i < kCopies; ++i) {
        const uint8_t* const to = staged + ((j % kStagedDepth) * kStagedRows + warp + 16 * i) * 512 + lane * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from[i] + 256 * j) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int j = 0; j < kStagedDepth - 1; ++j) stage(j);
  logits::Sums<4, 8> sums;
  for (int j = 0; j < nj; ++j) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStagedDepth - 2) : "memory");
    __syncthreads();   // stage j is there, and stage j - 1 has been read by all
    stage(j + kStagedDepth - 1);
    const uint4* const in = reinterpret_cast<const uint4*>(staged + (j % kStagedDepth) * kStagedRows * 512) + lane;
    logits::Columns<4, 8> k;
#pragma unroll
    for (int r = 0; r < 4; ++r) k.x[r] = in[((warp >> 2) * 4 + r) * 32];
#pragma unroll
    for (int c = 0; c < 8; ++c) k.w[c] = in[(kStagedTokens + (warp & 3) * 8 + c) * 32];
    sums.multiply(k);
  }
  sums.store(out, E, t0 + (warp >> 2) * 4, T, e0 + (warp & 3) * 8, E);
}

template <int R, int C>
static cudaError_t launch_router_tiles(const bf16* x, const bf16* wr, float* logits, int T, int H, int E, cudaStream_t stream) {
  const int blocks = (T + R - 1) / R * ((E + 4 * C - 1) / (4 * C));
  return launch_chained(router_logits_kernel<R, C>, blocks, 128, 0, stream, x, wr, logits, T, H, E);
}

// -------------------------------------------------------------- router top-k
// One block per chunk of 32 tokens, one warp per token.

__device__ __forceinline__ void topk_chunk(const RouterParams& A) {
  __shared__ int s_ids[kChunkTokens * kMaxTopK];
  __shared__ int s_hist[kMaxExperts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = A.E, K = A.K;
  const int r = blockIdx.x * kChunkTokens + warp;
  if (threadIdx.x < kMaxExperts) s_hist[threadIdx.x] = 0;
  if (r < A.T) {
    int my_id;
    float my_w;
    route_row(A.logits + static_cast<size_t>(r) * E, A.bias, E, K, A.scoring, A.renorm, A.scale, A.zero_logits, my_id,
              my_w);
    if (lane < K) {
      A.topk_ids[static_cast<size_t>(r) * K + lane] = my_id;
      A.topk_w[static_cast<size_t>(r) * K + lane] = my_w;
      s_ids[warp * K + lane] = my_id;
    }
  }
  __syncthreads();
  const int rows = min(kChunkTokens, A.T - blockIdx.x * kChunkTokens);
  const int pairs = rows * K;
  if (static_cast<int>(threadIdx.x) < pairs) {
    const int me = s_ids[threadIdx.x];
    int rank = 0;
    for (int q = 0; q < static_cast<int>(threadIdx.x); ++q) rank += s_ids[q] == me;
    if (A.pair_rank) A.pair_rank[static_cast<size_t>(blockIdx.x) * kChunkTokens * K + threadIdx.x] = rank;
    atomicAdd(&s_hist[me], 1);
  }
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < E) {
    const int c = s_hist[threadIdx.x];
    if (A.chunk_counts) A.chunk_counts[static_cast<size_t>(blockIdx.x) * E + threadIdx.x] = c;
    if (A.counts && c) atomicAdd(A.counts + threadIdx.x, c);
  }
}

__global__ void __launch_bounds__(1024) router_topk_kernel(const RouterParams A) {
  chain_release();
  chain_wait();
  topk_chunk(A);
}

// ------------------------------------------------------------- chunk ranks
// The rank step of the stable pack on its own, for routing that was computed
// elsewhere: one block per chunk of 32 tokens; thread p = (token, pick) counts
// the earlier pairs of the chunk that chose the same expert, and the block
// writes the chunk's per-expert pair counts.
// A pair whose expert id lies outside [0, E) is dropped (rank -1, counted nowhere) and
// reported as kErrBadArgs when a status word is given.
__global__ void __launch_bounds__(kChunkTokens * kMaxTopK) chunk_rank_kernel(const int* __restrict__ topk_ids,
                                                                             int* __restrict__ pair_rank,
                                                                             int* __restrict__ chunk_counts,
                                                                             int T, int E, int K, int* status) {
  __shared__ int s_ids[kChunkTokens * kMaxTopK];
  __shared__ int s_hist[kMaxExperts];
  chain_release();
  chain_wait();
  const int rows = min(kChunkTokens, T - static_cast<int>(blockIdx.x) * kChunkTokens);
  const int pairs = rows * K;
  const int p = threadIdx.x;
  const size_t base = static_cast<size_t>(blockIdx.x) * kChunkTokens * K;
  if (p < kMaxExperts) s_hist[p] = 0;
  if (p < pairs) s_ids[p] = topk_ids[base + p];
  __syncthreads();
  if (p < pairs) {
    const int me = s_ids[p];
    if (me >= 0 && me < E) {
      int rank = 0;
      for (int q = 0; q < p; ++q) rank += s_ids[q] == me;
      pair_rank[base + p] = rank;
      atomicAdd(&s_hist[me], 1);
    } else {
      pair_rank[base + p] = -1;
      if (status) atomicOr(status, kErrBadArgs);
    }
  }
  __syncthreads();
  for (int e = p; e < E; e += blockDim.x) chunk_counts[static_cast<size_t>(blockIdx.x) * E + e] = s_hist[e];
}

// ---------------------------------------------------------------------- plan

// Exclusive scan of one int per thread over the block's first 256 threads (the others' values are not counted); returns the
// exclusive prefix and writes the total.
__device__ __forceinline__ int block_scan_256(int v, int* s_warp, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();
  if (lane == 31 && warp < 8) s_warp[warp] = incl;
  __syncthreads();
  int base = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const int s = s_warp[w];
    if (w < warp) base += s;
    total += s;
  }
  return base + incl - v;
}

// One block, bound by its chain of dependent steps.  1024 threads: a quarter of the chunks each while the chunk counts are
// summed (16 loads in flight; one thread per expert walking 256 chunks one load at a time: 75 us against 30), and 32 warps for
// the tile lists.
constexpr int kPlanThreads = 1024, kPlanParts = kPlanThreads / kMaxExperts;

__device__ __forceinline__ void make_plan(const PlanParams& A) {
  __shared__ int s_warp[8];
  const int e = threadIdx.x;
  const int E = A.E;
  int cnt = 0;
  bool bad = false;
  if (e < E && A.seg_counts) {
    const int tables = A.seg_tables > 0 ? A.seg_tables : 1;
    for (int i = 0; i < tables; ++i) {
      const int c = A.seg_counts[static_cast<size_t>(i) * A.seg_stride + e];
      bad |= c < 0;
      cnt += c;
    }
    if (bad) cnt = 0;
    A.counts[e] = cnt;
  } else if (!A.seg_counts) {
    __shared__ int s_part[kPlanParts][kMaxExperts];
    const int x = e % kMaxExperts, part = e / kMaxExperts, per = (A.chunks + kPlanParts - 1) / kPlanParts;
    const int c_lo = min(part * per, A.chunks), c_hi = min(c_lo + per, A.chunks);
    auto each = [&](auto&& f) {   // f(chunk's count of expert x, its cell), chunks in order
      if (x >= E) return;
      for (int c0 = c_lo; c0 < c_hi; c0 += 16) {
        int v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = c0 + i < c_hi ? __ldcg(A.chunk_counts + static_cast<size_t>(c0 + i) * E + x) : 0;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c0 + i < c_hi) f(v[i], A.chunk_counts + static_cast<size_t>(c0 + i) * E + x);
      }
    };
    int sum = 0;
    each([&](int v, int*) { sum += v; });
    s_part[part][x] = sum;
    __syncthreads();
    int run = 0;
    for (int q = 0; q < part; ++q) run += s_part[q][x];
    each([&](int v, int* cell) {
      *cell = run;
      run += v;
    });
    if (e < E) {
      for (int q = 0; q < kPlanParts; ++q) cnt += s_part[q][e];
      A.counts[e] = cnt;
      if (A.hist) A.hist[e] += cnt;
    }
  }
  int total;
  const int start = block_scan_256(cnt, s_warp, total);
  if (e < E) A.starts[e] = start;
  if (e == 0) A.starts[E] = total;

  if (!A.q) return;   // scan only: counts, starts and chunk prefixes
  // Row blocks of an expert in HBM.  bf16 weights: one of up to 64 rows, or "wide" ones with tiles of two weight slices (row_blocks.h).  e4m3 weights: of 256 rows and tiles of one slice, which
  // read and expand the slice once where two blocks of 128 rows do it twice, with two stages of 96 KB in the ring instead of three of
  // 64 (4096 x 1408, blocks of 128 -> 256 rows: 2048 tokens 1284 -> 1271 us, with a Zipf-skewed choice of experts 1378 -> 1260;
  // 1000 tokens 818 -> 821, the same).
  int tier = kTierHot, z = 0, bh = 256, nb = 0;
  RowBlocks wide_blocks{0, 0, 0};
  const int expert = (e < E && A.seg_expert) ? A.seg_expert[e] : e;
  // A segment of an expert the table does not hold, a negative count or more rows than the packed-row
  // buffers take: no tile is emitted and the layer reports a plan overflow.
  bad |= e < E && cnt > 0 && (expert < 0 || expert >= A.n_experts);
  const bool refuse = __syncthreads_or(bad) || total > A.rows_cap;
  if (e < E && cnt > 0 && !refuse) {
    tier = A.table[2 * expert] == 0 ? kTierHost : kTierHot;
    z = A.table[2 * expert + 1];
    if (tier == kTierHost) bh = A.form ? A.form : 256;
    else if (A.slices > 1) wide_blocks = row_blocks(cnt, total);
    nb = wide_blocks.n ? wide_blocks.n + (wide_blocks.rest > 0) : (cnt + bh - 1) / bh;
  }
  const int nw = wide_blocks.n;
  const int f13 = (A.I + 63) / 64, f2 = (A.H + 127) / 128;
  const int h13 = (f13 + 1) / 2, h2 = (f2 + 1) / 2;   // tiles of a wide block
  // per tier: [w13 tiles of every expert][w2 tiles of every expert]; row blocks numbered over all experts
  int first13[2], first2[2], total13[2], total2[2], blocks_total;
  const int block0 = block_scan_256(nb, s_warp, blocks_total);
  for (int tq = 0; tq < 2; ++tq) {
    const int wide = tier == tq ? nw : 0, narrow = tier == tq ? nb - nw : 0;
    first13[tq] = block_scan_256(wide * h13 + narrow * f13, s_warp, total13[tq]);
    first2[tq] = block_scan_256(wide * h2 + narrow * f2, s_warp, total2[tq]);
  }
  bool overflow = refuse || blocks_total > A.block_cap;
  for (int tq = 0; tq < 2; ++tq) overflow |= total13[tq] + total2[tq] > A.tile_cap;
  for (int b = e; b < blocks_total && !overflow; b += blockDim.x) A.done[b] = 0;
  if (e == 0) {
    for (int tq = 0; tq < 2; ++tq) {
      A.q->n_tiles[tq] = overflow ? 0 : total13[tq] + total2[tq];
      A.q->head[tq] = 0;
    }
    A.q->slots = 0;
    A.q->n_blocks = blocks_total;
    A.q->need = 4 * f13;   // four epilogue warps arrive per w13 slice
    if (overflow) atomicOr(A.status, kErrPlanOverflow);
  }
  // Every expert's tile list is written by a warp, a tile per lane (an expert at decode batch sizes has
  // 28 tiles; written from one thread per expert they were the longest serial stretch of the layer).
  __shared__ int s_job[kMaxExperts][8];   // nb, bh, rows, first row, slot, tier, first w13 tile, first w2 tile (+ block0 below)
  __shared__ int s_block0[kMaxExperts], s_expert[kMaxExperts];
  __shared__ RowBlocks s_wide[kMaxExperts];
  if (e < E) {
    s_job[e][0] = overflow ? 0 : nb;
    s_job[e][1] = bh;
    s_job[e][2] = cnt;
    s_job[e][3] = start;
    s_job[e][4] = z;
    s_job[e][5] = tier;
    s_job[e][6] = first13[tier];
    s_job[e][7] = total13[tier] + first2[tier];
    s_block0[e] = block0;
    s_expert[e] = expert;
    s_wide[e] = wide_blocks;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int x = warp; x < E; x += static_cast<int>(blockDim.x >> 5)) {
    const int x_nb = s_job[x][0];
    if (x_nb == 0) continue;
    const int x_bh = s_job[x][1], x_cnt = s_job[x][2], x_start = s_job[x][3], x_tier = s_job[x][5];
    const RowBlocks x_wide = s_wide[x];
    GemmTile* const list = A.tiles[x_tier];
    const int x_nw = x_wide.n, n13 = x_nw * h13 + (x_nb - x_nw) * f13, n2 = x_nw * h2 + (x_nb - x_nw) * f2;
    for (int j = lane; j < n13 + n2; j += 32) {
      const bool up = j >= n13;   // a w2 tile
      const int jj = up ? j - n13 : j, per = up ? f2 : f13, half = up ? h2 : h13;
      const bool wide = jj < x_nw * half;
      const int past = jj - x_nw * half;   // among the tiles of one slice
      // wide blocks: those of a weight slice are neighbours in the list, so that they read it at about the same time
      const int b = wide ? jj % x_nw : x_nw + past / per, f = wide ? 2 * (jj / x_nw) : past % per;   // f: first slice
      const int first = x_nw ? row_block_first(x_wide, b) : b * x_bh;
      const int rows = x_nw ? row_block_rows(x_wide, b, x_cnt) : min(x_bh, x_cnt - first);
      int n = 16;
      while (n < rows) n <<= 1;
      GemmTile t;
      t.w_row0 = up ? f * 128 : f * 64;
      t.act_row0 = x_start + first;
      t.rows = rows;
      t.n = n;
      t.z = s_job[x][4];
      t.tier_phase = x_tier | (up ? 1 << 8 : 0) | ((wide && f + 1 < per ? 2 : 1) << 16);
      t.expert = s_expert[x];
      t.block = s_block0[x] + b;
      list[(up ? s_job[x][7] : s_job[x][6]) + jj] = t;
    }
  }
}

__global__ void __launch_bounds__(kPlanThreads) plan_kernel(const PlanParams A) {
  chain_release();
  chain_wait();
  if (A.wait_flags) {   // expert parallelism: the counts and the rows they describe come from peers
    if (static_cast<int>(threadIdx.x) < A.wait_n && !wait_flag(A.wait_flags + threadIdx.x, A.wait_epoch)) atomicOr(A.status, kErrWaitTimeout);
    __syncthreads();
  }
  make_plan(A);
}

// ---------------------------------------------------------------------- pack

// Token t by one warp.
__device__ __forceinline__ void pack_token(const PackParams& A, int t) {
  const int lane = threadIdx.x & 31;
  const int K = A.K;
  int pos = -1;   // stays -1 for a pair whose expert id is outside [0, E): it is dropped
  if (lane < K) {
    const int e = A.topk_ids[static_cast<size_t>(t) * K + lane];
    if (e >= 0 && e < A.E) {
      pos = A.starts[e] + A.chunk_prefix[static_cast<size_t>(t / kChunkTokens) * A.E + e] +
            A.pair_rank[static_cast<size_t>(t) * K + lane];
      A.pair_token[pos] = t;
      A.pair_weight[pos] = A.topk_w[static_cast<size_t>(t) * K + lane];
    } else if (A.status) {
      atomicOr(A.status, kErrBadArgs);
    }
    A.pair_pos[static_cast<size_t>(t) * K + lane] = pos;
  }
  if (!A.src) return;   // pair lists only
  const uint4* src = reinterpret_cast<const uint4*>(A.src + static_cast<size_t>(t) * A.H);
  const int n16 = A.H / 8;
  for (int c0 = 0; c0 < n16; c0 += 32 * 8) {
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + 32 * i + lane < n16) v[i] = src[c0 + 32 * i + lane];
    for (int k = 0; k < K; ++k) {
      const int pk = __shfl_sync(0xffffffffu, pos, k);
      if (pk < 0) continue;
      uint4* dst = reinterpret_cast<uint4*>(A.dst + static_cast<size_t>(pk) * A.H);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + 32 * i + lane < n16) dst[c0 + 32 * i + lane] = v[i];
    }
  }
}

__global__ void __launch_bounds__(256) pack_kernel(const PackParams A) {
  chain_release();
  chain_wait();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t < A.T) pack_token(A, t);
}

// Top-k, plan and, for a few tokens, pack in one launch, for up to two chunks of tokens: the block that counts its chunk last
// makes the plan, and packs the rows when one SM copies them in less time than a launch takes.  (One token 42.3 -> 41.3 us a layer,
// 64 tokens of the e4m3 layer 561 -> 554; 256 tokens, eight blocks, 178 -> 181, so they keep the launches apart.)
constexpr int kPackTokens = 4, kRouteChunks = 2;
__global__ void __launch_bounds__(kPlanThreads) route_kernel(const RouterParams R, const PlanParams P, const PackParams K) {
  __shared__ int s_last;
  chain_release();
  chain_wait();
  topk_chunk(R);
  if (gridDim.x > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(&P.q->routed, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
  } else {
    __syncthreads();
  }
  make_plan(P);
  if (R.T > kPackTokens) return;
  __syncthreads();
  if (static_cast<int>(threadIdx.x >> 5) < R.T) pack_token(K, threadIdx.x >> 5);
}

// ------------------------------------------------------------------- combine

// Warps per token when no row reduction follows: four, and for batches that leave the schedulers idle (kFew) one per 256 columns.
// There a warp's chain of loads is what it takes; where warps are many, four rows' loads in each cost registers and 1 % (8192
// tokens).  64 tokens of 4096 columns, with the projection's smaller tiles: the layer 638 -> 626 us.
constexpr int kFewTokens = 74;   // four warps a token leave every other scheduler (4 x 148) without one
__host__ __device__ __forceinline__ int combine_split(int H, bool norm, bool few) { return norm ? 1 : few ? max(4, H / 256) : 4; }

template <bool kFew>
__global__ void __launch_bounds__(256) combine_kernel(const CombineParams A) {
  // Without the fused RMSNorm a row needs no reduction, so several warps share a token's columns:
  // a decode batch of a few hundred tokens otherwise leaves most of the machine idle.  Every column is
  // computed by the same instructions either way: the result does not depend on the split.
  const int lane = threadIdx.x & 31;
  chain_release();
  chain_wait();
  if (A.wait_flags) {   // expert parallelism: y is written by peers
    if (static_cast<int>(threadIdx.x) < A.wait_n && !wait_flag(A.wait_flags + threadIdx.x, A.wait_epoch))
      atomicOr(A.status, kErrWaitTimeout);
    __syncthreads();
  }
  const int split = combine_split(A.H, A.norm_w != nullptr, kFew);
  const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int t = unit / split, part = unit - t * split;
  if (t >= A.T) return;
  const int K = A.K, H = A.H, n16 = H / 8;
  const int c_begin = part * n16 / split, c_end = (part + 1) * n16 / split;
  int pos = 0;
  float w = 0.f;
  if (lane < K) {
    pos = A.pair_pos[static_cast<size_t>(t) * K + lane];
    w = A.topk_w[static_cast<size_t>(t) * K + lane];
  }
  const uint4* x2 = A.x2 ? reinterpret_cast<const uint4*>(A.x2 + static_cast<size_t>(t) * H) : nullptr;
  uint4* xo = reinterpret_cast<uint4*>(A.x + static_cast<size_t>(t) * H);
  float ss = 0.f;
  // Same trip count in every lane: the shuffles inside need the whole warp.  A lane past the end of its
  // part goes through the motions on the part's last column and neither stores nor counts it.
  for (int c0 = c_begin; c0 < c_end; c0 += 32) {
    const int c = min(c0 + lane, c_end - 1);
    const bool on = c0 + lane < c_end;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    if constexpr (kFew) {   // four expert rows' loads are issued before the first is used
      for (int k0 = 0; k0 < K; k0 += 4) {
        float4 a[4], b[4];
        bool there[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int pk = __shfl_sync(0xffffffffu, pos, min(k0 + i, K - 1));
          there[i] = k0 + i < K && pk >= 0 && !(A.y_rows && pk >= A.y_rows);   // a dropped pair adds nothing
          const float4* yr = reinterpret_cast<const float4*>(A.y + static_cast<size_t>(there[i] ? pk : 0) * H) + 2 * c;
          if (there[i]) {
            a[i] = __ldcs(yr);
            b[i] = __ldcs(yr + 1);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float wk = __shfl_sync(0xffffffffu, w, min(k0 + i, K - 1));
          if (!there[i]) continue;
          acc[0] = __fmaf_rn(wk, a[i].x, acc[0]);
          acc[1] = __fmaf_rn(wk, a[i].y, acc[1]);
          acc[2] = __fmaf_rn(wk, a[i].z, acc[2]);
          acc[3] = __fmaf_rn(wk, a[i].w, acc[3]);
          acc[4] = __fmaf_rn(wk, b[i].x, acc[4]);
          acc[5] = __fmaf_rn(wk, b[i].y, acc[5]);
          acc[6] = __fmaf_rn(wk, b[i].z, acc[6]);
          acc[7] = __fmaf_rn(wk, b[i].w, acc[7]);
        }
      }
    } else {
      for (int k = 0; k < K; ++k) {
        const int pk = __shfl_sync(0xffffffffu, pos, k);
        const float wk = __shfl_sync(0xffffffffu, w, k);
        if (pk < 0 || (A.y_rows && pk >= A.y_rows)) continue;   // a dropped pair adds nothing
        const float4* yr = reinterpret_cast<const float4*>(A.y + static_cast<size_t>(pk) * H) + 2 * c;
        const float4 a = __ldcs(yr), b = __ldcs(yr + 1);
        acc[0] = __fmaf_rn(wk, a.x, acc[0]);
        acc[1] = __fmaf_rn(wk, a.y, acc[1]);
        acc[2] = __fmaf_rn(wk, a.z, acc[2]);
        acc[3] = __fmaf_rn(wk, a.w, acc[3]);
        acc[4] = __fmaf_rn(wk, b.x, acc[4]);
        acc[5] = __fmaf_rn(wk, b.y, acc[5]);
        acc[6] = __fmaf_rn(wk, b.z, acc[6]);
        acc[7] = __fmaf_rn(wk, b.w, acc[7]);
      }
    }
    float f[8];
    if (x2) {
      unpack8(x2[c], f);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f[j] = round_bf16(__fadd_rn(f[j], acc[j]));
      if (on) ss = __fmaf_rn(f[j], f[j], ss);
    }
    if (on) xo[c] = pack8(f);
  }
  if (!A.norm_w) return;
  norm_store_row(xo, ss, A.norm_w, A.normed + static_cast<size_t>(t) * H, nullptr, H, A.eps);
}

// ------------------------------------------------------------------ launchers
cudaError_t launch_router_logits(const void* x, const void* wr, float* logits, int T, int H, int E,
                                 cudaStream_t stream) {
  if (T == 0) return cudaSuccess;
  const bf16* xb = static_cast<const bf16*>(x);
  const bf16* wb = static_cast<const bf16*>(wr);
  constexpr long long kWarps = 4 * 148;
  const long long n = static_cast<long long>(T) * E;
  if (n >= 32 * 4 * kWarps) {   // a block of 16 warps for every SM
    static PerDeviceOnce once;
    const cudaError_t err = once.run([] {
      return cudaFuncSetAttribute(router_logits_staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStagedBytes);
    });
    if (err != cudaSuccess) return err;
    const int blocks = (T + kStagedTokens - 1) / kStagedTokens * ((E + kStagedExperts - 1) / kStagedExperts);
    return launch_chained(router_logits_staged_kernel, blocks, 512, kStagedBytes, stream, xb, wb, logits, T, H, E);
  }
  if (n >= 32 * kWarps) return launch_router_tiles<4, 8>(xb, wb, logits, T, H, E, stream);
  if (n >= 8 * kWarps) return launch_router_tiles<2, 4>(xb, wb, logits, T, H, E, stream);
  return launch_router_tiles<1, 1>(xb, wb, logits, T, H, E, stream);
}

cudaError_t launch_router_topk(const RouterParams& A, cudaStream_t stream) {
  if (A.T == 0) return cudaSuccess;
  return launch_chained(router_topk_kernel, (A.T + kChunkTokens - 1) / kChunkTokens, 1024, 0, stream, A);
}

cudaError_t launch_chunk_rank(const int* topk_ids, int* pair_rank, int* chunk_counts, int T, int E, int K,
                              int* status, cudaStream_t stream) {
  if (T == 0) return cudaSuccess;
  return launch_chained(chunk_rank_kernel, (T + kChunkTokens - 1) / kChunkTokens, kChunkTokens * kMaxTopK, 0, stream,
                        topk_ids, pair_rank, chunk_counts, T, E, K, status);
}

cudaError_t launch_plan(const PlanParams& A, cudaStream_t stream) {
  return launch_chained(plan_kernel, 1, kPlanThreads, 0, stream, A);
}

cudaError_t launch_route(const RouterParams& R, const PlanParams& P, const PackParams& K, cudaStream_t stream) {
  if (R.T == 0) return cudaSuccess;
  return launch_chained(route_kernel, (R.T + kChunkTokens - 1) / kChunkTokens, kPlanThreads, 0, stream, R, P, K);
}

bool route_in_one(int T) { return T <= kRouteChunks * kChunkTokens; }
bool route_packs(int T) { return T <= kPackTokens; }

cudaError_t launch_pack(const PackParams& A, cudaStream_t stream) {
  if (A.T == 0) return cudaSuccess;
  return launch_chained(pack_kernel, (A.T + 7) / 8, 256, 0, stream, A);
}

size_t pack_scratch_bytes(int T, int E, int K) {
  const size_t chunks = (static_cast<size_t>(T) + kChunkTokens - 1) / kChunkTokens;
  return chunks * E * sizeof(int) + static_cast<size_t>(T) * K * sizeof(int);
}

cudaError_t launch_pack_chain(const int* topk_ids, const float* topk_w, int T, int E, int K, int H, const bf16* src,
                              bf16* dst, int* counts, int* starts, int* pair_token, float* pair_weight,
                              int* pair_pos, void* scratch, int* status, cudaStream_t stream) {
  const int chunks = (T + kChunkTokens - 1) / kChunkTokens;
  int* chunk_counts = static_cast<int*>(scratch);
  int* pair_rank = chunk_counts + static_cast<size_t>(chunks) * E;
  cudaError_t err = launch_chunk_rank(topk_ids, pair_rank, chunk_counts, T, E, K, status, stream);
  if (err != cudaSuccess) return err;
  PlanParams pp{};
  pp.chunk_counts = chunk_counts;
  pp.counts = counts;
  pp.starts = starts;
  pp.chunks = chunks;
  pp.E = E;
  pp.n_experts = E;
  err = launch_plan(pp, stream);
  if (err != cudaSuccess) return err;
  PackParams kp{topk_ids, topk_w, pair_rank, chunk_counts, starts, src, dst, pair_token, pair_weight, pair_pos,
                T, E, K, H, status};
  return launch_pack(kp, stream);
}

cudaError_t launch_combine(const CombineParams& A, cudaStream_t stream) {
  if (A.T == 0) return cudaSuccess;
  const bool few = A.T <= kFewTokens;
  const int units = A.T * combine_split(A.H, A.norm_w != nullptr, few);
  return launch_chained(few ? combine_kernel<true> : combine_kernel<false>, (units + 7) / 8, 256, 0, stream, A);
}

}  // namespace mf
