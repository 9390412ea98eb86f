// The weight x activation GEMM tile on tcgen05 / TMEM / TMA, as three warp-role
// device functions shared by the stand-alone grouped expert GEMM kernel and by
// the persistent fabric worker.
//
// One tile (the reference's GEMM tile, csrc/fabric/tiles/gemm.cuh:1-18,133-346,
// csrc/fabric/model_types.h:37-49): 128 weight rows (output features) as the MMA
// M operand times up to 256 activation rows as the N operand, over a range of
// 64-element K steps; fp32 accumulation in TMEM.  Tiles of at least 128 activation rows swap
// the operands (takes_rows): rows on M, 128 or, of two slices, 256 weight rows on N.  Both operands are K-major with
// the 128-byte swizzle.  A weight slice is one TMA box of 128 rows, or eight of 16
// rows, which interleave the 64 gate rows and 64 up rows of a SwiGLU tile in groups
// of 16: TMEM lane 32q+i (i < 16) then holds gate feature 16q+i and lane 32q+16+i
// the matching up feature, so the epilogue pairs them with a warp shuffle instead
// of a trip through shared memory (with the rows on M they are columns of one lane).
//
// What bounds the products of prompts: with all SMs at it, the operands.  8192 tokens over 128 experts, hidden 2048, width 768, cut into
// tiles of 128 x 256 only: 997 K steps a CTA in 880 thousand cycles, 880 a step, of which the MMAs are 512 and the MMA warp waits for
// operands (48 KB a step) 300; in tiles of 256 x 256 (64 KB a step) 605 K steps of 1024 cycles of MMA take 890 thousand,
// the rest in epilogues that nothing hides, under the power cap (1.47 GHz).  In the way before were the producer's loop (a stage by itself 770
// cycles, now 550; a small tile's two K steps a stage, 650 a step, now 310), weights evicted from the L2 before their other row
// blocks read them, and an epilogue of 13000 cycles a 256 x 256 tile.  4096 x 12288 x 2048: 221 -> 159 us a stage of the fabric; those
// experts and all around them: 1180 -> 1108 us a layer, with the row blocks of row_blocks.h 1010.
//
// Roles: produce() runs in one warp (an elected lane issues TMA), mma() in one warp (one lane
// issues tcgen05.mma / tcgen05.commit), epilogue() in the four warps whose
// warp index modulo 4 covers the four TMEM lane quadrants.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <type_traits>

#include "ptx.cuh"
#include "types.h"

namespace mf {

constexpr int kBlockK = 64;                      // elements per K step (128 bytes of bf16)
constexpr int kATileBytes = 128 * kBlockK * 2;   // 16 KB
constexpr int kGemmMaxN = 256;
// Operand stages live in one byte ring: a stage takes 16 KB for the weight tile
// plus n * 128 bytes for the activation tile a K step: five stages of two K steps of a decode tile of 16 rows, four of 64 rows and of
// 128 x 256, three of 256 x 256; six of 32 KB at most.  Twelve barrier pairs: a stage's pair has long been let go when its turn comes.
constexpr int kGemmStages = 12;
static_assert(kRingBytes / (32 * 1024) < kGemmStages, "barrier pairs are never what a stage waits for");
constexpr int kGemmSmemBytes = kRingBytes + kOutBytes + 1024;
constexpr int kTmemCols = 512;
constexpr int kAccCols = 256;                    // TMEM columns per accumulator buffer (two buffers)
constexpr unsigned long long kWaitBudgetNs = 4000000000ull;   // 4 s of device time per wait

// Epilogues (csrc/fabric/model_types.h:29-35).
constexpr int kEpiStoreBf16 = 0;   // out[m][n] = bf16(acc (+ bias[n]) (+ residual[m][n]))
constexpr int kEpiSiluMul = 1;     // 64 gate + 64 up rows: out[m][f] = bf16(silu(g) * u)
constexpr int kEpiWeightedAdd = 2;  // out32[pair_token[m]][n] += pair_weight[m] * acc (fp32 atomics, arrival order)
constexpr int kEpiStoreF32 = 3;    // out32[m][n] = acc (+ bias[n])
constexpr int kEpiAtomicF32 = 4;   // out32[m][n] += acc : K-split partial sums
constexpr int kEpiRowsF32 = 5;     // out32[m][n] = acc : per-pair rows for the deterministic combine (not in the reference)
constexpr int kEpiGeluMul = 6;     // as kEpiSiluMul with the tanh form of gelu on the gate (not in the reference)
constexpr int kEpiDecay = 7;       // out32[m][n] = expm1(-coef[n] softplus(acc + bias[n])), coef in pair_weight (not in the reference)
// A tile of 64 gate and 64 up rows whose epilogue multiplies act(gate) by up.
__host__ __device__ __forceinline__ bool epi_gated(int epi) { return epi == kEpiSiluMul || epi == kEpiGeluMul; }

// Everything the three roles need to know about one tile; lives in shared memory.
struct GemmWork {
  const CUtensorMap* a_map;   // weights: dims (K, rows, Z); box (64, 16, 1) for SwiGLU tiles, else (64, 128, 1)
  const CUtensorMap* b_map;   // activations: dims (K, rows), box (64, n)
  void* out;
  const float* scale;         // fp32 per weight row (FP8 weights), or null
  const __nv_bfloat16* bias;      // per output feature, or null
  const __nv_bfloat16* residual;  // [rows][ld_res], or null
  const int32_t* pair_token;      // kEpiWeightedAdd: token of every activation row
  const float* pair_weight;       // kEpiWeightedAdd: routing weight of every activation row
  int32_t a_row_lo;           // first weight row
  int32_t a_row_hi;           // kEpiSiluMul: first up row; otherwise ignored
  int32_t a_z;
  int32_t b_row0;             // first activation row
  int32_t rows;               // valid activation rows (<= n)
  int32_t n;                  // MMA N: 16, 32, 64, 128 or 256
  int32_t k0, k_tiles;        // K steps [k0, k0 + k_tiles)
  int32_t epi;
  int32_t ld_out, ld_res;
  int32_t n_limit;            // valid output features
  int32_t valid;              // 0: no tile (the consumer roles stop or skip)
  int32_t a_packed;           // bit 0 (two slabs): the weight rows are already interleaved in memory (one 128-row box);
                              // bit 2: two slabs (64 rows at a_row_lo, 64 at a_row_hi) under kEpiAtomicF32, whose
                              // partial sums go to column = weight row (kEpiSiluMul always reads two slabs)
  int32_t block;              // row block whose counter the epilogue bumps, or -1
  int32_t w_fp8;              // the weight tensor holds e4m3 bytes: W8A16 (exact e4m3 -> bf16 in shared memory)
  int32_t slices;             // 1, or 2: two adjacent weight slices (bf16 weights, no epilogue that adds)
  int32_t by_rows;            // the activation rows are the MMA's M dimension: an accumulator holds 128 of them times the
                              // weight rows (takes_rows); otherwise 128 weight rows times the n activation rows
  // A fetch record moves fetch_bytes from fetch_src (host-resident weights) to `out` (an HBM staging
  // buffer) through the operand ring, in stages of kFetchStageBytes: no MMA, no accumulator.
  int32_t fetch;
  uint32_t fetch_bytes;
  const uint8_t* fetch_src;
};

struct GemmPipe {   // a role's cursor over the stage ring; producer and MMA warp replay the same sequence
  uint32_t vwr = 0;     // virtual write position in bytes (wraps modulo 2^32; only differences are used)
  uint32_t phys = 0;    // ring offset of the next stage
  uint32_t slot = 0;    // barrier pair of the next stage
  uint32_t parity = 0;  // parity of that pair's current use
  uint32_t i = 0;       // stages allocated so far
  // MMA role: one bit per barrier pair = parity of the pair's converter barrier.  That barrier
  // completes a phase only for stages with e4m3 weights, so when bf16 and e4m3 tiles share the
  // ring its parity is not a function of the stage's position, unlike full / empty.
  uint32_t conv_bits = 0;
  // Next stage of `size` bytes (a multiple of 1024): its offset in the ring, and
  // the virtual interval it covers (including a skipped tail when it wraps).
  __device__ __forceinline__ uint32_t alloc(uint32_t size, uint32_t& vbegin, uint32_t& vend) {
    vbegin = vwr;
    if (phys + size > kRingBytes) {
      vwr += kRingBytes - phys;
      phys = 0;
    }
    const uint32_t at = phys;
    phys += size;
    vwr += size;
    vend = vwr;
    return at;
  }
  __device__ __forceinline__ void advance() {
    ++i;
    if (++slot == kGemmStages) {
      slot = 0;
      parity ^= 1;
    }
  }
};

// Producer-only bookkeeping of the stages in flight, the same in every lane but for vbegin.
struct GemmInflight {
  uint32_t vbegin = 0;        // lane i: where the stage of barrier pair i begins (an array indexed by the pair would live in local memory)
  uint32_t tail_vbegin = 0;   // of the oldest
  uint32_t tail = 0;          // oldest stage not yet known to be consumed
  uint32_t tail_slot = 0;
  uint32_t tail_parity = 0;
};

// Which tiles put the activation rows on the MMA's M dimension (TMEM lanes): those of at least 128 rows whose epilogue stores,
// of bf16 weights.  A lane then owns a row of the output and stores its 32 columns as whole 32-byte sectors, and gate and up of
// a feature lie in one lane; with the weights on M a warp's store covers one feature of 32 lanes, 2 bytes each, and a
// 256-column accumulator took 6500 to 8600 cycles to drain, more than half of it exposed behind the MMAs of a tile of two
// accumulators (they fill TMEM).  Fewer than 128 rows would leave MMA rows empty, e4m3 weights bring a scale per column, and
// the adding epilogues are for small tiles.
__host__ __device__ __forceinline__ bool takes_rows(int n, int epi, bool w_fp8, bool scaled) {
  return n >= 128 && !w_fp8 && !scaled && epi != kEpiWeightedAdd && epi != kEpiAtomicF32;
}
// Accumulators a tile uses, one after the other; rows past the end of the last block get none.
__device__ __forceinline__ uint32_t gemm_accs(const GemmWork& w) { return w.by_rows ? (w.rows > 128 ? 2u : 1u) : w.slices; }

// K steps (of kBlockK elements) one stage holds.  A stage of e4m3 weights holds two: a row of the raw
// tile is then 128 bytes, which is what makes reads of host-resident weights over the link efficient
// (64-byte reads reach 42 GB/s, 128-byte reads 51 GB/s).  So does one of bf16 weights for up to 64 rows: their MMAs take 32 to 128
// cycles a K step where the producer takes 540 a stage, which is what a worker with one or two tiles waits for.
constexpr uint32_t kFetchStageBytes = 32 * 1024;
__device__ __forceinline__ int gemm_ksteps(const GemmWork& w) { return w.w_fp8 || (w.n <= 64 && w.slices == 1) ? 2 : 1; }
// kFetch = false (a kernel that never sees fetch records) compiles their handling away.
template <bool kFetch = true>
__device__ __forceinline__ int gemm_stage_count(const GemmWork& w) {
  if (kFetch && w.fetch) return static_cast<int>((w.fetch_bytes + kFetchStageBytes - 1) / kFetchStageBytes);
  return gemm_ksteps(w) == 2 ? (w.k_tiles + 1) >> 1 : w.k_tiles;
}
// Bytes of one stage: per K step the bf16 weight tile and the activation tile; layout: weight tiles,
// then activation tiles.  The raw e4m3 tile (128 rows of 128 bytes) lands in the second weight tile
// and is expanded in place: the 128-byte swizzle permutes 16-byte chunks inside a row, so row r of the
// second K step's bf16 tile covers exactly the bytes of raw row r, which one converter thread owns.
template <bool kFetch = true>
__device__ __forceinline__ uint32_t gemm_stage_bytes(const GemmWork& w) {
  if (kFetch && w.fetch) return kFetchStageBytes;
  return gemm_ksteps(w) * (w.slices * kATileBytes + w.n * kBlockK * 2);
}

struct GemmBarriers {
  uint64_t full[kGemmStages];
  uint64_t conv[kGemmStages];    // FP8: converter warps -> MMA (4 arrivals)
  uint64_t empty[kGemmStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
};

__device__ __forceinline__ void gemm_barriers_init(GemmBarriers& b) {
  for (int i = 0; i < kGemmStages; ++i) {
    mbar_init(&b.full[i], 1);
    mbar_init(&b.conv[i], 4);
    mbar_init(&b.empty[i], 1);
  }
  for (int i = 0; i < 2; ++i) {
    mbar_init(&b.acc_full[i], 1);
    mbar_init(&b.acc_empty[i], 4);
  }
}

// TMA issue for one tile.  The WHOLE producer warp calls it in step: every lane keeps the same bookkeeping, and one elected
// lane arms the barrier and issues the copies of a stage (one or two weight boxes and the activation rows).  Weights that are
// gathered from eight 16-row boxes go out as a single warp-wide instruction (lanes 0..7 the boxes, lane 8 the activation box,
// lanes 16..23 the second slice's).  What a stage costs here bounds every tile whose MMAs and loads take less: 770 cycles for 128 x 256
// with an array of stages in flight and lanes in roles, now 548 (of a tile that waits for nothing else), 650 -> 520 for 16 rows.
// Returns false when a wait was abandoned.
template <bool kFetch = true>
__device__ __forceinline__ bool gemm_produce(const GemmWork& w, uint8_t* ring, GemmBarriers& bar, GemmPipe& pipe,
                                             GemmInflight& fl, volatile int* abort_flag, uint64_t pol_w,
                                             uint64_t pol_x) {
  const int lane = threadIdx.x & 31;
  const uint32_t size = gemm_stage_bytes<kFetch>(w);
  const uint32_t b_bytes = w.n * kBlockK * 2;
  const int ks = gemm_ksteps(w);
  // FP8 weights land as raw bytes in the second weight tile (128-byte rows = two K steps, no swizzle)
  const uint32_t a_off = w.w_fp8 ? kATileBytes : 0;
  const uint32_t a_box = 2048;   // bytes of one 16-row box: 128-byte rows either way
  const int slices = w.slices;
  const uint32_t b_off = ks * slices * kATileBytes;
  const int n_stages = gemm_stage_count<kFetch>(w);
  // SwiGLU tiles of a tensor in the reference row order gather eight 16-row boxes;
  // every other tile is one 128-row box (a packed SwiGLU tensor stores gate/up
  // groups of 16 rows alternately, so its tile starts at row 2 * a_row_lo).
  const bool slab2 = epi_gated(w.epi) || (w.a_packed & 4);
  const bool gather = slab2 && !(w.a_packed & 1);
  const bool leader = elect_one();
  const int a_row0 = slab2 ? 2 * w.a_row_lo : w.a_row_lo;
  const bool wide_k = ks == 2 && !w.w_fp8;   // two weight tiles, one for each K step
  const int second = lane >> 4;   // lanes 16.. bring the boxes of the second slice, or of the second K step
  const int a_row = ((lane & 1) ? w.a_row_hi : w.a_row_lo) + 16 * ((lane & 7) >> 1) + (wide_k ? 0 : 64 * second);
  const int a_x = wide_k ? kBlockK * second : 0;
  const bool brings_a = (lane & 15) < 8 && second < (wide_k ? 2 : slices);
  const uint32_t a_at = a_off + second * kATileBytes + (lane & 7) * a_box;
  // read once: the record lives in shared memory and every copy below is a memory barrier to the compiler
  const bool fetch = kFetch && w.fetch != 0;
  const uint32_t fetch_bytes = kFetch ? w.fetch_bytes : 0;
  const uint8_t* const fetch_src = kFetch ? w.fetch_src : nullptr;
  const CUtensorMap* const a_map = w.a_map;
  const CUtensorMap* const b_map = w.b_map;
  const int a_z = w.a_z, b_row0 = w.b_row0, k0 = w.k0;
  // A block of 128 rows or more is one of several that read the slice; evicted first, 8192 tokens over 128 experts read 3.1 GB
  // from HBM where the weights and rows are 1.6.
  const uint64_t pol_a = w.n >= 128 ? policy_evict_normal() : pol_w;
  const uint32_t tx_bytes = (wide_k ? 2 : slices) * kATileBytes + ks * b_bytes;
  for (int st = 0; st < n_stages; ++st) {
    uint32_t vb, ve;
    const uint32_t phys = pipe.alloc(size, vb, ve);
    // room in the ring and a free barrier pair: retire the oldest stages as needed
    while (pipe.i - fl.tail >= kGemmStages ||
           (pipe.i != fl.tail && ve - fl.tail_vbegin > kRingBytes)) {
      if (!mbar_wait_warp(&bar.empty[fl.tail_slot], fl.tail_parity, abort_flag, kWaitBudgetNs)) return false;
      ++fl.tail;
      if (++fl.tail_slot == kGemmStages) {
        fl.tail_slot = 0;
        fl.tail_parity ^= 1;
      }
      fl.tail_vbegin = __shfl_sync(0xffffffffu, fl.vbegin, fl.tail_slot);
    }
    const uint32_t slot = pipe.slot;
    if (lane == static_cast<int>(slot)) fl.vbegin = vb;
    if (pipe.i == fl.tail) fl.tail_vbegin = vb;
    uint8_t* a = ring + phys;
    uint64_t* full = &bar.full[slot];
    if (fetch) {
      if (lane == 0) {
        const uint32_t at = st * kFetchStageBytes;
        const uint32_t bytes = min(kFetchStageBytes, fetch_bytes - at);
        mbar_arrive_expect_tx(full, bytes);
        bulk_load(a, fetch_src + at, bytes, full, pol_w);
      }
      __syncwarp();
      pipe.advance();
      continue;
    }
    // the second K step of an odd K range's last stage is loaded but not multiplied (gemm_mma)
    const int x = (k0 + st * ks) * kBlockK;
    if (!gather) {
      if (leader) {
        mbar_arrive_expect_tx(full, tx_bytes);
        tma_load_3d(a + a_off, a_map, full, x, a_row0, a_z, pol_a);
        if (slices == 2) tma_load_3d(a + kATileBytes, a_map, full, x, a_row0 + 128, a_z, pol_a);
        if (wide_k) tma_load_3d(a + kATileBytes, a_map, full, x + kBlockK, a_row0, a_z, pol_a);
        tma_load_2d(a + b_off, b_map, full, x, b_row0, pol_x);
        if (ks == 2) tma_load_2d(a + b_off + b_bytes, b_map, full, x + kBlockK, b_row0, pol_x);
      }
      pipe.advance();
      continue;
    }
    if (lane == 0) mbar_arrive_expect_tx(full, tx_bytes);
    __syncwarp();
    if (brings_a) {
      tma_load_3d(a + a_at, a_map, full, x + a_x, a_row, a_z, pol_a);
    } else if (lane >= 8 && lane < 8 + ks) {
      tma_load_2d(a + b_off + (lane - 8) * b_bytes, b_map, full, x + (lane - 8) * kBlockK, b_row0, pol_x);
    }
    pipe.advance();
  }
  return true;
}

// MMA issue for a tile of two accumulators (bf16 weights), g and g + 1, eight MMAs a stage: two weight slices against the
// activation rows, or (by_rows) two blocks of 128 activation rows against the weight rows.  A loop of its own: the
// one-accumulator loop bounds small tiles, and a branch on their number inside it cost it 100 cycles a stage.
__device__ __forceinline__ bool gemm_mma_two(const GemmWork& w, uint8_t* ring, GemmBarriers& bar, GemmPipe& pipe,
                                             uint32_t tmem_base, uint32_t g, volatile int* abort_flag) {
  const bool leader = elect_one();
  const uint32_t b0 = g & 1, b1 = b0 ^ 1;
  int ok = mbar_wait_bounded(&bar.acc_empty[b0], ((g >> 1) & 1) ^ 1, abort_flag, kWaitBudgetNs);
  const uint32_t idesc = umma_idesc_bf16(128, w.by_rows ? 128 * w.slices : w.n);
  const uint32_t acc0 = tmem_base + b0 * kAccCols, acc1 = tmem_base + b1 * kAccCols;
  const uint32_t size = gemm_stage_bytes<false>(w), ring_addr = smem_u32(ring), w_bytes = w.slices * kATileBytes;
  const uint64_t desc0 = umma_desc_sw128(0), m_off = (w.by_rows ? w_bytes : 0) >> 4, n_off = (w.by_rows ? 0 : w_bytes) >> 4;
  const int n_stages = w.k_tiles;
  for (int kt = 0; kt < n_stages; ++kt) {
    uint32_t vb, ve;
    const uint32_t phys = pipe.alloc(size, vb, ve);
    ok = ok && mbar_wait_bounded(&bar.full[pipe.slot], pipe.parity, abort_flag, kWaitBudgetNs);
    __syncwarp();   // as in gemm_mma
    tc_fence_after_sync();
    const uint64_t stage = desc0 + ((ring_addr + phys) >> 4), da = stage + m_off, db = stage + n_off;
    if (leader && ok) {
#pragma unroll
      for (int k = 0; k < kBlockK / 16; ++k) umma_bf16(acc0, da + 2 * k, db + 2 * k, idesc, (kt | k) != 0);
    }
    if (kt == 0) {   // the first accumulator's MMAs run while the second is still being drained
      ok = ok && mbar_wait_bounded(&bar.acc_empty[b1], (((g + 1) >> 1) & 1) ^ 1, abort_flag, kWaitBudgetNs);
      tc_fence_after_sync();
    }
    if (leader && ok) {
#pragma unroll
      for (int k = 0; k < kBlockK / 16; ++k)
        umma_bf16(acc1, da + (kATileBytes >> 4) + 2 * k, db + 2 * k, idesc, (kt | k) != 0);
      umma_commit(&bar.empty[pipe.slot]);
    }
    pipe.advance();
  }
  if (leader && ok) {
    umma_commit(&bar.acc_full[b0]);
    umma_commit(&bar.acc_full[b1]);
  }
  return __all_sync(0xffffffffu, ok != 0);
}

// MMA issue for one tile into accumulator g (buffer g & 1).
// The whole MMA warp runs the K loop in step (every lane waits for the stage itself, and the warp meets behind the wait) and one
// elected lane issues the four tcgen05.mma and the commit of a stage.  Because the loop is convergent code,
// its descriptors and addresses are warp-uniform values; with the loop inside a single-lane branch
// the MMA warp spent twice as long issuing (measured: 67 -> 32 us of a 150 us launch), which is
// what bounds small-N tiles.
template <bool kFetch = true>
__device__ __forceinline__ bool gemm_mma(const GemmWork& w, uint8_t* ring, GemmBarriers& bar, GemmPipe& pipe,
                                         uint32_t tmem_base, uint32_t g, volatile int* abort_flag,
                                         long long* wait_cycles = nullptr) {
  if (gemm_accs(w) == 2) return gemm_mma_two(w, ring, bar, pipe, tmem_base, g, abort_flag);
  int ok = 1;
  const uint32_t buf = g & 1, acc_parity = (g >> 1) & 1;
  const bool leader = elect_one();
  {
    const long long ta = wait_cycles ? clock64() : 0;
    if (!mbar_wait_bounded(&bar.acc_empty[buf], acc_parity ^ 1, abort_flag, kWaitBudgetNs)) ok = 0;
    if (wait_cycles) wait_cycles[2] += clock64() - ta;
    tc_fence_after_sync();
    const uint32_t idesc = umma_idesc_bf16(128, w.by_rows ? 128 * w.slices : w.n);
    const uint32_t acc = tmem_base + buf * kAccCols;
    const uint32_t size = gemm_stage_bytes<kFetch>(w);
    uint64_t* ready = w.w_fp8 ? bar.conv : bar.full;
    const uint32_t ring_addr = smem_u32(ring);
    const uint64_t desc0 = umma_desc_sw128(0);
    const int n_stages = gemm_stage_count<kFetch>(w);
    const uint32_t b_bytes = w.n * kBlockK * 2;
    const uint64_t m_off = (w.by_rows ? w.slices * kATileBytes : 0) >> 4, n_off = (w.by_rows ? 0 : kATileBytes) >> 4;
    // read once: the record lives in shared memory and every wait below is a memory barrier to the compiler
    const bool fp8 = w.w_fp8 != 0, fetch = kFetch && w.fetch != 0, one_step = gemm_ksteps(w) == 1;
    const int k_steps = w.k_tiles;
    const uint32_t fetch_bytes = kFetch ? w.fetch_bytes : 0;
    uint8_t* const fetch_out = static_cast<uint8_t*>(w.out);
    for (int kt = 0; kt < n_stages; ++kt) {
      uint32_t vb, ve;
      const uint32_t phys = pipe.alloc(size, vb, ve);
      const long long tw = wait_cycles ? clock64() : 0;
      const uint32_t ready_parity = fp8 ? (pipe.conv_bits >> pipe.slot) & 1u : pipe.parity;
      ok = ok && mbar_wait_bounded(&ready[pipe.slot], ready_parity, abort_flag, kWaitBudgetNs);
      // a lane that has not seen the stage when the leader frees it would miss its phase once it is filled again, and wait for good
      __syncwarp();
      if (fp8) pipe.conv_bits ^= 1u << pipe.slot;
      if (wait_cycles) wait_cycles[0] += clock64() - tw;
      if (fetch) {
        // the stage goes on to the staging buffer; its shared memory is free once the store has read it
        if (leader && ok) {
          const uint32_t at = kt * kFetchStageBytes;
          bulk_store(fetch_out + at, ring + phys, min(kFetchStageBytes, fetch_bytes - at));
          bulk_commit();
          bulk_wait_read_all();
          mbar_arrive(&bar.empty[pipe.slot]);
        }
        pipe.advance();
        continue;
      }
      const long long ti = wait_cycles ? clock64() : 0;
      if (!leader || !ok) {
      } else if (one_step) {   // weight tile, activation tile
        const uint64_t stage = desc0 + ((ring_addr + phys) >> 4), da = stage + m_off, db = stage + n_off;
#pragma unroll
        for (int k = 0; k < kBlockK / 16; ++k) umma_bf16(acc, da + 2 * k, db + 2 * k, idesc, (kt | k) != 0);
      } else {      // two K steps: weight tiles 0 and 1, then activation tiles 0 and 1
        const uint64_t da = desc0 + ((ring_addr + phys) >> 4);
        const uint64_t db = da + (2 * kATileBytes >> 4);
#pragma unroll
        for (int k = 0; k < kBlockK / 16; ++k) umma_bf16(acc, da + 2 * k, db + 2 * k, idesc, (kt | k) != 0);
        // the last stage of an odd K range holds one K step of the range; its second half belongs to the
        // next range (a K split) or lies past the tensor, and is left out
        if (2 * kt + 1 < k_steps) {
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
            umma_bf16(acc, da + (kATileBytes >> 4) + 2 * k, db + (b_bytes >> 4) + 2 * k, idesc, true);
        }
      }
      if (leader && ok) umma_commit(&bar.empty[pipe.slot]);
      if (wait_cycles) wait_cycles[1] += clock64() - ti;
      pipe.advance();
    }
    if (ok && fetch) {
      // the record counts as done when its bytes are in the staging buffer, for readers of either proxy
      if (leader) {
        bulk_wait_all();
        fence_proxy_async_all();
        __threadfence();
        mbar_arrive(&bar.acc_full[buf]);
      }
    } else if (ok && leader) {
      umma_commit(&bar.acc_full[buf]);
    }
  }
  return __all_sync(0xffffffffu, ok != 0);
}

// FP8 weights (W8A16, csrc/fabric/tiles/gemm.cuh:14-18,73-94): the four converter
// warps expand the raw e4m3 tile of every stage into the bf16 weight tile with the
// 128-byte swizzle.  Every e4m3 value is exactly a bf16 value, so the MMA sees the
// exact weights; the per-output-channel fp32 scale is applied in the epilogue.
// Thread t converts row t: per K step 64 bytes in, 128 bytes out in eight 16-byte chunks,
// chunk c of row r going to chunk c ^ (r & 7).  A lane whose wait gave up goes through the loop with its warp, and the warp answers as
// one at the end (a vote behind each wait: 64 tokens of the e4m3 layer 538 -> 549 us).
__device__ __forceinline__ bool gemm_convert(const GemmWork& w, uint8_t* ring, GemmBarriers& bar, GemmPipe& pipe,
                                             int row, volatile int* abort_flag) {
  const uint32_t size = gemm_stage_bytes(w);
  const int ks = gemm_ksteps(w), n_stages = gemm_stage_count(w);
  const uint32_t raw_off = kATileBytes;
  int ok = 1;
  for (int kt = 0; kt < n_stages; ++kt) {
    uint32_t vb, ve;
    const uint32_t phys = pipe.alloc(size, vb, ve);
    ok = ok && mbar_wait_bounded(&bar.full[pipe.slot], pipe.parity, abort_flag, kWaitBudgetNs);
    // The row's raw bytes [64 h, 64 h + 64) are K step h.  The thread reads its whole row before it
    // writes (the second K step's output overwrites the raw row), starting at 16-byte chunk t & 7 so
    // that the eight threads of a shared-memory phase read eight different bank groups.
    const uint4* src = reinterpret_cast<const uint4*>(ring + phys + raw_off + row * 128);
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = src[(i + row) & 7];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = (i + row) & 7, h = q >> 2, c = q & 3;
      uint8_t* dst = ring + phys + h * kATileBytes + row * 128;
      const uint32_t in[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      uint32_t out[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(in[j] & 0xffffu), __NV_E4M3);
        const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(in[j] >> 16), __NV_E4M3);
        const float2 fl = __half22float2(*reinterpret_cast<const __half2*>(&lo));
        const float2 fh = __half22float2(*reinterpret_cast<const __half2*>(&hi));
        const __nv_bfloat162 bl = __floats2bfloat162_rn(fl.x, fl.y), bh = __floats2bfloat162_rn(fh.x, fh.y);
        out[2 * j] = *reinterpret_cast<const uint32_t*>(&bl);
        out[2 * j + 1] = *reinterpret_cast<const uint32_t*>(&bh);
      }
      // 16 input bytes -> 32 output bytes = chunks 2c and 2c + 1 of the row
      *reinterpret_cast<uint4*>(dst + (((2 * c) ^ (row & 7)) << 4)) = make_uint4(out[0], out[1], out[2], out[3]);
      *reinterpret_cast<uint4*>(dst + (((2 * c + 1) ^ (row & 7)) << 4)) = make_uint4(out[4], out[5], out[6], out[7]);
    }
    fence_proxy_async_smem();   // generic-proxy writes -> visible to the tensor core's operand reads
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(&bar.conv[pipe.slot]);
    pipe.advance();
  }
  return __all_sync(0xffffffffu, ok != 0);
}

__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

// gelu in its tanh form, times u: 0.5 g (1 + tanh(t)) = g / (1 + exp(-2 t)), t = sqrt(2 / pi) (g + 0.044715 g^3).
__device__ __forceinline__ float gelu_mul(float g, float u) {
  const float t2 = 1.5957691216057308f * fmaf(0.044715f * g * g, g, g);
  return __fdividef(g, 1.f + __expf(-t2)) * u;
}

// expm1(-coef softplus(z)), coef >= 0: the distance to one of a decay e^(-coef softplus(z)).  Power series where the sums
// 1 + t and e^x - 1 would cancel; no branches.
__device__ __forceinline__ float decay_less_one(float z, float coef) {
  const float t = __expf(-fabsf(z));
  const float log_small = t * fmaf(t, fmaf(t, fmaf(t, -0.25f, 1.f / 3.f), -0.5f), 1.f), log_large = __logf(1.f + t);
  const float x = -coef * (fmaxf(z, 0.f) + (t < 0.02f ? log_small : log_large));
  const float small = x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.f / 720.f, 1.f / 120.f), 1.f / 24.f), 1.f / 6.f), 0.5f), 1.f);
  const float large = __expf(x) - 1.f;
  return x > -0.25f ? small : large;
}

// One value of kEpiStoreBf16 / the fp32 epilogues / kEpiDecay.
template <int E>
__device__ __forceinline__ float epi_value(uint32_t acc, float sc, float bias, float coef) {
  const float v = __uint_as_float(acc) * sc + bias;
  return E == kEpiDecay ? decay_less_one(v, coef) : v;
}

// The chunks (32 accumulator columns = activation rows) of one slice, all of them by epilogue E.  The epilogue is fixed at
// compile time and a whole chunk has no per-row conditions, so that a chunk's 16 or 32 values are computed side by side:
// with a branch per row (two activations, rows past the end) a chunk took 1.9 us and the epilogue, one warp per
// scheduler, bounded the products: 128 rows of a SwiGLU tile 8.2 us, now 2.2.  The next chunk's TMEM load, and the
// residual's values of the next chunk, are under way while this one is converted and stored.  (The residual loaded where
// it was added, a 2-byte load behind each 2-byte store, took 0.6 us a row.)  kSixteen: a tile may have 16 rows only.
template <int E, bool kSixteen = false>
__device__ __forceinline__ void epilogue_chunks(const GemmWork& w, uint32_t tacc, int f, int wrow, bool f_ok, float sc,
                                                float bias, float coef) {
  const int lane = threadIdx.x & 31;
  const int n = w.n, rows = w.rows, ld = w.ld_out, c_end = min(n, rows);
  const bool lo = lane < 16;
  constexpr bool kGated = E == kEpiSiluMul || E == kEpiGeluMul;
  const size_t first = static_cast<size_t>(w.b_row0) * ld + (E == kEpiAtomicF32 && (w.a_packed & 4) ? wrow : f);
  unsigned short* const out16 = reinterpret_cast<unsigned short*>(w.out) + first;
  float* const out32 = reinterpret_cast<float*>(w.out) + first;
  const unsigned short* const res = E == kEpiStoreBf16 && w.residual && f_ok
      ? reinterpret_cast<const unsigned short*>(w.residual) + static_cast<size_t>(w.b_row0) * w.ld_res + f : nullptr;
  const int ld_res = w.ld_res;
  constexpr int kRes = E == kEpiStoreBf16 ? 32 : 1;
  unsigned short rn[kRes];   // the next chunk's residual values
  auto load_res = [&](int c0) {
    if (E != kEpiStoreBf16 || !res) return;
    const unsigned short* p = res + static_cast<size_t>(c0) * ld_res;
#pragma unroll
    for (int j = 0; j < kRes; ++j) rn[j] = c0 + j < rows ? p[static_cast<size_t>(j) * ld_res] : 0;
  };
  uint32_t next[32];
  load_res(0);
  if (!kSixteen || n >= 32) {
    tmem_ld_32x32(tacc, next);
  } else {
    uint32_t r16[16];
    tmem_ld_32x16(tacc, r16);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      next[j] = r16[j];
      next[16 + j] = 0;
    }
  }
  if (c_end <= 0) tmem_ld_wait();
#pragma unroll 1
  for (int c0 = 0; c0 < c_end; c0 += 32) {
    uint32_t r[32];
    unsigned short rv[kRes];
    __syncwarp();
    tmem_ld_wait_for(next);
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = next[j];
#pragma unroll
    for (int j = 0; j < kRes; ++j) rv[j] = rn[j];
    if (c0 + 32 < c_end) {   // n is a power of two: a whole chunk
      tmem_ld_32x32(tacc + c0 + 32, next);
      load_res(c0 + 32);
    }
    const bool whole = c0 + 32 <= rows;
    if constexpr (kGated) {
      // lanes < 16 own gate rows, lanes >= 16 the matching up rows; exchange halves: the lower lanes take the chunk's
      // first 16 rows, the upper ones the others
      float mine[16], other[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        mine[j] = __uint_as_float(lo ? r[j] : r[16 + j]) * sc;
        other[j] = __shfl_xor_sync(0xffffffffu, __uint_as_float(lo ? r[16 + j] : r[j]) * sc, 16);
      }
      unsigned short hv[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float gate = lo ? mine[j] : other[j], up = lo ? other[j] : mine[j];
        hv[j] = __bfloat16_as_ushort(__float2bfloat16(E == kEpiGeluMul ? gelu_mul(gate, up) : silu_mul(gate, up)));
      }
      const int t0 = c0 + (lo ? 0 : 16);
      unsigned short* const o = out16 + static_cast<size_t>(t0) * ld;
      if (whole && f_ok) {
#pragma unroll
        for (int j = 0; j < 16; ++j) o[static_cast<size_t>(j) * ld] = hv[j];
      } else if (f_ok) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (t0 + j < rows) o[static_cast<size_t>(j) * ld] = hv[j];
      }
    } else if constexpr (E == kEpiStoreBf16) {
      unsigned short hv[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        float v = epi_value<E>(r[j], sc, bias, coef);
        if (res) v += __bfloat162float(__ushort_as_bfloat16(rv[j]));
        hv[j] = __bfloat16_as_ushort(__float2bfloat16(v));
      }
      unsigned short* const o = out16 + static_cast<size_t>(c0) * ld;
      if (whole && f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j) __stcs(o + static_cast<size_t>(j) * ld, hv[j]);
      } else if (f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c0 + j < rows) __stcs(o + static_cast<size_t>(j) * ld, hv[j]);
      }
    } else if constexpr (E == kEpiWeightedAdd) {
      if (f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (c0 + j < rows) {
            const int m = w.b_row0 + c0 + j;
            atomicAdd(reinterpret_cast<float*>(w.out) + f + static_cast<size_t>(w.pair_token[m]) * ld,
                      w.pair_weight[m] * (__uint_as_float(r[j]) * sc));
          }
        }
      }
    } else if constexpr (E == kEpiAtomicF32) {
      // a two-slab tile (partial sums of a SwiGLU pair) adds into the column of its weight row
      if (f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c0 + j < rows) atomicAdd(out32 + static_cast<size_t>(c0 + j) * ld, __uint_as_float(r[j]) * sc + bias);
      }
    } else {
      // fp32 rows; those that are read once, later (per-pair expert outputs, logits) by streaming stores
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = epi_value<E>(r[j], sc, bias, coef);
      float* const o = out32 + static_cast<size_t>(c0) * ld;
      if (whole && f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (E == kEpiDecay) o[static_cast<size_t>(j) * ld] = v[j];
          else __stcs(o + static_cast<size_t>(j) * ld, v[j]);
        }
      } else if (f_ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c0 + j < rows) __stcs(o + static_cast<size_t>(j) * ld, v[j]);
      }
    }
  }
}

// 32 bytes to a 32-byte aligned address, one sector; kStream: read once, later.
template <bool kStream>
__device__ __forceinline__ void st_sector(void* p, const uint32_t (&v)[8]) {
  if constexpr (kStream)
    asm volatile("st.global.cs.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  else
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// The rows [row0, row0 + 32) of a warp under a by_rows tile, one in each lane; columns of the accumulator are weight rows.
// 32 columns at a time (16 features of a gated tile: 16 gate columns, then their up columns), the next 32 under way
// meanwhile, as are the residual's.  A lane puts its values into the warp's 4 KB of shared memory (`buf`, 16-byte pieces swizzled
// by the row), from where 128 bytes of a row leave as one line, four lanes a row.  (Each lane storing its own row, 32
// bytes of 32 rows an instruction, held the SM to 17 bytes a cycle.)  Rows that are not on sector boundaries, and a last chunk that
// the features do not fill, go element by element.
template <int E>
__device__ __forceinline__ void epilogue_rows(const GemmWork& w, uint32_t tacc, int row0, uint8_t* buf) {
  const int lane = threadIdx.x & 31, row = row0 + lane;
  constexpr bool kGated = E == kEpiSiluMul || E == kEpiGeluMul, kHalf = kGated || E == kEpiStoreBf16;
  constexpr int NF = kGated ? 16 : 32;   // features of a chunk
  const int first = w.a_row_lo, left = w.n_limit - first;   // features from here on
  const int chunks = min(4 * w.slices, (left + NF - 1) / NF), rows = w.rows;
  const bool row_ok = row < rows;
  using Out = typename std::conditional<kHalf, unsigned short, float>::type;
  const size_t ld = w.ld_out;
  Out* const out = reinterpret_cast<Out*>(w.out) + static_cast<size_t>(w.b_row0 + row0) * ld + first;
  const int whole = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && ((ld * sizeof(Out)) & 31) == 0 ? min(chunks, left / NF) : 0;
  constexpr int kBytes = NF * static_cast<int>(sizeof(Out)), kLine = 128 / kBytes;   // of a chunk's row; chunks of a line
  uint4* const mine = reinterpret_cast<uint4*>(buf) + 8 * lane;
  Out* const to = out + static_cast<size_t>(lane >> 2) * ld + (lane & 3) * (32 / sizeof(Out));
  const __nv_bfloat16* const bias = !kGated && E != kEpiRowsF32 && w.bias && w.k0 == 0 ? w.bias + first : nullptr;
  const float* const coef = E == kEpiDecay ? w.pair_weight + first : nullptr;
  const unsigned short* const res = E == kEpiStoreBf16 && w.residual && row_ok
      ? reinterpret_cast<const unsigned short*>(w.residual) + static_cast<size_t>(w.b_row0 + row) * w.ld_res + first : nullptr;
  const bool res16 = (reinterpret_cast<uintptr_t>(res) & 15) == 0;
  constexpr int kRes = E == kEpiStoreBf16 ? 4 : 1;
  uint4 rn[kRes];   // the next chunk's residual
  auto load_res = [&](int c) {
    if (E != kEpiStoreBf16 || !res) return;
    const unsigned short* p = res + c * NF;
    if (res16 && (c + 1) * NF <= left) {
#pragma unroll
      for (int i = 0; i < kRes; ++i) rn[i] = reinterpret_cast<const uint4*>(p)[i];
    } else {
      uint32_t v[4 * kRes];
#pragma unroll
      for (int i = 0; i < 4 * kRes; ++i) {
        const uint32_t a = c * NF + 2 * i < left ? p[2 * i] : 0, b = c * NF + 2 * i + 1 < left ? p[2 * i + 1] : 0;
        v[i] = a | b << 16;
      }
#pragma unroll
      for (int i = 0; i < kRes; ++i) rn[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
  };
  uint32_t next[32];
  load_res(0);
  __syncwarp();
  tmem_ld_32x32(tacc, next);
  if (chunks <= 0) tmem_ld_wait();
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    uint32_t r[32], rv[4 * kRes];
    __syncwarp();
    tmem_ld_wait_for(next);
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = next[j];
#pragma unroll
    for (int i = 0; i < kRes; ++i) {
      rv[4 * i] = rn[i].x;
      rv[4 * i + 1] = rn[i].y;
      rv[4 * i + 2] = rn[i].z;
      rv[4 * i + 3] = rn[i].w;
    }
    if (c + 1 < chunks) {
      tmem_ld_32x32(tacc + 32 * (c + 1), next);
      load_res(c + 1);
    }
    const int f = c * NF, n = min(NF, left - f);   // features of this chunk that exist
    uint32_t o[kHalf ? NF / 2 : NF];
    if constexpr (kGated) {
#pragma unroll
      for (int j = 0; j < NF; j += 2) {
        float h[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float gate = __uint_as_float(r[j + i]), up = __uint_as_float(r[16 + j + i]);
          h[i] = E == kEpiGeluMul ? gelu_mul(gate, up) : silu_mul(gate, up);
        }
        o[j / 2] = pack_bf16(h[0], h[1]);
      }
    } else {
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
      if (bias) {   // the same for every lane
        if (n == NF && (reinterpret_cast<uintptr_t>(bias) & 15) == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 b = reinterpret_cast<const uint4*>(bias + f)[i];
            const uint32_t u[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) v[8 * i + j] += __uint_as_float(j & 1 ? u[j / 2] & 0xffff0000u : u[j / 2] << 16);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += j < n ? __bfloat162float(bias[f + j]) : 0.f;
        }
      }
      if constexpr (E == kEpiDecay) {
        if (n == NF && (reinterpret_cast<uintptr_t>(coef) & 15) == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 k = reinterpret_cast<const float4*>(coef + f)[i];
            v[4 * i] = decay_less_one(v[4 * i], k.x);
            v[4 * i + 1] = decay_less_one(v[4 * i + 1], k.y);
            v[4 * i + 2] = decay_less_one(v[4 * i + 2], k.z);
            v[4 * i + 3] = decay_less_one(v[4 * i + 3], k.w);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = decay_less_one(v[j], j < n ? coef[f + j] : 0.f);
        }
      }
      if constexpr (E == kEpiStoreBf16) {
        if (res) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(j & 1 ? rv[j / 2] & 0xffff0000u : rv[j / 2] << 16);
        }
#pragma unroll
        for (int j = 0; j < 32; j += 2) o[j / 2] = pack_bf16(v[j], v[j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(v[j]);
      }
    }
    if (c < whole) {
      const int at = c % kLine;   // place in the line
#pragma unroll
      for (int i = 0; i < kBytes / 16; ++i)
        mine[(at * (kBytes / 16) + i) ^ (lane & 7)] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      if (at != kLine - 1 && c + 1 != whole) continue;
      __syncwarp();
      const int p = lane & 3;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        if (row0 + r < rows && p < (at + 1) * (kBytes / 32)) {
          const uint4* from = reinterpret_cast<const uint4*>(buf) + 8 * r;
          const uint4 a = from[(2 * p) ^ (r & 7)], b = from[(2 * p + 1) ^ (r & 7)];
          const uint32_t q[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          st_sector<!kHalf && E != kEpiDecay>(to + 8 * i * ld + (c - at) * NF, q);
        }
      }
      __syncwarp();
    } else if (row_ok) {
      Out* const own = out + lane * ld + f;
#pragma unroll
      for (int j = 0; j < NF; ++j) {
        if (j >= n) continue;
        if constexpr (kHalf) own[j] = static_cast<unsigned short>(j & 1 ? o[j / 2] >> 16 : o[j / 2] & 0xffffu);
        else own[j] = __uint_as_float(o[j]);
      }
    }
  }
}

// The fabric kernel calls them: seven of them inlined cost its other roles registers (252 bytes of spills against 48).
template <int E>
__device__ __noinline__ void epilogue_call(const GemmWork& w, uint32_t tacc, int f, int wrow, bool f_ok, float sc, float bias,
                                           float coef) {
  __builtin_assume(__isShared(&w));
  epilogue_chunks<E>(w, tacc, f, wrow, f_ok, sc, bias, coef);
}

// The one chunk of a tile of at most 32 activation rows, in the fabric: each row's store behind its own condition.  A decode step
// runs every epilogue once or twice per SM, so what it waits for is the fetch of the instructions, of which epilogue_chunks has
// several times as many.  (One step of 32 sequences of Sinotar 983 -> 961 us, of eight of the decoder 1515 -> 1499; the expert
// kernel has two epilogues, which stay in its instruction cache, and takes epilogue_chunks for any height: 256 tokens 189 -> 184.)
__device__ __forceinline__ void epilogue_few(const GemmWork& w, uint32_t tacc, int f, int wrow, bool f_ok, float sc, float bias) {
  const int lane = threadIdx.x & 31;
  uint32_t r[32];
  if (w.n >= 32) {
    tmem_ld_32x32(tacc, r);
  } else {
    uint32_t r16[16];
    tmem_ld_32x16(tacc, r16);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      r[j] = r16[j];
      r[16 + j] = 0;
    }
  }
  tmem_ld_wait();
  if (epi_gated(w.epi)) {
    // lanes < 16 own gate rows, lanes >= 16 the matching up rows; exchange halves
    const bool lo = lane < 16, gelu = w.epi == kEpiGeluMul;
    const int t0 = lo ? 0 : 16;
    unsigned short* out = reinterpret_cast<unsigned short*>(w.out) + static_cast<size_t>(w.b_row0 + t0) * w.ld_out + f;
    unsigned short hv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float mine = __uint_as_float(lo ? r[j] : r[16 + j]) * sc;
      const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(lo ? r[16 + j] : r[j]) * sc, 16);
      const float gate = lo ? mine : other, up = lo ? other : mine;
      hv[j] = __bfloat16_as_ushort(__float2bfloat16(gelu ? gelu_mul(gate, up) : silu_mul(gate, up)));
    }
    if (!f_ok) return;
    const int m_hi = w.rows - t0;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < m_hi) out[static_cast<size_t>(j) * w.ld_out] = hv[j];
    return;
  }
  if (!f_ok) return;
  if (w.epi == kEpiStoreBf16) {
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(w.out) + static_cast<size_t>(w.b_row0) * w.ld_out + f;
    const __nv_bfloat16* res = w.residual ? w.residual + static_cast<size_t>(w.b_row0) * w.ld_res + f : nullptr;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      if (j < w.rows) {
        float v = __uint_as_float(r[j]) * sc + bias;
        if (res) v += __bfloat162float(res[static_cast<size_t>(j) * w.ld_res]);
        __stcs(reinterpret_cast<unsigned short*>(out + static_cast<size_t>(j) * w.ld_out),
               __bfloat16_as_ushort(__float2bfloat16(v)));
      }
    }
    return;
  }
  if (w.epi == kEpiWeightedAdd) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      if (j < w.rows) {
        const int m = w.b_row0 + j;
        atomicAdd(reinterpret_cast<float*>(w.out) + f + static_cast<size_t>(w.pair_token[m]) * w.ld_out,
                  w.pair_weight[m] * (__uint_as_float(r[j]) * sc));
      }
    }
    return;
  }
  // a two-slab tile (partial sums of a SwiGLU pair) adds into the column of its weight row
  float* const out = reinterpret_cast<float*>(w.out) + static_cast<size_t>(w.b_row0) * w.ld_out +
                     (w.epi == kEpiAtomicF32 && (w.a_packed & 4) ? wrow : f);
  if (w.epi == kEpiAtomicF32) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < w.rows) atomicAdd(out + static_cast<size_t>(j) * w.ld_out, __uint_as_float(r[j]) * sc + bias);
  } else if (w.epi == kEpiDecay) {
    const float coef = w.pair_weight[f];
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(epi_value<kEpiDecay>(r[j], sc, bias, coef));
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < w.rows) out[static_cast<size_t>(j) * w.ld_out] = __uint_as_float(r[j]);
  } else {
    // fp32 rows that are read once, later (per-pair expert outputs, logits): streaming stores
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < w.rows) __stcs(out + static_cast<size_t>(j) * w.ld_out, __uint_as_float(r[j]) * sc + bias);
  }
}

template <int E>
__device__ __noinline__ void epilogue_rows_call(const GemmWork& w, uint32_t tacc, int row0, uint8_t* buf) {
  __builtin_assume(__isShared(&w));
  __builtin_assume(__isShared(buf));
  epilogue_rows<E>(w, tacc, row0, buf);
}

// Epilogue of one accumulator of a tile from buffer `buf` (the four epilogue warps
// call): everything except handing the buffer back to the MMA warp.  kFetch = false: the expert kernel, which has two
// epilogues and no fetch records.
template <bool kFetch = true>
__device__ __forceinline__ bool gemm_epilogue_body(const GemmWork& w, int slice, GemmBarriers& bar, uint32_t tmem_base,
                                                   uint32_t buf, uint32_t acc_parity, volatile int* abort_flag, uint8_t* ring,
                                                   unsigned long long* acc_seen = nullptr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
  if (!mbar_wait_warp(&bar.acc_full[buf], acc_parity, abort_flag, kWaitBudgetNs)) return false;
  tc_fence_after_sync();
  if (acc_seen && lane == 0) *acc_seen = globaltimer_ns();
  if (kFetch && w.fetch) {   // nothing to drain: the MMA warp has already moved the bytes
    __syncwarp();
    return true;
  }
  const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * kAccCols;
  if (w.by_rows) {
    const int row0 = 128 * slice + 32 * quad;
    uint8_t* const lines = ring + kRingBytes + 4096 * quad;
    if (row0 >= w.rows) {   // no row of this warp exists
    } else if constexpr (kFetch) {
      switch (w.epi) {
        case kEpiStoreBf16: epilogue_rows_call<kEpiStoreBf16>(w, tacc, row0, lines); break;
        case kEpiSiluMul: epilogue_rows_call<kEpiSiluMul>(w, tacc, row0, lines); break;
        case kEpiGeluMul: epilogue_rows_call<kEpiGeluMul>(w, tacc, row0, lines); break;
        case kEpiDecay: epilogue_rows_call<kEpiDecay>(w, tacc, row0, lines); break;
        default: epilogue_rows_call<kEpiStoreF32>(w, tacc, row0, lines); break;
      }
    } else if (w.epi == kEpiSiluMul) {
      epilogue_rows<kEpiSiluMul>(w, tacc, row0, lines);
    } else {
      epilogue_rows<kEpiRowsF32>(w, tacc, row0, lines);
    }
    fence_proxy_async_smem();   // a wide tile may fill the lines' memory by copies next
    tc_fence_before_sync();
    __syncwarp();
    return true;
  }
  const bool slab2 = epi_gated(w.epi) || (w.a_packed & 4);
  // output feature of this lane, and the weight row its accumulator row came from
  int f, wrow;
  if (slab2) {
    f = w.a_row_lo + 64 * slice + 16 * quad + (lane & 15);
    wrow = (lane < 16 ? w.a_row_lo : w.a_row_hi) + 64 * slice + 16 * quad + (lane & 15);
  } else {
    f = w.a_row_lo + 128 * slice + 32 * quad + lane;
    wrow = f;
  }
  const bool f_ok = f < w.n_limit;
  const float sc = (w.scale && f_ok) ? w.scale[wrow] : 1.f;
  if constexpr (kFetch) {
    const float bias = (w.bias && f_ok && w.k0 == 0) ? __bfloat162float(w.bias[f]) : 0.f;
    if (w.n <= 32) epilogue_few(w, tacc, f, wrow, f_ok, sc, bias);
    else switch (w.epi) {
      case kEpiStoreBf16: epilogue_call<kEpiStoreBf16>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
      case kEpiSiluMul: epilogue_call<kEpiSiluMul>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
      case kEpiGeluMul: epilogue_call<kEpiGeluMul>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
      case kEpiWeightedAdd: epilogue_call<kEpiWeightedAdd>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
      case kEpiAtomicF32: epilogue_call<kEpiAtomicF32>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
      case kEpiDecay:
        epilogue_call<kEpiDecay>(w, tacc, f, wrow, f_ok, sc, bias, f_ok ? w.pair_weight[f] : 0.f);
        break;
      default: epilogue_call<kEpiStoreF32>(w, tacc, f, wrow, f_ok, sc, bias, 0.f); break;
    }
  } else if (w.epi == kEpiSiluMul) {
    epilogue_chunks<kEpiSiluMul, true>(w, tacc, f, wrow, f_ok, sc, 0.f, 0.f);
  } else {
    epilogue_chunks<kEpiRowsF32, true>(w, tacc, f, wrow, f_ok, sc, 0.f, 0.f);
  }
  tc_fence_before_sync();
  __syncwarp();
  return true;
}

// The four epilogue warps: every accumulator of a tile whose first one is g.
template <bool kFetch = true>
__device__ __forceinline__ bool gemm_epilogue(const GemmWork& w, GemmBarriers& bar, uint32_t tmem_base, uint32_t g,
                                              volatile int* abort_flag, uint8_t* ring, unsigned long long* acc_seen = nullptr) {
  const int accs = static_cast<int>(gemm_accs(w));
#pragma unroll 1
  for (int i = 0; i < accs; ++i, ++g) {
    if (!gemm_epilogue_body<kFetch>(w, i, bar, tmem_base, g & 1, (g >> 1) & 1, abort_flag, ring, acc_seen)) return false;
    if ((threadIdx.x & 31) == 0) mbar_arrive(&bar.acc_empty[g & 1]);
  }
  return true;
}

}  // namespace mf
