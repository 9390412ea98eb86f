// Pieces of the wide tiles (tiles whose exec warps own the worker's operand ring and TMEM while they run): operand
// descriptors, TMA boxes, TMEM stores, bounded waits and the common decision to go on.
#pragma once
#include "fabric_layer_tiles.cuh"
#include "ptx.cuh"
#include "types.h"

namespace mf {
namespace fab {

constexpr unsigned long long kWideWaitNs = 4000000000ull;
constexpr float kSlack = 8.f;   // how far (exp2 domain) a row maximum may exceed the reference of its exponentials

// Matrix descriptor of an operand in 128-byte-swizzled shared memory; lead: bytes to the next 64 elements of an MN-major
// operand's major dimension, stride: bytes to the next eight rows.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, uint32_t lead, uint32_t stride) {
  return static_cast<uint64_t>((addr & 0x3ffffu) >> 4) | (static_cast<uint64_t>(lead >> 4) << 16) |
         (static_cast<uint64_t>(stride >> 4) << 32) | (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
__device__ __forceinline__ void tma_box_2d(void* smem, unsigned long long map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(smem)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_box_3d(void* smem, unsigned long long map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(smem)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_box_4d(void* smem, unsigned long long map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          smem_u32(smem)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_4d(unsigned long long map, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Barrier of the exec threads that also tells each whether `v` held in all / any of them.
__device__ __forceinline__ bool exec_and(bool v) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\tbar.red.and.pred p, 1, %2, q;\n\tselp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(r) : "r"(static_cast<int>(v)), "n"(kExecThreads) : "memory");
  return r != 0;
}

// NV values per lane summed over groups of LB lanes: lane l of a group ends with values [l NV / LB, ..), max(1, NV / LB) of
// them, at the front of v.
template <int N, int BIT, int NV>
__device__ __forceinline__ void group_sum_from(float (&v)[NV], int lane) {
  if constexpr (BIT >= 1) {
    if constexpr (N > 1) {
      const bool hi = lane & BIT;
#pragma unroll
      for (int c = 0; c < N / 2; ++c) {
        const float give = hi ? v[c] : v[c + N / 2], have = hi ? v[c + N / 2] : v[c];
        v[c] = have + __shfl_xor_sync(0xffffffffu, give, BIT);
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], BIT);
    }
    group_sum_from<(N > 1 ? N / 2 : 1), BIT / 2>(v, lane);
  }
}
template <int NV, int LB>
__device__ __forceinline__ void group_sum(float (&v)[NV], int lane) { group_sum_from<NV, LB / 2>(v, lane); }

// 16-byte asynchronous copies into shared memory, in groups of the issuing thread.
__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Untiled bulk copies; the load completes on an mbarrier, stores in bulk groups of the issuing thread.
__device__ __forceinline__ void bulk_in(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem)),
               "l"(gmem), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// More bytes for the barrier's current phase, without an arrival.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tmem_st_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The rows of a row-wise tile, one after the other through stages of the operand ring.  128 threads cannot hold enough loads
// of their own in flight to draw an SM's share of the memory bandwidth; bulk copies, issued by thread 0 as far ahead as the
// ring holds rows, can.  Barriers in the first 2 kRowStages ints of the scratch.
constexpr uint32_t kWideRingBytes = kRingBytes + kOutBytes;
constexpr int kRowStages = 12;
struct RowStages {
  uint8_t* ring;
  uint64_t* bar;
  volatile int* abort_flag;
  uint32_t bytes, head;    // of a row; of what the tile keeps in front of the stages
  int depth, rows;
  int at = 0;              // stage of the current row
  uint32_t phase = 0;

  // Rows whose stages are not filled yet are for the caller to fetch: the first `depth`, then one per `next`.
  __device__ __forceinline__ RowStages(const LayerCtx& ctx, uint32_t row_bytes, int n_rows, int tid, uint32_t head_bytes = 0)
      : ring(ctx.ring), bar(reinterpret_cast<uint64_t*>(ctx.scratch)), abort_flag(ctx.abort_flag), bytes(row_bytes), head(head_bytes),
        depth(min(min(kRowStages, n_rows), static_cast<int>((kWideRingBytes - head_bytes) / row_bytes))), rows(n_rows) {
    fence_proxy_async_all();   // the rows may have been written, and the ring used, by plain loads and stores
    if (tid < depth) mbar_init(bar + tid, 1);
    fence_barrier_init();
    exec_sync();
  }
  __device__ __forceinline__ uint8_t* stage(int s) const { return ring + head + static_cast<uint32_t>(s) * bytes; }
  __device__ __forceinline__ bool wait() const { return mbar_wait_bounded(bar + at, phase, abort_flag, kWideWaitNs); }
  __device__ __forceinline__ void next() {
    if (++at == depth) {
      at = 0;
      phase ^= 1u;
    }
  }
  // After the last row (left == 0), or with `left` rows fetched and not waited for: their copies land, or run out of time.
  __device__ __forceinline__ void close(int tid, int left) {
    for (; left > 0; --left) {
      for (int tries = 0; tries < 1 << 16 && !mbar_try_wait(bar + at, phase); ++tries) {}
      next();
    }
    exec_sync();
    if (tid < depth) mbar_inval(bar + tid);
  }
};

}  // namespace fab
}  // namespace mf
