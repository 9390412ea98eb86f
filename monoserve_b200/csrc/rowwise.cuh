// Warp-level row routines shared by the stream-launched kernels and the fabric's
// row-wise tiles: routing of one token, and the RMSNorm of one row.  Their results
// are defined bit for bit (detmath.cuh), so the oracle can be compared exactly.
#pragma once
#include <cuda_bf16.h>

#include "detmath.cuh"
#include "types.h"

namespace mf {

__device__ __forceinline__ void unpack8(const uint4& u, float f[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 pack8(const float f[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// Router projection of R tokens x C experts by one warp: logits[t][e] = sum_h x[t][h] wr[e][h] in the order that defines its
// bits: lane l sums h = 256 j + 8 l + i (j outer, i = 0..7 inner) in one fmaf chain, the 32 sums are added by the xor
// butterfly 16, 8, 4, 2, 1 (a sum of two lanes is the same in both, so each lane may keep half of its values at a step and
// the R C sums take R C + log steps, not five each).  Bound by the fp32 units; at one expert a token row (C = 1) it was
// bound by the loads and conversions of the weights, one per product.  The products of two experts go as packed pairs, each
// half rounded like the scalar instruction, which leaves issue slots to the conversions.  kAhead: the next 256 columns'
// loads are issued before this one's products (a lone warp per scheduler has nothing else to hide them behind).  kShared: x
// and wr are in shared memory.
// 8192 tokens x 128 experts, H = 2048: 326 -> 145 us; one token 16 -> 6.5.
namespace logits {

using Pair = unsigned long long;
__device__ __forceinline__ Pair pair(uint32_t a, uint32_t b) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ Pair fma_pair(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// N values per lane, N a power of two: lane l ends with the sum over the warp of value l / (32 / N) (N <= 32).
template <int N>
__device__ __forceinline__ float sum_each(float (&v)[N], int lane) {
#pragma unroll
  for (int half = N / 2, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
    const bool hi = lane & bit;
#pragma unroll
    for (int c = 0; c < half; ++c) {
      const float give = hi ? v[c] : v[c + half], have = hi ? v[c + half] : v[c];
      v[c] = __fadd_rn(have, __shfl_xor_sync(0xffffffffu, give, bit));
    }
  }
#pragma unroll
  for (int bit = 16 / N; bit >= 1; bit >>= 1) v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], bit));
  return v[0];
}

template <int R, int C>
struct Columns {   // 8 columns a lane of R token rows and C weight rows
  uint4 x[R], w[C];
};

template <int R, int C>
struct Sums {
  static_assert(R * C <= 32 && (C == 1 || C % 2 == 0), "a sum per lane, experts in pairs");
  static constexpr int P = C > 1 ? C / 2 : 1;
  Pair acc[R][P];   // C = 1: the upper halves stay zero
  __device__ __forceinline__ Sums() {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < P; ++p) acc[r][p] = 0ull;
  }
  __device__ __forceinline__ void multiply(const Columns<R, C>& k) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {   // a word: columns 2 q and 2 q + 1
      auto word = [&](const uint4& v) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; };
      Pair lo[P], hi[P];
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const uint32_t a = word(k.w[p * 2]), b = C > 1 ? word(k.w[C > 1 ? p * 2 + 1 : 0]) : 0u;
        lo[p] = pair(a << 16, b << 16);
        hi[p] = pair(a & 0xffff0000u, b & 0xffff0000u);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t v = word(k.x[r]);
        const Pair x_lo = pair(v << 16, v << 16), x_hi = pair(v & 0xffff0000u, v & 0xffff0000u);
#pragma unroll
        for (int p = 0; p < P; ++p) acc[r][p] = fma_pair(x_lo, lo[p], acc[r][p]);
#pragma unroll
        for (int p = 0; p < P; ++p) acc[r][p] = fma_pair(x_hi, hi[p], acc[r][p]);
      }
    }
  }
  // Tokens [t0, t_end) (at most R), experts [e0, e_end) (at most C).
  __device__ __forceinline__ void store(float* out, int E, int t0, int t_end, int e0, int e_end) {
    const int lane = threadIdx.x & 31;
    float v[R * C];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < P; ++p) {
        v[r * C + 2 * p] = __uint_as_float(static_cast<uint32_t>(acc[r][p]));
        if constexpr (C > 1) v[r * C + 2 * p + 1] = __uint_as_float(static_cast<uint32_t>(acc[r][p] >> 32));
      }
    const float sum = sum_each<R * C>(v, lane);
    constexpr int kPer = 32 / (R * C);
    const int n = lane / kPer, t = t0 + n / C, e = e0 + n % C;
    if (lane % kPer == 0 && t < t_end && e < e_end) out[static_cast<size_t>(t) * E + e] = sum;
  }
};

}  // namespace logits

// Tokens [t0, t_end) (at most R of them; the last is repeated for those missing), experts [e0, e_end) (at most C).
template <int R, int C, bool kAhead, bool kShared = false>
__device__ __forceinline__ void router_block(const __nv_bfloat16* x, const __nv_bfloat16* wr, float* out, int H, int E, int t0,
                                             int t_end, int e0, int e_end) {
  using namespace logits;
  const int lane = threadIdx.x & 31, nj = H / 256;
  const uint4 *xp[R], *wp[C];
#pragma unroll
  for (int r = 0; r < R; ++r) xp[r] = reinterpret_cast<const uint4*>(x + static_cast<size_t>(min(t0 + r, t_end - 1)) * H) + lane;
#pragma unroll
  for (int c = 0; c < C; ++c) wp[c] = reinterpret_cast<const uint4*>(wr + static_cast<size_t>(min(e0 + c, e_end - 1)) * H) + lane;
  auto load = [&](int j, Columns<R, C>& k) {
#pragma unroll
    for (int r = 0; r < R; ++r) k.x[r] = xp[r][32 * j];
#pragma unroll
    for (int c = 0; c < C; ++c) k.w[c] = kShared ? wp[c][32 * j] : __ldg(wp[c] + 32 * j);
  };
  Sums<R, C> sums;
  if constexpr (kAhead) {
    Columns<R, C> k, next;
    load(0, next);
#pragma unroll 1
    for (int j = 0; j < nj; ++j) {
      k = next;
      load(min(j + 1, nj - 1), next);
      sums.multiply(k);
    }
  } else {
#pragma unroll(R * C >= 16 ? 1 : 8 / R)
    for (int j = 0; j < nj; ++j) {
      Columns<R, C> k;
      load(j, k);
      sums.multiply(k);
    }
  }
  sums.store(out, E, t0, t_end, e0, e_end);
}

// Routing of one token by one warp: what the reference's router tile computes
// (csrc/fabric/tiles/aux.cuh:326-417): scores = softmax of the E <= 256 logits, or their sigmoid with
// an optional selection bias; K <= 16 picks, each the best remaining selection score with the lowest
// expert id winning ties; weights = the picks' scores, renormalised by their sum taken in pick
// order, times `scale`.  Lane k < K returns pick k in (pick_id, pick_weight).  zero_logits: clear the
// row once read.
//
// Lane l holds experts l, l + 32, ... (slot i = expert l + 32 i).  The floating-point order is part
// of the result's definition (the oracle repeats it): row maximum (any order: max is exact), per lane
// the exponentials summed over its slots in slot order, the lanes' sums by the xor butterfly 16..1,
// one IEEE division per score.  The K arg-max rounds only compare, so they are done on integers:
// a score and its expert id become one 64-bit key whose order is (score ascending, id descending).
namespace route {

constexpr int kSlots = kMaxExperts / 32;
constexpr float kAbsent = -1e30f;   // stands in for experts past E

// 32-bit pattern whose unsigned order is the order of the (non-NaN) floats.
__device__ __forceinline__ unsigned int ordered_bits(float v) {
  const unsigned int u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ unsigned long long pick_key(float score, int expert) {
  return (static_cast<unsigned long long>(ordered_bits(score)) << 32) | (0xffffffffu - static_cast<unsigned int>(expert));
}
__device__ __forceinline__ int key_expert(unsigned long long key) { return static_cast<int>(0xffffffffu - static_cast<unsigned int>(key)); }

// Two reductions of 32-bit words: the scores, then the experts of the lanes that hold the best one.  (Five exchanges of 64-bit
// keys, each waiting for the one before, were most of a row's routing.)  Every lane's key is zero or has a nonzero lower word.
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
  const uint32_t score = static_cast<uint32_t>(k >> 32), best = __reduce_max_sync(0xffffffffu, score);
  const uint32_t expert = __reduce_max_sync(0xffffffffu, score == best ? static_cast<uint32_t>(k) : 0u);
  return static_cast<unsigned long long>(best) << 32 | expert;
}

}  // namespace route

__device__ __forceinline__ void route_row(float* logits_row, const float* bias, int E, int K, int scoring, int renorm,
                                          float scale, int zero_logits, int& pick_id, float& pick_weight) {
  using namespace route;
  const int lane = threadIdx.x & 31;
  float score[kSlots];
#pragma unroll
  for (int i = 0; i < kSlots; ++i) {
    const int expert = lane + 32 * i;
    score[i] = expert < E ? logits_row[expert] : kAbsent;
    if (zero_logits && expert < E) logits_row[expert] = 0.f;
  }
  unsigned long long key[kSlots];   // selection key per slot; 0 once picked (below every real key)
  if (scoring == 0) {
    float top = kAbsent;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) top = fmaxf(top, score[i]);
#pragma unroll
    for (int o = 16; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    float lane_sum = 0.f;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      score[i] = det_expf(__fsub_rn(score[i], top));   // an absent expert gives exactly 0
      lane_sum = __fadd_rn(lane_sum, score[i]);
    }
    const float total = warp_sum_xor(lane_sum);
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      score[i] = __fdiv_rn(score[i], total);
      key[i] = pick_key(lane + 32 * i < E ? score[i] : kAbsent, lane + 32 * i);
    }
  } else {
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      const int expert = lane + 32 * i;
      score[i] = det_sigmoidf(score[i]);
      key[i] = pick_key(expert < E ? __fadd_rn(score[i], bias ? bias[expert] : 0.f) : kAbsent, expert);
    }
  }
  pick_id = 0;
  float mine = 0.f, picked_sum = 0.f;
  for (int k = 0; k < K; ++k) {
    unsigned long long best = 0;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) best = key[i] > best ? key[i] : best;
    const int expert = key_expert(warp_max_key(best));
    // the lane that holds the pick takes it out of the running and hands its score round
    float held = 0.f;
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
      if (lane + 32 * i == expert) {
        held = score[i];
        key[i] = 0;
      }
    const float weight = __shfl_sync(0xffffffffu, held, expert & 31);
    if (lane == k) {
      pick_id = expert;
      mine = weight;
    }
    picked_sum = __fadd_rn(picked_sum, weight);
  }
  pick_weight = __fmul_rn(renorm ? __fdiv_rn(mine, picked_sum) : mine, scale);
}

// RMSNorm of a bf16 row that this warp holds in `x` (H elements, lane l owns the
// 8-element groups l, l + 32, ...): out = bf16(bf16(x * inv) * w), inv = 1 / sqrt(ss / H + eps)
// with correctly rounded square root and divide (csrc/fabric/tiles/aux.cuh:60-122 uses
// rsqrtf).  ss is this lane's partial sum of squares, accumulated by the caller with
// one fmaf per element in storage order.  out2 optionally receives a copy.
__device__ __forceinline__ void norm_store_row(const uint4* x, float ss, const __nv_bfloat16* norm_w,
                                               __nv_bfloat16* out, __nv_bfloat16* out2, int H, float eps) {
  const int lane = threadIdx.x & 31, n16 = H / 8;
  ss = warp_sum_xor(ss);
  const float inv = det_rsqrtf(__fadd_rn(__fdiv_rn(ss, static_cast<float>(H)), eps));
  __syncwarp();
  const uint4* w4 = reinterpret_cast<const uint4*>(norm_w);
  uint4* o = reinterpret_cast<uint4*>(out);
  uint4* o2 = reinterpret_cast<uint4*>(out2);
  for (int c = lane; c < n16; c += 32) {
    float f[8], g[8];
    unpack8(x[c], f);
    unpack8(w4[c], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __fmul_rn(round_bf16(__fmul_rn(f[j], inv)), g[j]);
    const uint4 v = pack8(f);
    o[c] = v;
    if (o2) o2[c] = v;
  }
}

}  // namespace mf
