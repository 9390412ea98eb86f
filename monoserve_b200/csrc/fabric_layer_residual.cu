// The plain residual of the layer-list decoders, normed before and after each sublayer (fabric_layer_tiles.cuh).
#include "fabric_layer_tiles.cuh"
#include "wide_tile.cuh"

namespace mf {
namespace fab {

// Kind 66, ResidualArgs: rows [i0, i0 + i1), the four exec warps on one row.

// Sums of two values over the exec threads.  Successive reductions of a row use scratch of their own, so that one barrier
// each is enough.
__device__ __forceinline__ void block_sum2(float& a, float& b, float* red, int tid) {
  a = warp_sum(a);
  b = warp_sum(b);
  if ((tid & 31) == 0) {
    red[tid >> 5] = a;
    red[4 + (tid >> 5)] = b;
  }
  exec_sync();
  a = red[0] + red[1] + red[2] + red[3];
  b = red[4] + red[5] + red[6] + red[7];
}

// Column piece c of a sublayer's output: its K-range slabs added in order.
template <int V>
__device__ __forceinline__ void slab_sum(unsigned long long base, uint32_t parts, size_t slab, size_t at, float (&y)[V]) {
  const float* p = f32p(base) + at;
  ld_vec<V>(p, y);
  for (uint32_t q0 = 1; q0 < parts; q0 += 4) {   // four slabs' loads are issued before the first is used
    float b[4][V];
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) ld_vec<V>(p + min(q0 + i, parts - 1) * slab, b[i]);
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
      if (q0 + i < parts)
#pragma unroll
        for (int j = 0; j < V; ++j) y[j] += b[i][j];
  }
}

__device__ __forceinline__ float over_rms(float ss, const ResidualArgs& A) { return 1.f / sqrtf(ss / static_cast<float>(A.W) + A.eps); }

// Columns c .. c + V of the next sublayer's input.
template <int V>
__device__ __forceinline__ void put_input(const ResidualArgs& A, uint32_t r, int g, int c, const float (&h)[V]) {
  auto st16 = [&](unsigned long long base, size_t at) {
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(base) + at;
    if constexpr (V == 4) {
      const __nv_bfloat162 q[2] = {__floats2bfloat162_rn(h[0], h[1]), __floats2bfloat162_rn(h[2], h[3])};
      *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(q);
    } else {
      o[0] = __float2bfloat16(h[0]);
    }
  };
  if (A.h16) st16(A.h16, static_cast<size_t>(r) * A.ld_h16 + c);
  if (A.h32) st_vec<V>(reinterpret_cast<float*>(A.h32) + static_cast<size_t>(r) * A.ld_h32 + c, h);
  if (g >= 0 && A.out16) st16(A.out16, static_cast<size_t>(g) * A.ld_out + c);
  if (g >= 0 && A.out32) st_vec<V>(reinterpret_cast<float*>(A.out32) + static_cast<size_t>(g) * A.ld_out + c, h);
}

// Any width, and the embedding: a row is read again in each pass, x holding what the pass before has made of it (a thread
// keeps to its own columns).
template <int V>
__device__ __noinline__ void residual_rows(const TileDesc& t, int tid, int* scratch) {
  ResidualArgs A;
  load_block(A, t.a[0]);
  StepArgs St{};
  if (A.step) load_block(St, A.step);
  const int page = St.page_size ? static_cast<int>(St.page_size) : 64;
  const int W = static_cast<int>(A.W);
  const size_t slab = static_cast<size_t>(A.y_rows) * W;
  float* const red = reinterpret_cast<float*>(scratch);   // three reductions of a row, eight floats each
  for (uint32_t r = t.i0; r < t.i0 + t.i1; ++r) {
    float* const xr = reinterpret_cast<float*>(A.x) + static_cast<size_t>(r) * W;
    float* const sum_out = A.sum_out ? reinterpret_cast<float*>(A.sum_out) + static_cast<size_t>(r) * W : nullptr;
    float s0 = 0.f, s1 = 0.f;
    float x[V], y[V], z[V];
    if (A.embed) {
      int token, pos;
      if (A.step) {
        const int slot = reinterpret_cast<const int*>(St.row_req)[r];
        pos = min(reinterpret_cast<const int*>(St.seq_len)[slot], static_cast<int>(St.bt_stride) * page - 1);
        token = reinterpret_cast<const int*>(St.last_token)[slot];
        exec_sync();   // every thread has the position: the row's bookkeeping may advance it
        if (tid == 0) step_row(St, page, static_cast<int>(r), 0);
      } else {
        pos = reinterpret_cast<const int*>(A.tok_pos)[r];
        token = reinterpret_cast<const int*>(A.tokens)[r];
      }
      pos = min(pos, static_cast<int>(A.max_pos) - 1);
      const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(A.embed) + static_cast<size_t>(token) * W;
      const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(A.pos) + static_cast<size_t>(pos) * W;
#pragma unroll 4
      for (int c = tid * V; c < W; c += kExecThreads * V) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
          x[j] = __bfloat162float(e[c + j]) * A.embed_scale + (A.pos ? __bfloat162float(p[c + j]) : 0.f);
          s0 = fmaf(x[j], x[j], s0);
        }
        st_vec<V>(xr + c, x);
        if (sum_out) st_vec<V>(sum_out + c, x);
      }
    } else {
      float inv0 = 1.f, inv1 = 1.f;
      auto load_y = [&](int c) {
        slab_sum<V>(A.y0, A.y0_parts, slab, static_cast<size_t>(r) * W + c, y);
        if (A.y1_parts) slab_sum<V>(A.y1, A.y1_parts, slab, static_cast<size_t>(r) * W + c, z);
      };
      auto branches = [&](int c) {   // y = branch_scale (w0 norm(y0) + w1 norm(y1))
        float a[V], b[V];
        ld_vec<V>(f32p(A.w0) + c, a);
        ld_vec<V>(f32p(A.w1) + c, b);
#pragma unroll
        for (int j = 0; j < V; ++j) y[j] = A.branch_scale * (y[j] * inv0 * a[j] + z[j] * inv1 * b[j]);
      };
      for (int c = tid * V; c < W; c += kExecThreads * V) {
        load_y(c);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          s0 = fmaf(y[j], y[j], s0);
          if (A.y1_parts) s1 = fmaf(z[j], z[j], s1);
        }
      }
      block_sum2(s0, s1, red, tid);
      if (A.y1_parts) {
        inv0 = over_rms(s0, A);
        inv1 = over_rms(s1, A);
        s0 = s1 = 0.f;
        for (int c = tid * V; c < W; c += kExecThreads * V) {
          load_y(c);
          branches(c);
#pragma unroll
          for (int j = 0; j < V; ++j) s0 = fmaf(y[j], y[j], s0);
        }
        block_sum2(s0, s1, red + 8, tid);
      }
      const float inv = over_rms(s0, A);
      s0 = s1 = 0.f;
      for (int c = tid * V; c < W; c += kExecThreads * V) {
        float w[V];
        ld_vec<V>(xr + c, x);
        load_y(c);
        if (A.y1_parts) branches(c);
        ld_vec<V>(f32p(A.post_w) + c, w);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          x[j] += y[j] * inv * w[j];
          s0 = fmaf(x[j], x[j], s0);
        }
        st_vec<V>(xr + c, x);
        if (sum_out) st_vec<V>(sum_out + c, x);
      }
    }
    block_sum2(s0, s1, red + 16, tid);
    const float inv = over_rms(s0, A);
    const int g = A.gather ? reinterpret_cast<const int*>(A.gather)[r] : -1;
#pragma unroll 4
    for (int c = tid * V; c < W; c += kExecThreads * V) {
      float h[V];
      ld_vec<V>(xr + c, x);
      ld_vec<V>(f32p(A.w) + c, h);
#pragma unroll
      for (int j = 0; j < V; ++j) h[j] = x[j] * inv * h[j];
      put_input<V>(A, r, g, c, h);
    }
  }
}

// Rows of at most 512 NU columns, kept in registers; the next row's loads are issued before this one's arithmetic.
template <int NU, bool kTwo>
__device__ __noinline__ void residual_rows_ahead(const TileDesc& t, int tid, int* scratch) {
  ResidualArgs A;
  load_block(A, t.a[0]);
  const int W = static_cast<int>(A.W);
  const size_t slab = static_cast<size_t>(A.y_rows) * W;
  float* const red = reinterpret_cast<float*>(scratch);
  float x[NU][4], y[NU][4], z[kTwo ? NU : 1][4];           // this row
  float nx[NU][4], ny[NU][4], nz[kTwo ? NU : 1][4];        // the next
  int g = -1;
  auto each = [&](auto&& f) {   // f(register piece, first column)
#pragma unroll
    for (int i = 0; i < NU; ++i)
      if ((tid + i * kExecThreads) * 4 < W) f(i, (tid + i * kExecThreads) * 4);
  };
  auto load = [&](uint32_t r) {
    each([&](int i, int c) {
      const size_t at = static_cast<size_t>(r) * W + c;
      ld_vec<4>(f32p(A.x) + at, nx[i]);
      slab_sum<4>(A.y0, A.y0_parts, slab, at, ny[i]);
      if constexpr (kTwo) slab_sum<4>(A.y1, A.y1_parts, slab, at, nz[i]);
    });
  };
  load(t.i0);
  for (uint32_t r = t.i0; r < t.i0 + t.i1; ++r) {
#pragma unroll
    for (int i = 0; i < NU; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i][j] = nx[i][j];
        y[i][j] = ny[i][j];
        if constexpr (kTwo) z[i][j] = nz[i][j];
      }
    if (A.gather) g = reinterpret_cast<const int*>(A.gather)[r];
    float s0 = 0.f, s1 = 0.f;
    each([&](int i, int) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s0 = fmaf(y[i][j], y[i][j], s0);
        if constexpr (kTwo) s1 = fmaf(z[i][j], z[i][j], s1);
      }
    });
    if (r + 1 < t.i0 + t.i1) load(r + 1);
    block_sum2(s0, s1, red, tid);
    if constexpr (kTwo) {
      const float inv0 = over_rms(s0, A), inv1 = over_rms(s1, A);
      s0 = s1 = 0.f;
      each([&](int i, int c) {
        float a[4], b[4];
        ld_vec<4>(f32p(A.w0) + c, a);
        ld_vec<4>(f32p(A.w1) + c, b);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          y[i][j] = A.branch_scale * (y[i][j] * inv0 * a[j] + z[i][j] * inv1 * b[j]);
          s0 = fmaf(y[i][j], y[i][j], s0);
        }
      });
      block_sum2(s0, s1, red + 8, tid);
    }
    const float inv = over_rms(s0, A);
    s0 = s1 = 0.f;
    each([&](int i, int c) {
      float w[4];
      ld_vec<4>(f32p(A.post_w) + c, w);
      const size_t at = static_cast<size_t>(r) * W + c;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i][j] += y[i][j] * inv * w[j];
        s0 = fmaf(x[i][j], x[i][j], s0);
      }
      st_vec<4>(reinterpret_cast<float*>(A.x) + at, x[i]);
      if (A.sum_out) st_vec<4>(reinterpret_cast<float*>(A.sum_out) + at, x[i]);
    });
    block_sum2(s0, s1, red + 16, tid);
    const float inv_x = over_rms(s0, A);
    each([&](int i, int c) {
      float h[4];
      ld_vec<4>(f32p(A.w) + c, h);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = x[i][j] * inv_x * h[j];
      put_input<4>(A, r, g, c, h);
    });
  }
}

// The same rows through RowStages.  Bound by memory (a row of 2048 with one branch: 16 KB in, 12 KB out); 4096 such rows:
// 118 -> 68 us, with two branches 174 -> 105.
template <int NU, bool kTwo>
__device__ __noinline__ bool residual_bulk(const TileDesc& t, int tid, const LayerCtx& ctx) {
  __builtin_assume(__isShared(ctx.ring));
  __builtin_assume(__isShared(ctx.scratch));
  ResidualArgs A;
  load_block(A, t.a[0]);
  const int W = static_cast<int>(A.W), parts0 = static_cast<int>(A.y0_parts), parts1 = kTwo ? static_cast<int>(A.y1_parts) : 0;
  const int row0 = static_cast<int>(t.i0), rows = static_cast<int>(t.i1);
  const uint32_t piece = static_cast<uint32_t>(W) * 4;
  float* const red = reinterpret_cast<float*>(ctx.scratch) + 64;
  // the weights stay in the ring: what it leaves of the L1 does not hold them from one row to the next
  constexpr int kWeights = kTwo ? 4 : 2;
  RowStages pipe(ctx, static_cast<uint32_t>(1 + parts0 + parts1) * piece, rows, tid, kWeights * piece);
  const float* const weights = reinterpret_cast<const float*>(ctx.ring);   // post_w, w, w0, w1
  auto fetch = [&](int k, int s) {
    const size_t r = static_cast<size_t>(row0 + k);
    uint8_t* to = pipe.stage(s);
    mbar_arrive_expect_tx(pipe.bar + s, pipe.bytes);
    bulk_in(to, f32p(A.x) + r * W, piece, pipe.bar + s);
    for (int q = 0; q < parts0; ++q)
      bulk_in(to += piece, f32p(A.y0) + (static_cast<size_t>(q) * A.y_rows + r) * W, piece, pipe.bar + s);
    for (int q = 0; q < parts1; ++q)
      bulk_in(to += piece, f32p(A.y1) + (static_cast<size_t>(q) * A.y_rows + r) * W, piece, pipe.bar + s);
  };
  if (tid == 0) {
    mbar_expect_tx(pipe.bar, kWeights * piece);   // with the first row
    const unsigned long long from[4] = {A.post_w, A.w, A.w0, A.w1};
#pragma unroll
    for (int i = 0; i < kWeights; ++i) bulk_in(ctx.ring + i * piece, f32p(from[i]), piece, pipe.bar);
    for (int k = 0; k < pipe.depth; ++k) fetch(k, k);
  }
  auto each = [&](auto&& f) {   // f(register piece, first column)
#pragma unroll
    for (int i = 0; i < NU; ++i)
      if ((tid + i * kExecThreads) * 4 < W) f(i, (tid + i * kExecThreads) * 4);
  };
  int k = 0;
  bool ok = true;
  for (; k < rows; ++k) {
    const uint32_t r = static_cast<uint32_t>(row0 + k);
    const int g = A.gather ? reinterpret_cast<const int*>(A.gather)[r] : -1;
    float x[NU][4], y[NU][4], z[kTwo ? NU : 1][4];
    float s0 = 0.f, s1 = 0.f;
    ok = pipe.wait();
    const float* const in = reinterpret_cast<const float*>(pipe.stage(pipe.at));
    auto slabs = [&](const float* p, int parts, float (&v)[4]) {
      ld_vec<4>(p, v);
      for (int q = 1; q < parts; ++q) {
        float b[4];
        ld_vec<4>(p + q * W, b);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += b[j];
      }
    };
    if (ok)
      each([&](int i, int c) {
        ld_vec<4>(in + c, x[i]);
        slabs(in + W + c, parts0, y[i]);
        if constexpr (kTwo) slabs(in + (1 + parts0) * W + c, parts1, z[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s0 = fmaf(y[i][j], y[i][j], s0);
          if constexpr (kTwo) s1 = fmaf(z[i][j], z[i][j], s1);
        }
      });
    // this barrier also carries the decision to go on and the stage's release
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if ((tid & 31) == 0) {
      red[tid >> 5] = s0;
      red[4 + (tid >> 5)] = s1;
    }
    ok = exec_and(ok);
    if (!ok) break;
    if (tid == 0 && k + pipe.depth < rows) {
      fence_proxy_async_smem();
      fetch(k + pipe.depth, pipe.at);
    }
    pipe.next();
    s0 = red[0] + red[1] + red[2] + red[3];
    s1 = red[4] + red[5] + red[6] + red[7];
    if constexpr (kTwo) {
      const float inv0 = over_rms(s0, A), inv1 = over_rms(s1, A);
      s0 = s1 = 0.f;
      each([&](int i, int c) {
        float a[4], b[4];
        ld_vec<4>(weights + 2 * W + c, a);
        ld_vec<4>(weights + 3 * W + c, b);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          y[i][j] = A.branch_scale * (y[i][j] * inv0 * a[j] + z[i][j] * inv1 * b[j]);
          s0 = fmaf(y[i][j], y[i][j], s0);
        }
      });
      block_sum2(s0, s1, red + 8, tid);
    }
    const float inv = over_rms(s0, A);
    s0 = s1 = 0.f;
    each([&](int i, int c) {
      float w[4];
      ld_vec<4>(weights + c, w);
      const size_t at = static_cast<size_t>(r) * W + c;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i][j] += y[i][j] * inv * w[j];
        s0 = fmaf(x[i][j], x[i][j], s0);
      }
      st_vec<4>(reinterpret_cast<float*>(A.x) + at, x[i]);
      if (A.sum_out) st_vec<4>(reinterpret_cast<float*>(A.sum_out) + at, x[i]);
    });
    block_sum2(s0, s1, red + 16, tid);
    const float inv_x = over_rms(s0, A);
    each([&](int i, int c) {
      float h[4];
      ld_vec<4>(weights + W + c, h);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = x[i][j] * inv_x * h[j];
      put_input<4>(A, r, g, c, h);
    });
  }
  pipe.close(tid, ok ? 0 : min(rows - k, pipe.depth));
  return ok;
}

// The embedding of rows of at most 512 NU columns, through RowStages as well: the token's row and its position's.
template <int NU>
__device__ __noinline__ bool residual_embed(const TileDesc& t, int tid, const LayerCtx& ctx) {
  __builtin_assume(__isShared(ctx.ring));
  __builtin_assume(__isShared(ctx.scratch));
  ResidualArgs A;
  load_block(A, t.a[0]);
  const int W = static_cast<int>(A.W), row0 = static_cast<int>(t.i0), rows = static_cast<int>(t.i1);
  const uint32_t piece = static_cast<uint32_t>(W) * 2;
  float* const red = reinterpret_cast<float*>(ctx.scratch) + 64;
  int2* const at = reinterpret_cast<int2*>(ctx.scratch + 128);   // token and position of each row
  for (int k = tid; k < rows; k += kExecThreads)
    at[k] = make_int2(reinterpret_cast<const int*>(A.tokens)[row0 + k],
                      min(reinterpret_cast<const int*>(A.tok_pos)[row0 + k], static_cast<int>(A.max_pos) - 1));
  RowStages pipe(ctx, (A.pos ? 2 : 1) * piece, rows, tid, 2 * piece);
  const float* const weights = reinterpret_cast<const float*>(ctx.ring);
  auto fetch = [&](int k, int s) {
    uint8_t* const to = pipe.stage(s);
    const int2 x = at[k];
    mbar_arrive_expect_tx(pipe.bar + s, pipe.bytes);
    bulk_in(to, reinterpret_cast<const __nv_bfloat16*>(A.embed) + static_cast<size_t>(x.x) * W, piece, pipe.bar + s);
    if (A.pos) bulk_in(to + piece, reinterpret_cast<const __nv_bfloat16*>(A.pos) + static_cast<size_t>(x.y) * W, piece, pipe.bar + s);
  };
  if (tid == 0) {
    mbar_expect_tx(pipe.bar, 2 * piece);   // with the first row
    bulk_in(ctx.ring, f32p(A.w), 2 * piece, pipe.bar);
    for (int k = 0; k < pipe.depth; ++k) fetch(k, k);
  }
  int k = 0;
  bool ok = true;
  for (; k < rows; ++k) {
    const uint32_t r = static_cast<uint32_t>(row0 + k);
    const int g = A.gather ? reinterpret_cast<const int*>(A.gather)[r] : -1;
    float x[NU][4], ss = 0.f;
    ok = pipe.wait();
    const __nv_bfloat16* const in = reinterpret_cast<const __nv_bfloat16*>(pipe.stage(pipe.at));
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int c = (tid + i * kExecThreads) * 4;
      if (c >= W || !ok) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i][j] = __bfloat162float(in[c + j]) * A.embed_scale + (A.pos ? __bfloat162float(in[W + c + j]) : 0.f);
        ss = fmaf(x[i][j], x[i][j], ss);
      }
      const size_t to = static_cast<size_t>(r) * W + c;
      st_vec<4>(reinterpret_cast<float*>(A.x) + to, x[i]);
      if (A.sum_out) st_vec<4>(reinterpret_cast<float*>(A.sum_out) + to, x[i]);
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red[(k & 1) * 4 + (tid >> 5)] = ss;
    ok = exec_and(ok);
    if (!ok) break;
    if (tid == 0 && k + pipe.depth < rows) {
      fence_proxy_async_smem();
      fetch(k + pipe.depth, pipe.at);
    }
    pipe.next();
    const float* const sums = red + (k & 1) * 4;
    const float inv = over_rms(sums[0] + sums[1] + sums[2] + sums[3], A);
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int c = (tid + i * kExecThreads) * 4;
      if (c >= W) continue;
      float h[4];
      ld_vec<4>(weights + c, h);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = x[i][j] * inv * h[j];
      put_input<4>(A, r, g, c, h);
    }
  }
  pipe.close(tid, ok ? 0 : min(rows - k, pipe.depth));
  return ok;
}

__device__ bool tile_residual(const TileDesc& t, int tid, const LayerCtx& ctx) {
  int* const scratch = ctx.scratch;
  const ResidualArgs* p = reinterpret_cast<const ResidualArgs*>(t.a[0]);
  const uint32_t W = __ldcg(&p->W);
  const bool two = __ldcg(&p->y1_parts) != 0, embed = __ldcg(&p->embed) != 0, four = (W & 3) == 0;
  // (The rows are asked for first: what a step's few rows read of the block here, they wait for.  A pass of two sequences of
  // Teganex, seven such stages: 878 -> 871 us.)
  if (t.i1 >= kBulkRows) {
    const uint32_t parts0 = __ldcg(&p->y0_parts), parts1 = __ldcg(&p->y1_parts);
    // (W % 8: whole 16-byte pieces of bf16 rows)
    if (embed && __ldcg(&p->step) == 0 && t.i1 <= 256 && (W & 7) == 0 && W <= 4096 &&
        ((__ldcg(&p->embed) | __ldcg(&p->pos)) & 15) == 0)
      return W <= 2048 ? residual_embed<4>(t, tid, ctx) : residual_embed<8>(t, tid, ctx);
    // two rows in the ring at least, or nothing overlaps
    if (!embed && four && W <= 4096 && parts0 > 0 && (2 * (1 + parts0 + parts1) + (two ? 4 : 2)) * W * 4 <= kWideRingBytes) {
      if (W <= 2048) return two ? residual_bulk<4, true>(t, tid, ctx) : residual_bulk<4, false>(t, tid, ctx);
      return two ? residual_bulk<8, true>(t, tid, ctx) : residual_bulk<8, false>(t, tid, ctx);
    }
  }
  if (!embed && four && W <= 2048) {
    if (two) residual_rows_ahead<4, true>(t, tid, scratch);
    else residual_rows_ahead<4, false>(t, tid, scratch);
  } else if (!embed && four && W <= 4096) {
    if (two) residual_rows_ahead<8, true>(t, tid, scratch);
    else residual_rows_ahead<8, false>(t, tid, scratch);
  } else if (four) {
    residual_rows<4>(t, tid, scratch);
  } else {
    residual_rows<1>(t, tid, scratch);
  }
  return true;
}

}  // namespace fab
}  // namespace mf
