// Row blocks of an expert in HBM whose tiles take two slices of bf16 weights (256 weight rows): of 256 or 128 rows, the last of what is left
// (65 to 256); in passes of few rows, of 128, and one of up to 64 behind them whose tiles take one slice.
//
// What a tile costs is mostly the operands that it loads: 64 KB a K step with 256 rows, 48 with 128, and 36 to 48 for the two slices of a
// block of up to 64 rows.  So one block of 256 takes all rows of an expert that has no more, a remainder of up to 64 rows joins
// the block before it, and larger experts are cut into blocks of 256 where the pass has many rows.  These tiles are long, and their epilogues
// are not hidden: with fewer rows, the last round of them weighs more than they save (blocks of 256 for all experts above 256 rows:
// Zipf-skewed choice, 2560 tokens 438 -> 446 us, 3328 tokens 516 -> 524; uniform 7200 tokens 984 -> 890), and with few
// rows no tile is so long (one block of 129 to 256 rows: skewed 256 tokens 173 -> 188 us, 400 tokens 200 -> 212, 700 tokens 234 -> 238).
// Layer of 128 experts, hidden 2048, width 768, top 8, microseconds with blocks of 128 rows and one of up to 64 for the rest
// throughout, and with this rule:
//   uniform choice   2304 tokens 481 -> 407, 2560 511 -> 434, 3072 514 -> 463, 3840 535 -> 514, 6600 898 -> 835, 8192 1025 -> 995
//   Zipf-skewed 1.1  2304 tokens 402 -> 411, 2560 434 -> 439, 4096 580 -> 580, 6600 866 -> 851, 8192 1022 -> 1006
// and as lane programs, the experts of a layer: 2533 tokens of prompts 395 -> 334, 3706 tokens 412 -> 381.
#pragma once

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace mf {

constexpr int kNarrowRows = 64;        // a block of up to as many rows has tiles of one slice
constexpr int kSomeRows = 8 * 1024, kManyRows = 32 * 1024;   // of a pass, over all experts

struct RowBlocks {
  int n, tall;   // blocks with tiles of two slices; of them, leading ones of 256 rows
  int rest;      // rows of a block behind them with tiles of one, or 0
};

// Of `total` rows of the pass; `tall`: blocks of more than 128 rows can be taken.
__host__ __device__ __forceinline__ RowBlocks row_blocks(int rows, int total, bool tall = true) {
  if (rows <= kNarrowRows) return RowBlocks{0, 0, rows};
  if (!tall || total < kSomeRows) {
    const int n = (rows + 128 - kNarrowRows - 1) / 128, rest = rows - 128 * n;
    return RowBlocks{n, 0, rest > 0 ? rest : 0};
  }
  if (rows <= 256) return RowBlocks{1, 0, 0};
  if (total < kManyRows) return RowBlocks{(rows + 128 - kNarrowRows - 1) / 128, 0, 0};
  const int lead = (rows - kNarrowRows - 1) / 256, left = rows - 256 * lead;   // left: 65 to 320
  return RowBlocks{lead + (left > 256 ? 2 : 1), lead, 0};
}
// Block i's first row among the expert's, and its rows.
__host__ __device__ __forceinline__ int row_block_first(RowBlocks b, int i) { return 128 * (i + (i < b.tall ? i : b.tall)); }
__host__ __device__ __forceinline__ int row_block_rows(RowBlocks b, int i, int rows) {
  return i == b.n ? b.rest : i == b.n - 1 ? rows - b.rest - row_block_first(b, i) : i < b.tall ? 256 : 128;
}

}  // namespace mf
