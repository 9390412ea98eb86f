"""The row blocks of an expert (monoserve_b200/csrc/row_blocks.h), compiled for the host, over every number of rows: they cover the rows in
order, of 65 to 256 rows each and at most one of fewer behind them, whichever way the pass cuts its experts."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monoserve_b200", "csrc")
CHECK = r"""
#include "row_blocks.h"
#include <cstdio>
using namespace mf;
int main() {
  const int totals[] = {0, kSomeRows - 1, kSomeRows, kManyRows - 1, kManyRows, 1 << 20};
  for (int k = 0; k < 12; ++k)
    for (int rows = 0; rows < 70000; ++rows) {
      const int total = totals[k / 2];
      const bool tall = k & 1, few = !tall || total < kSomeRows;
      const RowBlocks b = row_blocks(rows, total, tall);
      if (rows <= kNarrowRows) {   // no rows among them: an expert whose tiles are not written, for want of room, has none
        if (b.n || b.tall || b.rest != rows) return printf("rows %d of %d: %d blocks\n", rows, total, b.n), 1;
        continue;
      }
      int at = 0;
      for (int i = 0; i < b.n; ++i) {
        const int n = row_block_rows(b, i, rows);
        if (row_block_first(b, i) != at || n <= kNarrowRows || n > (few ? 128 : 256)) return printf("rows %d of %d, block %d\n", rows, total, i), 1;
        if (total < kManyRows && rows > 256 && i < b.n - 1 && n != 128) return printf("rows %d: block %d of %d rows\n", rows, i, n), 1;
        at += n;
      }
      if (b.rest && (!few || b.rest > kNarrowRows || row_block_rows(b, b.n, rows) != b.rest || row_block_first(b, b.n) != at))
        return printf("rows %d of %d: a rest of %d\n", rows, total, b.rest), 1;
      if (at + b.rest != rows || b.n < 1 || b.tall > b.n) return printf("rows %d of %d: %d\n", rows, total, at), 1;
    }
  return 0;
}
"""


def test_blocks_cover_the_rows(tmp_path):
    (tmp_path / "check.cpp").write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")], check=True)
    r = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
