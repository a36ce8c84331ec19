// Host checks of csrc/coarse_index.h (built and called by test_coarse_index.py).
#include <climits>
#include <vector>

#include "coarse_index.h"

using namespace nnpp;

extern "C" {

// The growth's passes over L planes with blocks of `tiles` x `tiles` tiles: every block in range, every
// tile of every plane pair formed exactly once (i > j by symmetry counted at (j, i)); the largest grid in
// *most.  0: right.
int check_growth(int L, int tiles, long long* most) {
  std::vector<int> seen((size_t)L * L * tiles * tiles, 0);
  auto mark = [&](int i, int j, int r, int c) { ++seen[(((size_t)i * L + j) * tiles + r) * tiles + c]; };
  for (int r = 0; r < tiles; ++r)
    for (int c = 0; c < tiles; ++c) mark(0, 0, r, c);
  *most = 0;
  int s = 1;
  while (s < L) s *= 2;
  for (s /= 2; s >= 1; s /= 2) {
    const int odd = (L - 1 - s) / (2 * s) + 1, kept = (L - 1) / (2 * s) + 1;
    for (int first = 0; first < 2; ++first) {
      const GrowPass p = {s, odd, first ? odd : kept, first, tiles};
      if (p.blocks() < 1 || p.blocks() > INT_MAX) return 1;
      if (p.blocks() > *most) *most = p.blocks();
      for (int b = 0; b < (int)p.blocks(); ++b) {
        const GrowPass::Block k = p.block(b);
        if (k.i < s || k.i >= L || k.j < 0 || k.j >= L) return 2;
        if (k.row_tile < 0 || k.row_tile >= tiles || k.col_tile < 0 || k.col_tile >= tiles) return 3;
        if (first && k.j < k.i) continue;
        mark(k.i, k.j, k.row_tile, k.col_tile);
        if (k.i != k.j) mark(k.j, k.i, k.col_tile, k.row_tile);
      }
    }
  }
  for (int v : seen)
    if (v != 1) return 4;
  return 0;
}

}  // extern "C"
