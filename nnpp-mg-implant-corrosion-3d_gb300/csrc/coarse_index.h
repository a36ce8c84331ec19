// coarse_index.h -- index arithmetic of the coarse operator's kernels, host and device alike (plain C++, so
// that its limits are checked without a GPU: tests/test_coarse_index.py).
#ifndef NNPP_COARSE_INDEX_H
#define NNPP_COARSE_INDEX_H

#ifdef __CUDACC__
#define NNPP_HD __host__ __device__ __forceinline__
#else
#define NNPP_HD inline
#endif

namespace nnpp {

// The blocks of one pass of the inverse's growth over a level of stride s: plane pairs (i, j),
// i = s (2 t + 1) for t < rows and j = s (2 u + first) for u < cols, times the tiles x tiles tiles of a
// plane's block.  They are one list along gridDim.x (2^31 - 1 blocks): a long, thin domain has up to 1024
// planes (kMaxAxisBins) and so 512 x 512 pairs, and gridDim.z ends at 65535, which 512 planes pass.
struct GrowPass {
  int s, rows, cols, first, tiles;
  struct Block {
    int i, j, row_tile, col_tile;
  };
  NNPP_HD long long blocks() const { return (long long)rows * cols * tiles * tiles; }
  NNPP_HD Block block(int b) const {
    const int tt = tiles * tiles, pair = b / tt, tile = b - pair * tt, t = pair / cols, u = pair - t * cols;
    return Block{s * (2 * t + 1), s * (2 * u + first), tile / tiles, tile % tiles};
  }
};

}  // namespace nnpp

#endif  // NNPP_COARSE_INDEX_H
