// coarse_inverse.cuh -- direct inverse of the coarse operator (coarse_inverse.cu).
#ifndef NNPP_COARSE_INVERSE_CUH
#define NNPP_COARSE_INVERSE_CUH

#include "common.cuh"
#include "dbuf.cuh"

namespace nnpp {

constexpr int kPlaneMax = 208;  // aggregates of a plane, the largest block one CTA inverts: kCoarseMax^(2/3)

// Work arrays of the direct inverse: planes * m * m floats each.
struct CoarseBlocks {
  int m = 0, planes = 0, axis = 2;
  DBuf<float> d, e[2], wl, wr;  // diagonal blocks, couplings (two levels), multipliers
  DBuf<float> diag;             // A_c's diagonal in plane order
  DBuf<int> bad;                // set when a pivot is too small to trust
};

// The planes of an na[0] x na[1] x na[2] aggregate grid along its longest axis; false when a
// plane has more than kPlaneMax aggregates.
bool coarse_planes(const int na[3], CoarseBlocks& b);
bool coarse_blocks_alloc(CoarseBlocks& b);

// The inverse of the operator given by its stencil rows (st[27 I + q], neighbour q of aggregate
// I) into inv (natural order, rows of stride ld), symmetrised; x is an n x n work matrix.
// rowabs[I] < 0 marks an aggregate without unknowns (its diagonal entry of the inverse is
// zeroed).  *b.bad is set on the device when a pivot fell below kPivotMin of its diagonal:
// inv must not be used then.  Asynchronous on st.
nnpp_status coarse_direct_inverse(CoarseBlocks& b, const int na[3], const float* st27, const float* rowabs, float* x,
                                  float* inv, int ld, cudaStream_t st);

}  // namespace nnpp

#endif  // NNPP_COARSE_INVERSE_CUH
