// coarse_inverse.cu -- the dense inverse of the coarse operator by block cyclic reduction.
//
// The coarse operator A_c couples an aggregate to its 26 neighbours only, so that with the
// aggregates grouped in planes along the grid's longest axis it is block tridiagonal: L planes
// of m = n / L aggregates, diagonal blocks D_i and couplings E_i = A_{i,i+1}.  A level of the
// reduction eliminates every other plane i (neighbours l and r among the planes left):
//   W_l = D_i^-1 A_{i,l},  W_r = D_i^-1 A_{i,r}
//   D_l -= A_{l,i} W_l,    D_r -= A_{r,i} W_r,    A_{l,r} = -A_{l,i} W_r
// until one plane is left; the inverse G then grows back level by level from the kept planes:
//   G_{i,j} = -(W_l G_{l,j} + W_r G_{r,j}) [+ D_i^-1 for j = i].
// With L = 14 planes of m = 196 (n = 2744) that is 14 inversions of 196 x 196 blocks on a
// chain of five, 1 GFLOP of eliminations and 4 GFLOP of growth, against the 1.5 TFLOP of the
// 36 n x n products that 18 Newton-Schulz steps take.  The inversions' chain bounds it: m
// dependent pivots each, one CTA a block, the block in registers.
#include <algorithm>

#include "coarse_index.h"
#include "coarse_inverse.cuh"

namespace nnpp {

namespace {

// A pivot below this fraction of its diagonal entry of A_c means an operator that is singular or
// nearly so (a liquid pocket without a Dirichlet value): the caller then takes the
// Newton-Schulz iteration, whose iterates stay positive.  The workloads' smallest is 0.82.
constexpr float kPivotMin = 1e-3f;

// plane of natural aggregate index I and its place in the plane, for planes along `axis`
struct PlaneMap {
  int na0, na1, na2, axis, m;
};
__device__ __forceinline__ int plane_index(const PlaneMap& g, int I) {
  const int ax = I % g.na0, ay = (I / g.na0) % g.na1, az = I / (g.na0 * g.na1);
  if (g.axis == 2) return I;
  if (g.axis == 1) return ay * g.m + ax + g.na0 * az;
  return ax * g.m + ay + g.na1 * az;
}

// the stencil rows into the planes' diagonal and coupling blocks (zeroed before), and A_c's
// diagonal in plane order
__global__ void k_blocks_fill(PlaneMap g, const float* st27, float* d, float* e, float* diag) {
  const int n = g.na0 * g.na1 * g.na2;
  const size_t mm = (size_t)g.m * g.m;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 27 * n; t += gridDim.x * blockDim.x) {
    const int I = t / 27, q = t - 27 * I;
    const int ax = I % g.na0, ay = (I / g.na0) % g.na1, az = I / (g.na0 * g.na1);
    const int jx = ax + q % 3 - 1, jy = ay + (q / 3) % 3 - 1, jz = az + q / 9 - 1;
    if (jx < 0 || jy < 0 || jz < 0 || jx >= g.na0 || jy >= g.na1 || jz >= g.na2) continue;
    const float v = st27[t];
    const int p = plane_index(g, I);
    if (q == 13) diag[p] = v;
    if (v == 0.0f) continue;
    const int r = plane_index(g, jx + g.na0 * (jy + g.na1 * jz));
    const int pi = p / g.m, ri = r / g.m;
    const size_t o = pi * mm + (size_t)(p - pi * g.m) * g.m + (r - ri * g.m);
    if (ri == pi)
      d[o] = v;
    else if (ri == pi + 1)
      e[o] = v;  // row plane i, column plane i + 1; the transpose is implied
  }
}

// In-place inverse of one symmetric positive definite m x m block per CTA by sweeps (Gauss-Jordan
// without pivoting in the form that keeps the matrix symmetric: pivot row v, d = v_k:
// a_ij -= v_i v_j / d, a_ik = a_ki = v_i / d, a_kk = -1 / d; the result is -A^-1).  Thread (r, c) of
// 16 x 32 holds the entries (r + 16 a, c + 32 b) in 91 registers; a step shares the pivot's row
// and reciprocal through shared memory, double buffered: one barrier a step, then 91 FMAs against
// 11 shared loads (the row values of a thread's rows lie together).  196 dependent steps: 134
// us, 147 with row and column shared and 201 with 1024 threads of 49 entries, which spill.
constexpr int kGjR = kPlaneMax / 16, kGjC = (kPlaneMax + 31) / 32;
constexpr int kGjPad = 20;  // floats between the threads' row values (16-byte aligned, few conflicts)
__global__ void __launch_bounds__(512, 1) k_gj(int m, float* d, const float* diag, int first, int stride, int* bad) {
  __shared__ float s_row[2][32 * kGjC], s_inv[2];
  __shared__ __align__(16) float s_own[2][16 * kGjPad];  // the same values: entry r + 16 a at kGjPad r + a
  static_assert(kGjR <= 16 && kGjR > 12, "a thread's row values are four 16-byte loads");
  float* blk = d + (size_t)(first + stride * (int)blockIdx.x) * m * m;
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5;
  float x[kGjR][kGjC];
#pragma unroll
  for (int a = 0; a < kGjR; ++a)
#pragma unroll
    for (int b = 0; b < kGjC; ++b) {
      const int i = r + 16 * a, j = c + 32 * b;
      x[a][b] = i < m && j < m ? blk[(size_t)i * m + j] : 0.0f;
    }
  const float* dg = diag + (size_t)(first + stride * (int)blockIdx.x) * m;
  for (int t = threadIdx.x; t < 2 * 16 * kGjPad; t += 512) s_own[0][t] = 0.0f;
  bool ok = true;
  __syncthreads();
#pragma unroll
  for (int ka = 0; ka < kGjR; ++ka) {
    const int kb = ka / 2;  // the pivots' column group
#pragma unroll 1
    for (int kr = 0; kr < 16; ++kr) {
      const int k = 16 * ka + kr;
      if (k >= m) break;
      const int kc = kr + 16 * (ka & 1);
      float* row = s_row[k & 1];
      float* own = s_own[k & 1];
      if (r == kr) {
#pragma unroll
        for (int b = 0; b < kGjC; ++b) {
          row[c + 32 * b] = x[ka][b];
          if (2 * b < kGjR && (c < 16 || 2 * b + 1 < kGjR)) own[kGjPad * (c & 15) + 2 * b + (c >> 4)] = x[ka][b];
        }
        if (c == kc) {
          ok = ok && x[ka][kb] >= kPivotMin * dg[k];  // false for NaN
          s_inv[k & 1] = 1.0f / x[ka][kb];
        }
      }
      __syncthreads();
      const float p = s_inv[k & 1];
      float rj[kGjC];
#pragma unroll
      for (int b = 0; b < kGjC; ++b) rj[b] = row[c + 32 * b] * p;
      if (c == kc) {
        rj[kb] = -p;
#pragma unroll
        for (int a = 0; a < kGjR; ++a) x[a][kb] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 vi = *reinterpret_cast<const float4*>(own + kGjPad * r + 4 * q);
        const float v4[4] = {-vi.x, -vi.y, -vi.z, -vi.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (4 * q + u < kGjR)
#pragma unroll
            for (int b = 0; b < kGjC; ++b) x[4 * q + u][b] = fmaf(v4[u], rj[b], x[4 * q + u][b]);
      }
      if (r == kr)
#pragma unroll
        for (int b = 0; b < kGjC; ++b) x[ka][b] = rj[b];
    }
  }
#pragma unroll
  for (int a = 0; a < kGjR; ++a)
#pragma unroll
    for (int b = 0; b < kGjC; ++b) {
      const int i = r + 16 * a, j = c + 32 * b;
      if (i < m && j < m) blk[(size_t)i * m + j] = -x[a][b];
    }
  if (!ok) *bad = 1;
}

// One 64 x 64 tile of C += op(A) op(B), 256 threads, 4 x 4 entries a thread: rows row0.. of
// op(A) (M x K), columns col0.. of op(B) (K x N).  TA / TB: the operand is stored transposed.
constexpr int kTile = 64;
constexpr int kTK = 16;
struct TileSm {
  float a[kTK][kTile + 4];
  float b[kTK][kTile + 4];
};
template <bool TA, bool TB>
__device__ __forceinline__ void tile_mma(TileSm& s, const float* A, int lda, const float* B, int ldb, int M, int N,
                                         int K, int row0, int col0, float (&acc)[4][4]) {
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  for (int k0 = 0; k0 < K; k0 += kTK) {
#pragma unroll
    for (int u = 0; u < kTile * kTK / 256; ++u) {
      const int e = t + 256 * u;
      {
        const int i = TA ? e % kTile : e / kTK, k = TA ? e / kTile : e % kTK;
        const bool ok = row0 + i < M && k0 + k < K;
        s.a[k][i] = ok ? (TA ? A[(size_t)(k0 + k) * lda + row0 + i] : A[(size_t)(row0 + i) * lda + k0 + k]) : 0.0f;
      }
      {
        const int j = TB ? e / kTK : e % kTile, k = TB ? e % kTK : e / kTile;
        const bool ok = col0 + j < N && k0 + k < K;
        s.b[k][j] = ok ? (TB ? B[(size_t)(col0 + j) * ldb + k0 + k] : B[(size_t)(k0 + k) * ldb + col0 + j]) : 0.0f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kTK; ++k) {
      const float4 av = *reinterpret_cast<const float4*>(&s.a[k][4 * ty]);
      const float4 bv = *reinterpret_cast<const float4*>(&s.b[k][4 * tx]);
      const float a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
}

// multipliers of the planes i = s, 3 s, ... of a level of stride s: W_l = D_i^-1 E_l^T (the
// coupling l -> i transposed), W_r = D_i^-1 E_i.  blockIdx.z = 2 (index among the planes) + side
__global__ void __launch_bounds__(256) k_multipliers(int m, int planes, int s, const float* d, const float* e, float* wl,
                                                     float* wr) {
  __shared__ TileSm sm;
  const int i = s * (2 * (int)(blockIdx.z >> 1) + 1);
  const bool right = blockIdx.z & 1;
  if (right && i + s >= planes) return;
  const size_t mm = (size_t)m * m;
  const int row0 = blockIdx.y * kTile, col0 = blockIdx.x * kTile;
  float acc[4][4] = {};
  if (right)
    tile_mma<false, false>(sm, d + i * mm, m, e + i * mm, m, m, m, m, row0, col0, acc);
  else
    tile_mma<false, true>(sm, d + i * mm, m, e + (i - s) * mm, m, m, m, m, row0, col0, acc);
  float* w = (right ? wr : wl) + i * mm;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = row0 + 4 * ty + u, c = col0 + 4 * tx + v;
      if (r < m && c < m) w[(size_t)r * m + c] = acc[u][v];
    }
}

// the kept planes j = 0, 2 s, ... of a level: D_j -= E_j W_l(j + s) + E_{j-s}^T W_r(j - s)
// (blockIdx.z even), and their next coupling e2_j = -E_j W_r(j + s) (odd)
__global__ void __launch_bounds__(256) k_eliminate(int m, int planes, int s, float* d, const float* e, const float* wl,
                                                   const float* wr, float* e2) {
  __shared__ TileSm sm;
  const int j = 2 * s * (int)(blockIdx.z >> 1);
  const bool next = blockIdx.z & 1;
  const size_t mm = (size_t)m * m;
  const int row0 = blockIdx.y * kTile, col0 = blockIdx.x * kTile;
  if (next && j + 2 * s >= planes) return;
  float acc[4][4] = {};
  if (next) {
    tile_mma<false, false>(sm, e + j * mm, m, wr + (j + s) * mm, m, m, m, m, row0, col0, acc);
  } else {
    if (j + s < planes) tile_mma<false, false>(sm, e + j * mm, m, wl + (j + s) * mm, m, m, m, m, row0, col0, acc);
    if (j >= s) tile_mma<true, false>(sm, e + (j - s) * mm, m, wr + (j - s) * mm, m, m, m, m, row0, col0, acc);
  }
  float* o = (next ? e2 : d) + j * mm;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = row0 + 4 * ty + u, c = col0 + 4 * tx + v;
      if (r < m && c < m) o[(size_t)r * m + c] = next ? -acc[u][v] : o[(size_t)r * m + c] - acc[u][v];
    }
}

// the inverse's growth by a level of stride s, plane pairs (i, j), i = s (2 t + 1):
//   ODD == 0: j = 2 s u (kept planes): G_{i,j} and its transpose G_{j,i};
//   ODD == 1: j = s (2 u + 1) >= i, from the transposes written by ODD == 0 (+ D_i^-1 for
//             j = i), and its transpose.
template <int ODD>
__global__ void __launch_bounds__(256) k_grow(int m, int planes, GrowPass pass, const float* d, const float* wl,
                                              const float* wr, float* x) {
  __shared__ TileSm sm;
  const GrowPass::Block blk = pass.block((int)blockIdx.x);
  const int s = pass.s, i = blk.i, j = blk.j;
  if (ODD && j < i) return;
  const size_t mm = (size_t)m * m;
  const size_t n = (size_t)planes * m;
  const int row0 = blk.row_tile * kTile, col0 = blk.col_tile * kTile;
  float acc[4][4] = {};
  tile_mma<false, false>(sm, wl + i * mm, m, x + (size_t)(i - s) * m * n + (size_t)j * m, (int)n, m, m, m, row0, col0, acc);
  if (i + s < planes)
    tile_mma<false, false>(sm, wr + i * mm, m, x + (size_t)(i + s) * m * n + (size_t)j * m, (int)n, m, m, m, row0, col0, acc);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int r = row0 + 4 * ty + a, c = col0 + 4 * tx + b;
      if (r >= m || c >= m) continue;
      float v = -acc[a][b];
      if (ODD && i == j) v += d[i * mm + (size_t)r * m + c];
      x[((size_t)i * m + r) * n + (size_t)j * m + c] = v;
      if (i != j) x[((size_t)j * m + c) * n + (size_t)i * m + r] = v;
    }
}

// the last plane's inverse into its block of x (n x n, rows in plane order)
__global__ void k_first_block(int m, int n, const float* d, float* x) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < m * m; t += gridDim.x * blockDim.x)
    x[(size_t)(t / m) * n + t % m] = d[t];
}

// inv (natural order, rows of stride ld) = (x + x^T) / 2 from plane order; the diagonal entry
// of an aggregate without unknowns (rowabs < 0) is zero, as k_symmetrize leaves it.  Nothing is
// written when a pivot failed: inv may hold the Newton-Schulz warm start.
__global__ void k_inverse_out(PlaneMap g, int n, int ld, const float* x, const float* rowabs, const int* bad, float* inv) {
  if (*bad) return;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const size_t pi = plane_index(g, i);
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      const size_t pj = plane_index(g, j);
      inv[(size_t)i * ld + j] = (i == j && rowabs[i] < 0.0f) ? 0.0f : 0.5f * (x[pi * n + pj] + x[pj * n + pi]);
    }
  }
}

}  // namespace

bool coarse_planes(const int na[3], CoarseBlocks& b) {
  b.axis = 2;
  for (int a = 1; a >= 0; --a)
    if (na[a] > na[b.axis]) b.axis = a;
  b.planes = na[b.axis];
  b.m = na[0] * na[1] * na[2] / std::max(1, b.planes);
  return b.m >= 1 && b.m <= kPlaneMax;
}

bool coarse_blocks_alloc(CoarseBlocks& b) {
  const size_t all = (size_t)b.planes * b.m * b.m;
  return b.d.alloc(all) && b.e[0].alloc(all) && b.e[1].alloc(all) && b.wl.alloc(all) && b.wr.alloc(all) &&
         b.diag.alloc((size_t)b.planes * b.m) && b.bad.alloc(1);
}

nnpp_status coarse_direct_inverse(CoarseBlocks& b, const int na[3], const float* st27, const float* rowabs, float* x,
                                  float* inv, int ld, cudaStream_t st) {
  const int m = b.m, L = b.planes, n = m * L;
  const PlaneMap g = {na[0], na[1], na[2], b.axis, m};
  NNPP_CUDA(cudaMemsetAsync(b.d.get(), 0, b.d.bytes(), st));
  NNPP_CUDA(cudaMemsetAsync(b.e[0].get(), 0, b.e[0].bytes(), st));
  NNPP_CUDA(cudaMemsetAsync(b.bad.get(), 0, sizeof(int), st));
  k_blocks_fill<<<std::max(1, std::min((27 * n + 255) / 256, 1216)), 256, 0, st>>>(g, st27, b.d.get(), b.e[0].get(),
                                                                                   b.diag.get());
  const unsigned nt = (unsigned)((m + kTile - 1) / kTile);
  int level = 0;
  int s = 1;
  for (; s < L; s *= 2, ++level) {
    const int odd = (L - 1 - s) / (2 * s) + 1, kept = (L - 1) / (2 * s) + 1;
    const float* e = b.e[level & 1].get();
    k_gj<<<odd, 512, 0, st>>>(m, b.d.get(), b.diag.get(), s, 2 * s, b.bad.get());
    k_multipliers<<<dim3(nt, nt, 2 * odd), 256, 0, st>>>(m, L, s, b.d.get(), e, b.wl.get(), b.wr.get());
    k_eliminate<<<dim3(nt, nt, 2 * kept), 256, 0, st>>>(m, L, s, b.d.get(), e, b.wl.get(), b.wr.get(),
                                                       b.e[(level + 1) & 1].get());
  }
  k_gj<<<1, 512, 0, st>>>(m, b.d.get(), b.diag.get(), 0, 1, b.bad.get());
  k_first_block<<<std::max(1, std::min((m * m + 255) / 256, 152)), 256, 0, st>>>(m, n, b.d.get(), x);
  for (s /= 2; s >= 1; s /= 2) {
    const int odd = (L - 1 - s) / (2 * s) + 1, kept = (L - 1) / (2 * s) + 1;
    const GrowPass even = {s, odd, kept, 0, (int)nt}, odds = {s, odd, odd, 1, (int)nt};
    k_grow<0><<<(unsigned)even.blocks(), 256, 0, st>>>(m, L, even, b.d.get(), b.wl.get(), b.wr.get(), x);
    k_grow<1><<<(unsigned)odds.blocks(), 256, 0, st>>>(m, L, odds, b.d.get(), b.wl.get(), b.wr.get(), x);
  }
  k_inverse_out<<<std::min(n, 152 * 8), 256, 0, st>>>(g, n, ld, x, rowabs, b.bad.get(), inv);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

}  // namespace nnpp
