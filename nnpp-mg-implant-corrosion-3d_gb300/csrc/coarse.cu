// coarse.cu -- the coarse space of the two-level preconditioner of the potential solve.
//
// Aggregates are blocks of f x f x f bins (bins of side >= the horizon radius, so every bond
// joins the same or an adjacent aggregate).  The preconditioner is
//   M^-1 r = D^-1 r + P A_c^-1 P^T r,   P = the aggregate indicator of the unknowns,
// A_c = P^T A P the Galerkin coarse operator (27 nonzeros per row), and its inverse a dense
// n x n FP32 matrix (n <= kCoarseMax).  The inverse is formed directly, by block cyclic
// reduction over the planes of aggregates (coarse_inverse.cu).  Where a pivot of that is too
// small to trust (a singular or nearly singular operator: a liquid pocket without a Dirichlet
// value), it comes instead from the Newton-Schulz iteration X <- X (2I - A_c X),
// X_0 = I / ||A_c||_inf: every iterate is a positive polynomial of A_c, so the preconditioner
// stays symmetric positive definite even on a singular operator.  Its GEMMs are FP32 products
// that cuBLAS runs on the BF16 tensor cores by the BF16x9 split (each FP32 operand as three
// BF16 parts, nine partial products accumulated in FP32: FP32 accuracy, not TF32's).  A
// periodic rebuild of such an operator within a run starts from the previous inverse when
// ||I - A_c X_0||_F < 1/2: the error then squares every step, and a few steps replace the 18 of
// the cold start.  The coarse operator is rebuilt when the state is replaced, and every
// `coarse_every` steps (counted from the last replacement) if a phase changed since the last
// rebuild; in between a stale one is still a valid preconditioner.  The schedule depends only
// on the step count and the phases, so it is reproducible, and forward_ckpt records each
// rebuilt inverse for backward to replay.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include <cublas_v2.h>

#include "engine.cuh"

namespace nnpp {

namespace {

constexpr int kNsIterations = 18;
constexpr int kNormBlocks = 128;      // block partials of the warm start's residual norm
constexpr double kNsWarmMax = 0.5;    // warm start when ||I - A_c X_0||_F is below this
constexpr double kNsTarget = 1e-8;    // warm start: steps until the bound ||.||^(2^m) meets this

// C = A B for n x n column-major FP32 matrices, emulated FP32 on the BF16 tensor cores (the
// handle's emulation strategy is EAGER, so cuBLAS takes the emulated kernels wherever they
// exist and its FP32 kernels elsewhere)
cublasStatus_t ns_gemm(cublasHandle_t hb, int n, const float* a, const float* b, float* c) {
  const float one = 1.0f, zero = 0.0f;
  return cublasGemmEx(hb, CUBLAS_OP_N, CUBLAS_OP_N, n, n, n, &one, a, CUDA_R_32F, n, b, CUDA_R_32F, n, &zero, c,
                      CUDA_R_32F, n, CUBLAS_COMPUTE_32F_EMULATED_16BFX9, CUBLAS_GEMM_DEFAULT);
}

// block partials of ||I - T||_F^2 (T n x n): FP32 sums per thread, FP64 across the block
__global__ void k_resid_sq(int n, const float* T, double* partials) {
  __shared__ double sm[256 / 32];
  const size_t nn = (size_t)n * n;
  float s = 0.0f;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < nn; e += (size_t)gridDim.x * blockDim.x) {
    const float d = ((e / n == e % n) ? 1.0f : 0.0f) - T[e];
    s = fmaf(d, d, s);
  }
  double x = s;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 256 / 32; ++w) t += sm[w];
    partials[blockIdx.x] = t;
  }
}

// aggregate of every node (internal order), from the bins' node ranges
__global__ void k_agg_fill(const int* bin_start, int nb0, int nb1, int nb2, int f, int na0, int na1,
                           int* agg) {
  const int nbins = nb0 * nb1 * nb2;
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nbins; b += gridDim.x * blockDim.x) {
    const int bx = b % nb0, by = (b / nb0) % nb1, bz = b / (nb0 * nb1);
    const int I = bx / f + na0 * (by / f + na1 * (bz / f));
    for (int i = bin_start[b]; i < bin_start[b + 1]; ++i) agg[i] = I;
  }
}

__device__ __forceinline__ bool node_liquid(const KParams& k, int i, int mixed) {
  return (mixed ? k.rec32_cur[i].phase : (float)k.rec64_cur[i].phase) == 0.0f;
}

// What the bond walk needs of a node in one word: its aggregate's place (10 bits an axis: build_tiles, which
// runs before any coarse operator, refuses more than kMaxAxisBins bins an axis), liquid and
// potential-Dirichlet flags.
static_assert(kMaxAxisBins <= 1024, "a place's fields are 10 bits an axis");
constexpr unsigned int kTagLiquid = 1u << 30, kTagDir = 1u << 31;
__global__ void k_node_tags(KParams k, int mixed, int na0, int na1, unsigned int* tag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k.N; i += gridDim.x * blockDim.x) {
    const int I = k.agg[i];
    tag[i] = (unsigned int)(I % na0) | (unsigned int)((I / na0) % na1) << 10 | (unsigned int)(I / (na0 * na1)) << 20 |
             (node_liquid(k, i, mixed) ? kTagLiquid : 0u) | (((k.dirmask[i] >> S) & 1) ? kTagDir : 0u);
  }
}

// Rows of A P off the diagonal term, for the deflated CG: for an unknown i (a liquid node off the
// potential's Dirichlet set) and an aggregate J, -sum of w_ij over the unknowns j of J.  Thread
// per node, the neighbour aggregates' sums in the row's bond order (four bonds' loads in flight),
// written in neighbour order into the K-slot layout
// col/val[s * N + i], the unused slots with value 0 (sliced like ELLPACK: the threads of a warp
// read consecutive words); kmax takes the largest number of used slots.  Also, for A_c: the sum of
// the node's liquid bonds (dn) and the neighbours in use (mask, bit 31: the node is an unknown).
constexpr int kApBlock = 128;
// FEW: aggregates two or more bins wide, so that a node's neighbours lie on one side an axis at most:
// eight sums in registers, by the axes on which the neighbour's aggregate differs (27 columns of
// shared memory leave the L1 too small for the rows' lines: 0.91 ms at 512k nodes against 0.185)
template <bool FEW>
__global__ void __launch_bounds__(kApBlock) k_ap_rows(KParams k, const unsigned int* tag, int na0, int na1, int K,
                                                      int* kmax, int* col, float* val, float* dn, unsigned int* mask) {
  __shared__ float s_acc[FEW ? 1 : 27 * kApBlock];
  float* sa = s_acc + threadIdx.x;
  const size_t N = k.N;
  int most = 0;
  for (int i = blockIdx.x * kApBlock + threadIdx.x; i < k.N; i += gridDim.x * kApBlock) {
    const unsigned int me = tag[i];
    unsigned int touched = 0u;
    float d = 0.0f;
    bool ll = false;
    float acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
    if (!FEW)
#pragma unroll
      for (int q = 0; q < 27; ++q) sa[q * kApBlock] = 0.0f;
    if ((me & kTagLiquid) && !(me & kTagDir)) {
      const int ax = me & 1023u, ay = (me >> 10) & 1023u, az = (me >> 20) & 1023u;
      const int j1 = k.row[i + 1];
      for (int j = k.row[i]; j < j1; j += 4) {
        unsigned int t[4];
        float w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          t[u] = j + u < j1 ? tag[k.col[j + u]] : 0u;
          w[u] = j + u < j1 ? k.w32[j + u] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (!(t[u] & kTagLiquid)) continue;
          d += w[u];
          ll = true;
          if (t[u] & kTagDir) continue;
          const int dx = (int)(t[u] & 1023u) - ax, dy = (int)((t[u] >> 10) & 1023u) - ay, dz = (int)((t[u] >> 20) & 1023u) - az;
          const int q = (dx + 1) + 3 * ((dy + 1) + 3 * (dz + 1));
          touched |= 1u << q;
          if (FEW) {
            const int slot = (dx != 0) + 2 * (dy != 0) + 4 * (dz != 0);
#pragma unroll
            for (int b = 0; b < 8; ++b) acc[b] -= b == slot ? w[u] : 0.0f;
          } else {
            sa[q * kApBlock] -= w[u];
          }
        }
      }
      int o = 0;
      for (unsigned int left = touched; left; left &= left - 1) {
        const int q = __ffs(left) - 1;
        const int dx = q % 3 - 1, dy = (q / 3) % 3 - 1, dz = q / 9 - 1;
        float v = 0.0f;
        if (FEW) {
          const int slot = (dx != 0) + 2 * (dy != 0) + 4 * (dz != 0);
#pragma unroll
          for (int b = 0; b < 8; ++b) v = b == slot ? acc[b] : v;
        } else {
          v = sa[q * kApBlock];
        }
        col[o * N + i] = (ax + dx) + na0 * ((ay + dy) + na1 * (az + dz));
        val[o * N + i] = v;
        ++o;
      }
    }
    const int used = __popc(touched);
    for (int o = used; o < K; ++o) {
      col[o * N + i] = k.agg[i];
      val[o * N + i] = 0.0f;
    }
    dn[i] = d;
    mask[i] = touched | (ll ? 0x80000000u : 0u);
    most = max(most, used);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most) atomicMax(kmax, most);
}

// Warp per aggregate row I: the 27 entries of A_c = P^T A P summed from its nodes' rows of A P and
// their diagonals.  Lanes own fixed node subsets and reduce in a fixed order, so the matrix is
// reproducible.  (Walking the bonds once more from the aggregates took 1.45 ms at 512k nodes, a
// warp per aggregate with 27 selects a bond; this pass takes 0.035 ms.)
constexpr int kSumWarps = 4;
__global__ void __launch_bounds__(32 * kSumWarps) k_coarse_assemble(KParams k, const int* bin_start, int nb0, int nb1, int nb2,
                                                                    int f, int na0, int na1, int na2, const float* val,
                                                                    const float* dn, const unsigned int* mask,
                                                                    float* st27, float* rowabs) {
  __shared__ float s_acc[kSumWarps][27 * 32];
  const int lane = threadIdx.x & 31;
  float* acc = s_acc[threadIdx.x >> 5] + lane;
  const int n = na0 * na1 * na2;
  const size_t N = k.N;
  for (int I = blockIdx.x * kSumWarps + (threadIdx.x >> 5); I < n; I += gridDim.x * kSumWarps) {
    const int ax = I % na0, ay = (I / na0) % na1, az = I / (na0 * na1);
#pragma unroll
    for (int q = 0; q < 27; ++q) acc[32 * q] = 0.0f;
    int unknowns = 0;
    const int bx0 = ax * f, bx1 = min(ax * f + f, nb0);
    for (int bz = az * f; bz < min(az * f + f, nb2); ++bz)
      for (int by = ay * f; by < min(ay * f + f, nb1); ++by) {
        // the bins along x are one contiguous node range
        const int b = bx0 + nb0 * (by + nb1 * bz);
        const int i1 = bin_start[b + (bx1 - bx0)];
        for (int i = bin_start[b] + lane; i < i1; i += 32) {
          const unsigned int m = mask[i];
          if (!(m >> 31)) continue;
          ++unknowns;
          acc[32 * 13] += dn[i];
          size_t o = i;
          for (unsigned int left = m & 0x7ffffffu; left; left &= left - 1, o += N) acc[32 * (__ffs(left) - 1)] += val[o];
        }
      }
    unknowns = __reduce_add_sync(0xffffffffu, unknowns);
    // lane q keeps entry q
    float mine = 0.0f, ra = 0.0f;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
      float x = acc[32 * q];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      ra += fabsf(x);
      if (lane == q) mine = x;
    }
    // no unknown in the aggregate: an identity row keeps A_c regular (rowabs -1 marks it: the
    // inverse's diagonal entry there is zeroed)
    if (lane < 27) {
      const int jx = ax + lane % 3 - 1, jy = ay + (lane / 3) % 3 - 1, jz = az + lane / 9 - 1;
      const bool in = jx >= 0 && jy >= 0 && jz >= 0 && jx < na0 && jy < na1 && jz < na2;
      st27[27 * (size_t)I + lane] = unknowns == 0 ? (lane == 13 ? 1.0f : 0.0f) : (in ? mine : 0.0f);
    }
    if (lane == 0) rowabs[I] = unknowns == 0 ? -1.0f : ra;
  }
}

// the dense operator from its stencil rows (mat zeroed before; the Newton-Schulz iteration's)
__global__ void k_dense_operator(const float* st27, int na0, int na1, int na2, float* mat) {
  const int n = na0 * na1 * na2;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 27 * n; t += gridDim.x * blockDim.x) {
    const int I = t / 27, q = t - 27 * I;
    const int jx = I % na0 + q % 3 - 1, jy = (I / na0) % na1 + (q / 3) % 3 - 1, jz = I / (na0 * na1) + q / 9 - 1;
    if (jx < 0 || jy < 0 || jz < 0 || jx >= na0 || jy >= na1 || jz >= na2) continue;
    mat[(size_t)I * n + (jx + na0 * (jy + na1 * jz))] = st27[t];
  }
}

// X = I / max_i rowabs[i]  (column-major n x n)
__global__ void k_ns_init(int n, const float* rowabs, float* X) {
  __shared__ float smax;
  if (threadIdx.x == 0) {
    float m = 0.0f;
    for (int i = 0; i < n; ++i) m = fmaxf(m, fabsf(rowabs[i]));  // identity rows count 1
    smax = m > 0.0f ? m : 1.0f;
  }
  __syncthreads();
  const float inv = 1.0f / smax;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * n; e += (size_t)gridDim.x * blockDim.x)
    X[e] = (e / n == e % n) ? inv : 0.0f;
}

// T = 2I - T
__global__ void k_two_i_minus(int n, float* T) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * n; e += (size_t)gridDim.x * blockDim.x)
    T[e] = ((e / n == e % n) ? 2.0f : 0.0f) - T[e];
}

// Y = (X + X^T) / 2, Y with rows of stride ld; the diagonal entry of an aggregate that held
// no unknown (rowabs < 0) is zero.  Its row and column of X are those of the identity; once
// a front reaches the aggregate, a coarse inverse that has not been rebuilt yet would scale
// the aggregate's residual sum by 1 instead of by the inverse of its new diagonal, so the
// stale additive correction leaves such aggregates to the diagonal part.
__global__ void k_symmetrize(int n, int ld, const float* X, const float* rowabs, float* Y) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * n; e += (size_t)gridDim.x * blockDim.x) {
    const size_t i = e / n, j = e % n;
    Y[i * ld + j] = (i == j && rowabs[i] < 0.0f) ? 0.0f : 0.5f * (X[e] + X[j * n + i]);
  }
}

// phases in internal order (1: solid) from the current records
__global__ void k_phase_snap(KParams k, int mixed, unsigned char* snap) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k.N; i += gridDim.x * blockDim.x)
    snap[i] = node_liquid(k, i, mixed) ? 0 : 1;
}

// number of nodes whose phase differs from snap
__global__ void k_phase_diff(KParams k, int mixed, const unsigned char* snap, int* count) {
  int c = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k.N; i += gridDim.x * blockDim.x)
    c += (node_liquid(k, i, mixed) ? 0 : 1) != snap[i];
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

// deflation flag from a phase comparison: on when no node differs from the operator's phases
__global__ void k_defl_from_count(DevState* ds, const int* count) { ds->defl = *count == 0 ? 1 : 0; }

}  // namespace

Coarse::~Coarse() {
  if (cublas) cublasDestroy(static_cast<cublasHandle_t>(cublas));
}

nnpp_status coarse_build(Handle& h) {
  Coarse& c = h.coarse;
  c.valid = false;
  c.n = 0;
  if (!h.coarse_enabled) return NNPP_OK;
  const Layout& L = h.lay;
  int f = 1;
  auto count = [&](int ff) {
    long long n = 1;
    for (int d = 0; d < 3; ++d) n *= (L.nb[d] + ff - 1) / ff;
    return n;
  };
  while (count(f) > kCoarseMax) ++f;
  c.f = f;
  for (int d = 0; d < 3; ++d) c.na[d] = (L.nb[d] + f - 1) / f;
  c.n = (int)count(f);
  c.ld = (c.n + 3) & ~3;
  // A P rows hold at most 27 aggregates each: allocated once, so that no pointer the
  // kernels hold changes when the operator is rebuilt or replayed
  if (!c.agg.alloc(h.N) || !c.inv.alloc(c.inv_elems()) || !c.rc.alloc(c.ld) || !c.xc.alloc(c.n) ||
      !c.dots.alloc(3 * (size_t)c.n) || !c.rowabs.alloc(c.n) || !c.ap_col.alloc(27 * (size_t)h.N) ||
      !c.ap_val.alloc(27 * (size_t)h.N))
    return set_error(NNPP_ERR_NOMEM, "coarse space");
  NNPP_CUDA(cudaMemsetAsync(c.dots.get(), 0, sizeof(double) * 3 * (size_t)c.n, h.st));
  NNPP_CUDA(cudaMemsetAsync(c.rc.get(), 0, sizeof(float) * c.ld, h.st));  // padding to ld stays 0
  c.ap_k = 1;
  NNPP_CUDA(cudaMemsetAsync(c.inv.get(), 0, sizeof(float) * c.inv_elems(), h.st));  // padding stays 0
  k_agg_fill<<<std::max(1, std::min((L.nbins + 255) / 256, 4096)), 256, 0, h.st>>>(
      L.bin_start.get(), L.nb[0], L.nb[1], L.nb[2], f, c.na[0], c.na[1], c.agg.get());
  NNPP_CUDA(cudaGetLastError());
  c.stale = true;
  return NNPP_OK;
}

// The Newton-Schulz inverse of the operator in c.st27 into c.inv (see the file comment).
static nnpp_status newton_schulz_inverse(Handle& h, bool* warm_out, int* steps_out) {
  Coarse& c = h.coarse;
  const int n = c.n;
  const size_t nn = (size_t)n * n;
  if (!c.cublas) {
    cublasHandle_t hb = nullptr;
    if (cublasCreate(&hb) != CUBLAS_STATUS_SUCCESS) return set_error(NNPP_ERR_CUDA, "cublasCreate");
    c.cublas = hb;
    if (cublasSetEmulationStrategy(hb, CUBLAS_EMULATION_STRATEGY_EAGER) != CUBLAS_STATUS_SUCCESS)
      return set_error(NNPP_ERR_CUDA, "cublasSetEmulationStrategy");
  }
  if (!c.a.alloc(nn) || !c.t.alloc(nn) || !c.x.alloc(nn) || !c.y.alloc(nn))
    return set_error(NNPP_ERR_NOMEM, "coarse inverse");
  DBuf<float>& A = c.a;
  DBuf<float>& T = c.t;
  DBuf<float>& X = c.x;
  NNPP_CUDA(cudaMemsetAsync(A.get(), 0, sizeof(float) * nn, h.st));
  k_dense_operator<<<std::max(1, std::min((27 * n + 255) / 256, 1216)), 256, 0, h.st>>>(c.st27.get(), c.na[0], c.na[1],
                                                                                       c.na[2], A.get());
  NNPP_CUDA(cudaGetLastError());
  const int eg = (int)std::min<size_t>((nn + 255) / 256, 152 * 64);
  cublasHandle_t hb = static_cast<cublasHandle_t>(c.cublas);
  if (cublasSetStream(hb, h.st) != CUBLAS_STATUS_SUCCESS) return set_error(NNPP_ERR_CUDA, "cublasSetStream");
  float* x = X.get();
  float* y = c.y.get();
  // a rebuild within a run (phases changed since the last one, the state not replaced)
  // starts from the last inverse if it is close enough: T = A X_0 is then the first step's
  // product already.  The residual norm is summed on the host in block order, so the
  // number of steps is reproducible.
  int steps = kNsIterations;
  bool warm = false;
  if (c.ns_valid && !c.stale && h.coarse_event_cur < 0) {
    if (!c.nrm.alloc(kNormBlocks)) return set_error(NNPP_ERR_NOMEM, "coarse inverse");
    NNPP_CUDA(cudaMemcpy2DAsync(x, sizeof(float) * n, c.inv.get(), sizeof(float) * c.ld, sizeof(float) * n, n,
                                cudaMemcpyDeviceToDevice, h.st));
    if (ns_gemm(hb, n, A.get(), x, T.get()) != CUBLAS_STATUS_SUCCESS)
      return set_error(NNPP_ERR_CUDA, "coarse inverse: GEMM");
    k_resid_sq<<<kNormBlocks, 256, 0, h.st>>>(n, T.get(), c.nrm.get());
    NNPP_CUDA(cudaGetLastError());
    std::vector<double> part(kNormBlocks);
    NNPP_CUDA(cudaMemcpyAsync(part.data(), c.nrm.get(), sizeof(double) * kNormBlocks, cudaMemcpyDeviceToHost, h.st));
    NNPP_CUDA(cudaStreamSynchronize(h.st));
    double ss = 0.0;
    for (double v : part) ss += v;
    const double r0 = std::sqrt(ss);
    if (std::isfinite(r0) && r0 < kNsWarmMax) {
      warm = true;
      steps = 1;
      while (steps < kNsIterations && std::pow(r0, std::ldexp(1.0, steps)) > kNsTarget) ++steps;
    }
  }
  if (!warm) {
    k_ns_init<<<eg, 256, 0, h.st>>>(n, c.rowabs.get(), X.get());
    NNPP_CUDA(cudaGetLastError());
  }
  for (int it = 0; it < steps; ++it) {
    // T = A X ; T = 2I - T ; X <- X T
    if (!(warm && it == 0) && ns_gemm(hb, n, A.get(), x, T.get()) != CUBLAS_STATUS_SUCCESS)
      return set_error(NNPP_ERR_CUDA, "coarse inverse: GEMM");
    k_two_i_minus<<<eg, 256, 0, h.st>>>(n, T.get());
    NNPP_CUDA(cudaGetLastError());
    if (ns_gemm(hb, n, x, T.get(), y) != CUBLAS_STATUS_SUCCESS) return set_error(NNPP_ERR_CUDA, "coarse inverse: GEMM");
    std::swap(x, y);
  }
  // x holds the last iterate; its symmetrised copy goes to c.inv (rows of stride ld)
  k_symmetrize<<<eg, 256, 0, h.st>>>(n, c.ld, x, c.rowabs.get(), c.inv.get());
  NNPP_CUDA(cudaGetLastError());
  *warm_out = warm;
  *steps_out = steps;
  return NNPP_OK;
}

nnpp_status coarse_refresh(Handle& h) {
  Coarse& c = h.coarse;
  if (!h.coarse_enabled || c.n == 0) return NNPP_OK;
  const Layout& L = h.lay;
  const int n = c.n;
  if (!c.st27.alloc(27 * (size_t)n) || !c.x.alloc((size_t)n * n))
    return set_error(NNPP_ERR_NOMEM, "coarse inverse");
  if (!c.snap.alloc(h.N) || !c.count.alloc(1) || !c.tag.alloc(h.N) || !c.dn.alloc(h.N) || !c.mask.alloc(h.N))
    return set_error(NNPP_ERR_NOMEM, "coarse operator");
  KParams kp = make_kparams(h, h.cur);
  const int mixed = h.state_prec == NNPP_MIXED ? 1 : 0;
  // A P (kept for the deflated CG) and from it A_c.  With aggregates two or more bins wide a node's
  // three bins an axis lie in at most two of them: eight neighbours, else 27.
  const int cap = c.f >= 2 ? 8 : 27;
  NNPP_CUDA(cudaMemsetAsync(c.count.get(), 0, sizeof(int), h.st));
  k_node_tags<<<std::max(1, std::min((h.N + 255) / 256, 152 * 16)), 256, 0, h.st>>>(kp, mixed, c.na[0], c.na[1],
                                                                                   c.tag.get());
  const int ab = std::max(1, std::min((h.N + kApBlock - 1) / kApBlock, 152 * 32));
  if (c.f >= 2)
    k_ap_rows<true><<<ab, kApBlock, 0, h.st>>>(kp, c.tag.get(), c.na[0], c.na[1], cap, c.count.get(), c.ap_col.get(),
                                               c.ap_val.get(), c.dn.get(), c.mask.get());
  else
    k_ap_rows<false><<<ab, kApBlock, 0, h.st>>>(kp, c.tag.get(), c.na[0], c.na[1], cap, c.count.get(), c.ap_col.get(),
                                                c.ap_val.get(), c.dn.get(), c.mask.get());
  k_coarse_assemble<<<std::max(1, std::min((n + kSumWarps - 1) / kSumWarps, 152 * 16)), 32 * kSumWarps, 0, h.st>>>(
      kp, L.bin_start.get(), L.nb[0], L.nb[1], L.nb[2], c.f, c.na[0], c.na[1], c.na[2], c.ap_val.get(), c.dn.get(),
      c.mask.get(), c.st27.get(), c.rowabs.get());
  NNPP_CUDA(cudaGetLastError());
  int bad = 1, used = 0;
  if (coarse_planes(c.na, c.blocks)) {
    if (!coarse_blocks_alloc(c.blocks)) return set_error(NNPP_ERR_NOMEM, "coarse inverse");
    NNPP_TRY(coarse_direct_inverse(c.blocks, c.na, c.st27.get(), c.rowabs.get(), c.x.get(), c.inv.get(), c.ld, h.st));
    NNPP_CUDA(cudaMemcpyAsync(&bad, c.blocks.bad.get(), sizeof(int), cudaMemcpyDeviceToHost, h.st));
  }
  NNPP_CUDA(cudaMemcpyAsync(&used, c.count.get(), sizeof(int), cudaMemcpyDeviceToHost, h.st));
  NNPP_CUDA(cudaStreamSynchronize(h.st));
  c.ap_k = std::max(1, std::min(used, cap));
  bool warm = false;
  int steps = 0;
  if (bad) NNPP_TRY(newton_schulz_inverse(h, &warm, &steps));
  c.ns_valid = bad != 0;
  k_phase_snap<<<std::max(1, std::min((h.N + 255) / 256, 152 * 16)), 256, 0, h.st>>>(
      kp, h.state_prec == NNPP_MIXED ? 1 : 0, c.snap.get());
  NNPP_CUDA(cudaGetLastError());
  c.valid = true;
  c.stale = false;
  c.rebuilds += 1;
  c.warm_rebuilds += warm ? 1 : 0;
  c.ns_steps = steps;
  h.coarse_event_cur = -1;
  // the coarse operator and A P match the phases now
  static const int kOne = 1;
  NNPP_CUDA(cudaMemcpyAsync(&h.dstate.get()->defl, &kOne, sizeof(int), cudaMemcpyHostToDevice, h.st));
  return NNPP_OK;
}

nnpp_status coarse_check(Handle& h) {
  Coarse& c = h.coarse;
  if (!h.coarse_enabled || !c.valid || h.coarse_replay) return NNPP_OK;
  KParams kp = make_kparams(h, h.cur);
  NNPP_CUDA(cudaMemsetAsync(c.count.get(), 0, sizeof(int), h.st));
  k_phase_diff<<<std::max(1, std::min((h.N + 255) / 256, 152 * 16)), 256, 0, h.st>>>(
      kp, h.state_prec == NNPP_MIXED ? 1 : 0, c.snap.get(), c.count.get());
  NNPP_CUDA(cudaGetLastError());
  int changed = 0;
  NNPP_CUDA(cudaMemcpyAsync(&changed, c.count.get(), sizeof(int), cudaMemcpyDeviceToHost, h.st));
  NNPP_CUDA(cudaStreamSynchronize(h.st));
  if (changed == 0) return NNPP_OK;
  const auto t0 = std::chrono::steady_clock::now();
  NNPP_TRY(coarse_refresh(h));
  NNPP_CUDA(cudaStreamSynchronize(h.st));
  c.rebuild_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  c.timed_rebuilds += 1;
  if (h.coarse_record) NNPP_TRY(coarse_record_event(h, h.nstep - h.coarse_base));
  return NNPP_OK;
}

nnpp_status coarse_record_event(Handle& h, long long step) {
  const Coarse& c = h.coarse;
  h.coarse_events.emplace_back();
  Handle::CoarseEvent& ev = h.coarse_events.back();
  ev.step = step;
  const size_t nn = c.inv_elems();
  const size_t na = (size_t)c.ap_k * h.N;
  ev.ap_k = c.ap_k;
  if (!ev.inv.alloc(nn) || !ev.ap_col.alloc(na) || !ev.ap_val.alloc(na) || !ev.snap.alloc(h.N))
    return set_error(NNPP_ERR_NOMEM, "recorded coarse operator");
  NNPP_CUDA(cudaMemcpyAsync(ev.snap.get(), c.snap.get(), (size_t)h.N, cudaMemcpyDeviceToDevice, h.st));
  NNPP_CUDA(cudaMemcpyAsync(ev.inv.get(), c.inv.get(), sizeof(float) * nn, cudaMemcpyDeviceToDevice, h.st));
  NNPP_CUDA(cudaMemcpyAsync(ev.ap_col.get(), c.ap_col.get(), sizeof(int) * na, cudaMemcpyDeviceToDevice, h.st));
  NNPP_CUDA(cudaMemcpyAsync(ev.ap_val.get(), c.ap_val.get(), sizeof(float) * na, cudaMemcpyDeviceToDevice, h.st));
  return NNPP_OK;
}

nnpp_status coarse_select(Handle& h, long long step, bool recompute) {
  if (h.coarse_events.empty()) return NNPP_OK;
  int e = 0;
  while (e + 1 < (int)h.coarse_events.size() && h.coarse_events[e + 1].step <= step) ++e;
  if (e != h.coarse_event_cur) {
    Coarse& c = h.coarse;
    const Handle::CoarseEvent& ev = h.coarse_events[e];
    const size_t nn = c.inv_elems();
    const size_t na = (size_t)ev.ap_k * h.N;
    c.ap_k = ev.ap_k;
    NNPP_CUDA(cudaMemcpyAsync(c.inv.get(), ev.inv.get(), sizeof(float) * nn, cudaMemcpyDeviceToDevice, h.st));
    NNPP_CUDA(cudaMemcpyAsync(c.ap_col.get(), ev.ap_col.get(), sizeof(int) * na, cudaMemcpyDeviceToDevice, h.st));
    NNPP_CUDA(cudaMemcpyAsync(c.ap_val.get(), ev.ap_val.get(), sizeof(float) * na, cudaMemcpyDeviceToDevice, h.st));
    NNPP_CUDA(cudaMemcpyAsync(c.snap.get(), ev.snap.get(), (size_t)h.N, cudaMemcpyDeviceToDevice, h.st));
    h.coarse_event_cur = e;
  }
  // recomputing the step the forward rebuilt the operator before: the deflation resumed there
  if (recompute && step > 0 && h.coarse_events[e].step == step) {
    static const int kOn = 1;
    NNPP_CUDA(cudaMemcpyAsync(&h.dstate.get()->defl, &kOn, sizeof(int), cudaMemcpyHostToDevice, h.st));
  }
  return NNPP_OK;
}

nnpp_status coarse_defl_check(Handle& h) {
  Coarse& c = h.coarse;
  if (!h.coarse_enabled || !c.valid) {
    NNPP_CUDA(cudaMemsetAsync(&h.dstate.get()->defl, 0, sizeof(int), h.st));
    return NNPP_OK;
  }
  KParams kp = make_kparams(h, h.cur);
  NNPP_CUDA(cudaMemsetAsync(c.count.get(), 0, sizeof(int), h.st));
  k_phase_diff<<<std::max(1, std::min((h.N + 255) / 256, 152 * 16)), 256, 0, h.st>>>(
      kp, h.state_prec == NNPP_MIXED ? 1 : 0, c.snap.get(), c.count.get());
  k_defl_from_count<<<1, 1, 0, h.st>>>(h.dstate.get(), c.count.get());
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

}  // namespace nnpp
