// implicit.cu -- the reference's production time step on the GPU: backward Euler with one
// tangent per step and modified Newton iterations, each solving every field's correction by
// left-Jacobi GMRES(30) (main.cpp:640-922, utils::NewtonMatrices utils.h:844-1849,
// Eigen::GMRES GMRES.h:56-203).  FP64 throughout, node order of the reference (the user's).
//
//   per step   tangents K_f at U^n: species k (utils.h:900-1102) off-diagonal
//              -(K1 D(BV) + K2 D(BV) z F/(RT) (phi^n_n - phi^n_i)) w per bond, diagonal
//              1/dt + sum K1 D(BV) w; the potential K11 (utils.h:1797-1848) -w on
//              liquid-liquid bonds, their sum on the diagonal; Dirichlet rows (and potential
//              rows without liquid-liquid bonds) identity; w = beta dV / xi^3.  The
//              off-diagonals of every field are stored per bond for the step (the GB300's FP64
//              rate made forming them in every GMRES product the product's bound), on slices
//              of 32 rows, bond column by bond column, one lane a row: a warp-wide FP64
//              instruction holds an SM sub-partition's FP64 pipe for 64 cycles, so the sums
//              over a warp's lanes that a warp per row needs cost more than the products.
//   Newton     F = Residuals(U^{n+1}, U^n) with the migration on phi^n (utils.h:126), F11's
//              charge from U^n (utils.h:829-831), and
//              F = U - bc on Dirichlet rows (main.cpp:676-712); K_f dU_f = -F_f by GMRES for
//              the species and the potential at once (independent Krylov solves advanced
//              together: one pass over the bonds serves every field); U += dU; the clamp
//              (main.cpp:805-837); stop when max_f | ||dU_f|| - ||dU_f||_prev | < EPS.
//   then       the phase flip (main.cpp:914-922) and the volume every sub_step_no steps.
//
// GMRES follows Eigen's (GMRES.h:56-203): initial guess x = b (GMRES.h:330-334), the
// diagonal preconditioner on the left, restarts every 30 steps, iterations counted across
// restarts up to MAX_ITER, stop when |g_k| / ||M^-1 (b - K x_0)|| < EPS.  The Arnoldi basis is
// orthogonalised by classical Gram-Schmidt applied twice (the same Krylov space and
// least-squares problem as Eigen's Householder form; one reduction pass per sweep instead of
// k dependent ones).  Reductions are block partials summed in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "engine.cuh"

using namespace nnpp;

struct nnpp_handle {
  Handle h;
};

namespace {

constexpr int F5 = S + 1;          // fields: the species and the potential
constexpr int kRestart = 30;       // Eigen::GMRES's default restart (GMRES.h:282)
constexpr double kEps = 10E-6;     // EPS, main.cpp:33-36
constexpr int kMaxIter = 200;      // MAX_ITER, main.cpp:33-36
constexpr int kTB = 256;
constexpr int kDotBlocks = 304;    // two per SM
constexpr int kChemFields = 11;    // fields of the complete model

// bond classes by the two nodes' phases; the coefficients' tables are indexed by them
enum BondClass { kLL = 0, kMixed = 1, kSS = 2 };

template <int NS>
struct ImpCtxT {
  int N;
  const int* ptr;                  // CSR row starts over user indices, self excluded
  // rows in slices of 32 (slice s: rows 32 s ..), bond c of row 32 s + l at
  // 32 (soff[s] + c) + l; padding: the row itself, weight 0
  int nslices;
  const int* soff;                 // nslices + 1, in columns
  const int* scol;
  const double* sw;                // per bond: beta dV / xi^3
  long long slots;
  const unsigned char* dir;        // (NS + 1) * N Dirichlet flags
  const double* bc;                // (NS + 1) * N boundary values (species / CSolid)
  const int* phase;                // N
  const double* u0;                // (NS + 1) * N: U^n (its potential is the migration's phi^n)
  const double* dinv;              // (NS + 1) * N: the tangents' inverse diagonals
  const double* toff;              // (NS + 1) * slots: the tangents' off-diagonals per bond
  double dt, csat, k_diss, sw_width, lam, kphis;
  // bond coefficients of species k by class (utils.h:100-153, 202-239; zero where the bond is
  // absent: solid-solid for k >= 1): K1 D(BV) and K2 D(BV) z F / (RT)
  double f1[3][NS], f2[3][NS], z[NS];
  double k7b, k8b, k9b;            // the complete model's rates in its tangents' diagonals
};
using ImpCtx = ImpCtxT<S>;

__device__ __forceinline__ int bond_class(int pi, int pn) { return pi + pn; }

template <int NS>
void set_coefficients(ImpCtxT<NS>& c, const double* K1, const double* K2zF, const double* DL, const double* DSo,
                      double bvmix) {
  for (int k = 0; k < NS; ++k) {
    const double D[3] = {DL[k], k == 0 ? DSo[k] * bvmix : DSo[k], k == 0 ? DSo[k] : 0.0};
    for (int q = 0; q < 3; ++q) {
      c.f1[q][k] = K1[k] * D[q];
      c.f2[q][k] = K2zF[k] * D[q];
    }
  }
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// columns of every slice: its longest row
__global__ void k_imp_widths(int N, const int* ptr, int nslices, int* width) {
  const int lane = threadIdx.x & 31;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < nslices; g += (gridDim.x * blockDim.x) >> 5) {
    const int i = 32 * g + lane;
    const int len = __reduce_max_sync(0xffffffffu, i < N ? ptr[i + 1] - ptr[i] : 0);
    if (lane == 0) width[g] = len;
  }
}

// the sliced columns and weights w = beta dV / xi^3 (utils.h:17-25, the bond terms'
// xi^(3+2s) beta dV with s = 0)
__global__ void k_imp_weights(int N, const int* ptr, const int* col, const double* x, const double* y,
                              const double* z, double delta, double dx, double dV, int nslices, const int* soff,
                              int* scol, double* sw) {
  const int lane = threadIdx.x & 31;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < nslices; g += (gridDim.x * blockDim.x) >> 5) {
    const int i = 32 * g + lane;
    const int c0 = soff[g], width = soff[g + 1] - c0;
    const int j0 = i < N ? ptr[i] : 0, len = i < N ? ptr[i + 1] - j0 : 0;
    for (int c = 0; c < width; ++c) {
      int n = i < N ? i : 0;
      double w = 0.0;
      if (c < len) {
        n = col[j0 + c];
        const double a = x[n] - x[i], b = y[n] - y[i], d = z[n] - z[i];
        const double xi = sqrt(a * a + b * b + d * d);
        w = beta_fn<double>(xi, delta, dx) * dV / (xi * xi * xi);
      }
      scol[32 * (size_t)(c0 + c) + lane] = n;
      sw[32 * (size_t)(c0 + c) + lane] = w;
    }
  }
}

// the tangents' inverse diagonals (lane per row): the classes' weight sums times their coefficients.  The
// complete model (NS = 10) adds the linearised reaction terms of utils::NewtonMatrices at U^n: H+
// on interface and liquid nodes (utils.h:1089-1098), species 3, 4, 5 and 7 on liquid nodes
// (1176-1182, 1266-1271, 1356-1361, 1546-1551).
template <int NS>
__global__ void k_imp_diag(ImpCtxT<NS> c, double* dinv) {
  const int lane = threadIdx.x & 31;
  const int N = c.N;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < c.nslices; g += (gridDim.x * blockDim.x) >> 5) {
    const int i = 32 * g + lane;
    if (i >= N) continue;
    const size_t s0 = 32 * (size_t)c.soff[g] + lane;
    const int len = c.ptr[i + 1] - c.ptr[i];
    const int pi = c.phase[i];
    double wl = 0.0, ws = 0.0;  // weight sums of the liquid and of the solid neighbours
    int liquids = 0;
    for (int j = 0; j < len; ++j) {
      const double w = c.sw[s0 + 32 * (size_t)j];
      if (c.phase[c.scol[s0 + 32 * (size_t)j]] == 0) {
        wl += w;
        ++liquids;
      } else {
        ws += w;
      }
    }
    const bool liq = pi == 0;
    const bool iface = !liq && liquids > 0;
    for (int k = 0; k < NS; ++k) {
      double R = 0.0;
      if (NS == 10) {
        auto u = [&](int f) { return c.u0[(size_t)f * N + i]; };
        if (k == 1 && (iface || liq))
          R = c.k7b * (-u(2)) + c.k8b * (-u(4)) + c.k9b * (-u(6));
        else if (k == 2 && liq)
          R = c.k7b * (-u(1));
        else if ((k == 3 || k == 4) && liq)
          R = c.k8b * (-u(1));
        else if (k == 6 && liq)
          R = c.k9b * (-u(1));
      }
      const double sk = c.f1[bond_class(pi, 0)][k] * wl + c.f1[bond_class(pi, 1)][k] * ws;
      dinv[(size_t)k * N + i] = c.dir[(size_t)k * N + i] ? 1.0 : 1.0 / (1.0 / c.dt + sk - R);
    }
    dinv[(size_t)NS * N + i] = (c.dir[(size_t)NS * N + i] || !liq || liquids == 0) ? 1.0 : 1.0 / wl;
  }
}

// Residual of the implicit step (utils.h:72-257, 798-841; Dirichlet rows main.cpp:676-712), K warps
// a slice (see k_imp_apply), each bond's terms w (c_n - c_i) and w dphi c_n summed apart for liquid
// and solid neighbours, the coefficients applied to the sums: 16 FP64 instructions a bond.
template <int K>
__global__ void __launch_bounds__(128) k_imp_residual(ImpCtx c, const double* u1, double* F) {
  constexpr int NV = 4 * S + 1;
  __shared__ double sm[K > 1 ? (K - 1) * NV * 32 : 1];
  __shared__ int s_liq[K > 1 ? K * 32 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = K > 1 ? warp : 0;
  const int N = c.N;
  const double* phi0 = c.u0 + (size_t)S * N;
  const double* phi1 = u1 + (size_t)S * N;
  const int per = 4 / K;
  for (int g0 = blockIdx.x * per; g0 < c.nslices; g0 += gridDim.x * per) {
    const int g = g0 + (K > 1 ? 0 : warp);
    const int i = 32 * g + lane;
    const bool live = g < c.nslices && i < N;
    double a[NV];  // [0, S): w d over liquid neighbours, then w dphi c_n; the same over solid ones; potential
#pragma unroll
    for (int q = 0; q < NV; ++q) a[q] = 0.0;
    double ci[S];
    int pi = 0, liquids = 0;
    if (live) {
      const size_t s0 = 32 * (size_t)c.soff[g] + lane;
      const int len = c.ptr[i + 1] - c.ptr[i];
      pi = c.phase[i];
      const double p0 = phi0[i], p1 = phi1[i];
#pragma unroll
      for (int k = 0; k < S; ++k) ci[k] = u1[(size_t)k * N + i];
#pragma unroll 2
      for (int j = part; j < len; j += K) {
        const int n = c.scol[s0 + 32 * (size_t)j];
        const double w = c.sw[s0 + 32 * (size_t)j];
        const double wd = w * (phi0[n] - p0);
        if (c.phase[n] == 0) {
          ++liquids;
#pragma unroll
          for (int k = 0; k < S; ++k) {
            const double cn = u1[(size_t)k * N + n];
            a[k] = fma(w, cn - ci[k], a[k]);
            a[S + k] = fma(wd, cn, a[S + k]);
          }
          if (pi == 0) a[4 * S] = fma(w, phi1[n] - p1, a[4 * S]);
        } else {
#pragma unroll
          for (int k = 0; k < S; ++k) {
            const double cn = u1[(size_t)k * N + n];
            a[2 * S + k] = fma(w, cn - ci[k], a[2 * S + k]);
            a[3 * S + k] = fma(wd, cn, a[3 * S + k]);
          }
        }
      }
    }
    if (K > 1) {
      if (part > 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sm[((part - 1) * NV + q) * 32 + lane] = a[q];
      s_liq[part * 32 + lane] = liquids;
      __syncthreads();
      if (part == 0)
        for (int h = 0; h < K - 1; ++h) {
#pragma unroll
          for (int q = 0; q < NV; ++q) a[q] += sm[(h * NV + q) * 32 + lane];
          liquids += s_liq[(h + 1) * 32 + lane];
        }
    }
    if (live && part == 0) {
      const bool iface = pi == 1 && liquids > 0, ll = pi == 0 && liquids > 0;
      const int cl = bond_class(pi, 0), cs = bond_class(pi, 1);
#pragma unroll
      for (int k = 0; k < S; ++k) {
        const double s1 = -(c.f1[cl][k] * a[k] + c.f1[cs][k] * a[2 * S + k]);
        const double s2 = -(c.f2[cl][k] * a[S + k] + c.f2[cs][k] * a[3 * S + k]);
        double R = 0.0;
        if (k == 0 && iface) {
          const double sw = c.sw_width > 0.0 ? 1.0 / (1.0 + exp(-(ci[0] - c.csat) / c.sw_width))
                                             : (ci[0] > c.csat ? 1.0 : 0.0);
          R = -c.k_diss * sw;
        }
        double f = ((ci[k] - c.u0[(size_t)k * N + i]) / c.dt) + s1 + s2 - R;
        if (c.dir[(size_t)k * N + i]) f = ci[k] - c.bc[(size_t)k * N + i];
        F[(size_t)k * N + i] = f;
      }
      // F11 from phi^{n+1} and the charge of U^n (utils.h:829-831)
      double f11 = 0.0;
      if (ll) {
        double r11 = 0.0;
        for (int k = 0; k < S; ++k) r11 += c.z[k] * c.u0[(size_t)k * N + i];
        f11 = -a[4 * S] - c.lam * r11;
      }
      if (c.dir[(size_t)S * N + i]) f11 = phi1[i] - c.bc[(size_t)S * N + i];
      F[(size_t)S * N + i] = f11;
    }
    if (K > 1) __syncthreads();
  }
}

// the tangents' off-diagonals of every bond: the species' -(K1 D(BV) + K2 D(BV) z F/(RT)
// (phi^n_n - phi^n_i)) w (utils.h:900-1792), zero where the bond is absent, and the potential's -w on
// liquid-liquid bonds; formed once a step, read by every GMRES iteration's product (lane per row)
template <int NS>
__global__ void k_imp_tangent(ImpCtxT<NS> c, double* toff) {
  const int lane = threadIdx.x & 31;
  const int N = c.N;
  const double* phi0 = c.u0 + (size_t)NS * N;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < c.nslices; g += (gridDim.x * blockDim.x) >> 5) {
    const int i = 32 * g + lane;
    const int c0 = c.soff[g], width = c.soff[g + 1] - c0;
    const int pi = i < N ? c.phase[i] : 0;
    const double p0 = i < N ? phi0[i] : 0.0;
    for (int j = 0; j < width; ++j) {
      const size_t o = 32 * (size_t)(c0 + j) + lane;
      const int n = c.scol[o];
      const double w = c.sw[o];
      const double wd = w * (phi0[n] - p0);
      const int q = bond_class(pi, c.phase[n]);
#pragma unroll
      for (int k = 0; k < NS; ++k) toff[(size_t)k * c.slots + o] = -fma(c.f2[q][k], wd, c.f1[q][k] * w);
      toff[(size_t)NS * c.slots + o] = q == kLL ? -w : 0.0;
    }
  }
}

// out_f = s_f M^-1 K_f v_f for NA fields f[0..NA) (s_f: the normalisation of v_f, scale[f * stride],
// or 1 without it): the tangents' products in one pass over the bonds, a
// lane per row.  K warps take a slice's columns in turn (K = 4 while the slices alone would leave
// the chip's warps idle) and their sums meet in shared memory.  Bound by the FP64 pipe for many
// fields (one FMA a bond and field) and by the loads in flight for one.
struct FieldList {
  int f[kChemFields];
};
template <int NA, int K>
__global__ void __launch_bounds__(128) k_imp_apply(int N, const int* __restrict__ ptr, int nslices,
                                                   const int* __restrict__ soff, const int* __restrict__ scol,
                                                   const double* __restrict__ toff, long long slots,
                                                   const double* __restrict__ dinv, const unsigned char* __restrict__ dir,
                                                   const double* __restrict__ v, double* __restrict__ out, FieldList fl,
                                                   const double* __restrict__ scale, int stride) {
  constexpr int U = NA == 1 ? 8 : NA <= 3 ? 4 : 2;  // bond columns in flight
  __shared__ double sm[K > 1 ? K * NA * 32 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = K > 1 ? warp : 0;
  const int per = 4 / K;
  for (int g0 = blockIdx.x * per; g0 < nslices; g0 += gridDim.x * per) {
    const int g = g0 + (K > 1 ? 0 : warp);
    const int i = 32 * g + lane;
    const bool live = g < nslices && i < N;
    double acc[NA];
#pragma unroll
    for (int q = 0; q < NA; ++q) acc[q] = 0.0;
    if (live) {
      const size_t s0 = 32 * (size_t)soff[g] + lane;
      const int len = ptr[i + 1] - ptr[i];
      int j = part;
      for (; j + (U - 1) * K < len; j += U * K) {
        int n[U];
#pragma unroll
        for (int u = 0; u < U; ++u) n[u] = scol[s0 + 32 * (size_t)(j + u * K)];
        double t[U][NA], x[U][NA];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < NA; ++q) t[u][q] = toff[(size_t)fl.f[q] * slots + s0 + 32 * (size_t)(j + u * K)];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < NA; ++q) x[u][q] = v[(size_t)fl.f[q] * N + n[u]];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < NA; ++q) acc[q] = fma(t[u][q], x[u][q], acc[q]);
      }
      for (; j < len; j += K) {
        const size_t o = s0 + 32 * (size_t)j;
        const int n = scol[o];
#pragma unroll
        for (int q = 0; q < NA; ++q) acc[q] = fma(toff[(size_t)fl.f[q] * slots + o], v[(size_t)fl.f[q] * N + n], acc[q]);
      }
    }
    // the parts' sums: part p takes the fields p, p + K, ... and finishes their rows
    if (K > 1) {
#pragma unroll
      for (int q = 0; q < NA; ++q) sm[(part * NA + q) * 32 + lane] = acc[q];
      __syncthreads();
    }
    if (live)
#pragma unroll
      for (int q = 0; q < NA; ++q) {
        if (K > 1 && q % K != part) continue;
        double sum = acc[q];
        if (K > 1) {
          sum = sm[q * 32 + lane];
#pragma unroll
          for (int h = 1; h < K; ++h) sum += sm[(h * NA + q) * 32 + lane];
        }
        const size_t o = (size_t)fl.f[q] * N + i;
        // identity rows: Dirichlet, and potential rows without liquid-liquid bonds (diagonal 1
        // and no off-diagonal term then; a Dirichlet row's bonds are dropped here)
        const double r = fma(dir[o] ? 0.0 : sum, dinv[o], v[o]);
        out[o] = scale ? scale[(size_t)fl.f[q] * stride] * r : r;
      }
    if (K > 1) __syncthreads();
  }
}

// ---------------------------------------------------------------- GMRES on the device ----
// State of the fields' GMRES solves (one block a field).  The Arnoldi vectors are stored as the
// orthogonalised vectors before their normalisation (V^_q, with V_q = s_q V^_q), so that no pass
// only scales; the Hessenberg columns, the rotations and the stop test live on the device, and
// the host launches iterations ahead of their outcome (kernels of finished fields return at
// once), so that no iteration waits for the host.
struct GmField {
  double H[(kRestart + 1) * kRestart];  // H[q * kRestart + k]: row q, column k
  double cs[kRestart], sn[kRestart], g[kRestart + 1], s[kRestart + 1], y[kRestart];
  double coef[kRestart + 1];            // the combination's coefficients of V^_q
  double r0n;                           // ||M^-1 (b - K x_0)||
  int it;                               // iterations, over restarts
  int k;                                // basis vectors of the finished cycle (0: none)
};
struct GmState {
  GmField f[kChemFields];
  int cycle;    // fields iterating in this cycle
  int restart;  // fields whose cycle ended without convergence
  unsigned int ticket[(kRestart + 1) * kChemFields];
};

// sum of a block's values in thread 0 (kTB threads)
__device__ __forceinline__ double block_sum1(double v, double* sm) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int u = 0; u < kTB / 32; ++u) t += sm[u];
  return t;
}

// true in every thread of the last of the gridDim.x blocks that share a ticket, once all of their
// partials are written (the values of a launch are independent of one another: each has its own
// ticket, and the blocks that finish them work side by side)
__device__ __forceinline__ bool last_block(unsigned int* ticket, int* s_flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const bool last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0;
    *s_flag = last ? 1 : 0;
  }
  __syncthreads();
  if (*s_flag) __threadfence();
  return *s_flag != 0;
}

// the sum of nb partials by one warp, in a fixed order (every lane holds it)
__device__ __forceinline__ double warp_partials(const double* part, int nb) {
  double t = 0.0;
  for (int b = threadIdx.x & 31; b < nb; b += 32) t += __ldcg(part + b);
  return warp_sum(t);
}

// A cycle's start for the fields fl (grid: blocks x fields): V^_0 = M^-1 (b - K x) = b dinv - t,
// its norm; the first cycle also finds the fields with b = 0 (x = 0) and records ||r_0||.  The
// fields that iterate enter st->cycle, which the previous cycle left empty.
__global__ void __launch_bounds__(kTB) k_gm_start(int N, int first, FieldList fl, const double* b, const double* dinv,
                                                  const double* t, double* V, GmState* st, double* part) {
  __shared__ double sm[kTB / 32];
  __shared__ int s_last;
  const int f = fl.f[blockIdx.y], nb = gridDim.x;
  const size_t o = (size_t)f * N;
  double rr = 0.0, bb = 0.0;
  for (int i = blockIdx.x * kTB + threadIdx.x; i < N; i += nb * kTB) {
    const double bi = b[o + i];
    const double r = fma(bi, dinv[o + i], -t[o + i]);
    V[o + i] = r;
    rr += r * r;
    bb += bi * bi;
  }
  const double trr = block_sum1(rr, sm);
  __syncthreads();
  const double tbb = block_sum1(bb, sm);
  if (threadIdx.x == 0) {
    part[(size_t)(2 * blockIdx.y) * nb + blockIdx.x] = trr;
    part[(size_t)(2 * blockIdx.y + 1) * nb + blockIdx.x] = tbb;
  }
  if (!last_block(&st->ticket[blockIdx.y], &s_last) || threadIdx.x >= 32) return;
  const double beta = sqrt(warp_partials(part + (size_t)(2 * blockIdx.y) * nb, nb));
  const double b2 = warp_partials(part + (size_t)(2 * blockIdx.y + 1) * nb, nb);
  if (threadIdx.x == 0) {
    GmField& g = st->f[f];
    bool on = true;
    if (first) {
      g.it = 0;
      g.r0n = beta;
      on = b2 != 0.0 && beta != 0.0;
    }
    g.k = 0;
    g.g[0] = beta;
    g.s[0] = beta != 0.0 ? 1.0 / beta : 0.0;
    if (on) atomicOr(&st->cycle, 1 << f);
  }
}

// A Gram-Schmidt pass's dot products h_q = <w, V_q>, q < k (grid: blocks x k x fields; w = V^_k);
// a product's last block adds it to the Hessenberg column and forms the combination's coefficient.
__global__ void __launch_bounds__(kTB) k_gm_dots(int N, int k, int pass, FieldList fl, int nf, const double* V,
                                                 GmState* st, double* part) {
  __shared__ double sm[kTB / 32];
  __shared__ int s_last;
  const int cycle = *(volatile const int*)&st->cycle;
  const int f = fl.f[blockIdx.z], q = blockIdx.y, nb = gridDim.x, na = gridDim.z;
  const size_t FN = (size_t)nf * N;
  if (!((cycle >> f) & 1)) return;
  const double* w = V + k * FN + (size_t)f * N;
  const double* v = V + q * FN + (size_t)f * N;
  double s = 0.0;
#pragma unroll 4
  for (int i = blockIdx.x * kTB + threadIdx.x; i < N; i += nb * kTB) s += w[i] * v[i];
  const double t = block_sum1(s, sm);
  if (threadIdx.x == 0) part[(size_t)(q * na + blockIdx.z) * nb + blockIdx.x] = t;
  if (!last_block(&st->ticket[q * kChemFields + f], &s_last) || threadIdx.x >= 32) return;
  GmField& g = st->f[f];
  const double h = g.s[q] * warp_partials(part + (size_t)(q * na + blockIdx.z) * nb, nb);
  if (threadIdx.x == 0) {
    double* H = &g.H[q * kRestart + k - 1];
    *H = pass == 0 ? h : *H + h;
    g.coef[q] = h * g.s[q];
  }
}

// the Givens step of a field's new Hessenberg column (k - 1, with norm2 = ||w||^2), the stop test of
// Eigen's GMRES and, when the field's cycle ends, y = H^-1 g.  One warp: the column, the earlier
// rotations and, at the end, the rows a lane each, handed on by shuffles.  Returns 0 (goes on), 1
// (converged or at the iteration cap) or 2 (restart), to every lane.
__device__ int gm_rotate(GmField& g, int k, int N, double norm2) {
  const int lane = threadIdx.x & 31;
  double* H = g.H;
  // lane q: H[q][k - 1] and rotation q (k <= 30)
  double h = lane < k ? H[lane * kRestart + k - 1] : 0.0;
  const double cl = lane < k - 1 ? g.cs[lane] : 1.0, sl = lane < k - 1 ? g.sn[lane] : 0.0;
  double a = __shfl_sync(0xffffffffu, h, 0);
  for (int q = 0; q < k - 1; ++q) {
    const double b = __shfl_sync(0xffffffffu, h, q + 1);
    const double c = __shfl_sync(0xffffffffu, cl, q), s = __shfl_sync(0xffffffffu, sl, q);
    if (lane == q) h = c * a + s * b;
    a = -s * a + c * b;
  }
  // den = sqrt(a^2 + ||w||^2) and the rotation from reciprocal square roots: a division takes two
  // dozen FP64 instructions of 64 cycles each, and this is a chain
  const double rk = norm2 > 0.0 ? rsqrt(norm2) : 0.0, hk = norm2 * rk;  // ||w||, its reciprocal
  const double d2 = fma(a, a, norm2), rd = d2 > 0.0 ? rsqrt(d2) : 0.0, den = d2 * rd;
  const double c = rd == 0.0 ? 1.0 : a * rd, s = hk * rd;
  if (lane == k - 1) h = den;
  if (lane < k) H[lane * kRestart + k - 1] = h;
  const double gk = g.g[k - 1], gn = -s * gk;
  const int it = g.it + 1;
  __syncwarp();
  if (lane == 0) {
    g.s[k] = rk;
    g.cs[k - 1] = c;
    g.sn[k - 1] = s;
    g.g[k] = gn;
    g.g[k - 1] = c * gk;
    g.it = it;
  }
  const bool stop = k == N || fabs(gn) < kEps * g.r0n || it == kMaxIter;
  const int end = stop ? 1 : k == kRestart ? 2 : 0;
  __syncwarp();
  if (end) {
    if (lane == 0) g.k = k;
    // back substitution, a row a lane
    double r = lane < k ? g.g[lane] : 0.0;
    for (int q = k - 1; q >= 0; --q) {
      const double y = __shfl_sync(0xffffffffu, r, q) / H[q * kRestart + q];
      if (lane == q) g.y[q] = y;
      if (lane < q) r -= H[lane * kRestart + q] * y;
    }
  }
  return end;
}

// w -= sum_q coef_q V^_q (grid: blocks x fields); NORM: the second pass, where a field's last block
// takes its norm and makes its Givens step and decision.
template <bool NORM>
__global__ void __launch_bounds__(kTB) k_gm_combine(int N, int k, FieldList fl, int nf, double* V, GmState* st,
                                                    double* part) {
  __shared__ double sm[kTB / 32];
  __shared__ int s_last;
  const int cycle = *(volatile const int*)&st->cycle;
  const int f = fl.f[blockIdx.y], nb = gridDim.x;
  const size_t FN = (size_t)nf * N;
  if (!((cycle >> f) & 1)) return;
  double n2 = 0.0;
  const double* coef = st->f[f].coef;
  double* w = V + k * FN + (size_t)f * N;
  const double* v0 = V + (size_t)f * N;
  for (int i = blockIdx.x * kTB + threadIdx.x; i < N; i += nb * kTB) {
    double a[4] = {w[i], 0.0, 0.0, 0.0};
    int q = 0;
    for (; q + 4 <= k; q += 4) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = v0[(size_t)(q + u) * FN + i];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = fma(-coef[q + u], v[u], a[u]);
    }
    for (; q < k; ++q) a[0] = fma(-coef[q], v0[(size_t)q * FN + i], a[0]);
    const double r = (a[0] + a[1]) + (a[2] + a[3]);
    w[i] = r;
    if (NORM) n2 += r * r;
  }
  if (!NORM) return;
  const double t = block_sum1(n2, sm);
  if (threadIdx.x == 0) part[(size_t)blockIdx.y * nb + blockIdx.x] = t;
  if (!last_block(&st->ticket[f], &s_last) || threadIdx.x >= 32) return;
  const int end = gm_rotate(st->f[f], k, N, warp_partials(part + (size_t)blockIdx.y * nb, nb));
  if (end && threadIdx.x == 0) {
    if (end == 2) atomicOr(&st->restart, 1 << f);
    atomicAnd(&st->cycle, ~(1 << f));
  }
}

// x_f += V y for the fields whose cycle ended (grid: blocks x fields)
__global__ void __launch_bounds__(kTB) k_gm_solution(int N, FieldList fl, int nf, const double* V, const GmState* st,
                                                     double* x) {
  const int f = fl.f[blockIdx.y];
  const GmField& g = st->f[f];
  const size_t FN = (size_t)nf * N;
  const int k = g.k;
  if (k == 0) return;
  for (int i = blockIdx.x * kTB + threadIdx.x; i < N; i += gridDim.x * kTB) {
    double s = 0.0;
#pragma unroll 4
    for (int q = 0; q < k; ++q) s += (g.y[q] * g.s[q]) * V[(size_t)q * FN + (size_t)f * N + i];
    x[(size_t)f * N + i] += s;
  }
}

// block partials of ||x_f||^2 (grid: blocks x fields) and, in the last block, their sums
__global__ void __launch_bounds__(kTB) k_imp_norms(int N, const double* x, GmState* st, double* part, double* out) {
  __shared__ double sm[kTB / 32];
  __shared__ int s_last;
  const int f = blockIdx.y, nb = gridDim.x;
  double s = 0.0;
  for (int i = blockIdx.x * kTB + threadIdx.x; i < N; i += nb * kTB) s += x[(size_t)f * N + i] * x[(size_t)f * N + i];
  const double t = block_sum1(s, sm);
  if (threadIdx.x == 0) part[(size_t)f * nb + blockIdx.x] = t;
  if (!last_block(&st->ticket[f], &s_last) || threadIdx.x >= 32) return;
  const double v = warp_partials(part + (size_t)f * nb, nb);
  if (threadIdx.x == 0) out[f] = v;
}

// U += dU, then the clamp of the species (main.cpp:805-837: U1..U9 always, U10 on liquid
// nodes; the four-species model's species are the always-clamped U1..U4)
template <int NS>
__global__ void k_imp_update(int N, double* u1, const double* du, double floor_c, const int* phase) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
    for (int f = 0; f <= NS; ++f) {
      const size_t q = (size_t)f * N + i;
      double v = u1[q] + du[q];
      if (f < NS && v < floor_c && (f < 9 || phase[i] == 0)) v = floor_c;
      u1[q] = v;
    }
}

// phase flip (main.cpp:914-922); flip step into the handle's record (internal order); the
// solid volume sum of main.cpp:944-949 into per-block partials
__global__ void k_imp_flip(int N, const double* u1, int* phase, double csat, int step, const int* iperm,
                           int* flip_step, double* part) {
  __shared__ double sm[kTB / 32];
  double v = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    if (phase[i] == 1 && u1[i] <= csat) {
      phase[i] = 0;
      if (flip_step) flip_step[iperm[i]] = step;
    }
    if (phase[i] == 1) v += u1[i] - csat;
  }
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int u = 0; u < kTB / 32; ++u) t += sm[u];
    part[blockIdx.x] = t;
  }
}

// The iterations' outcome on the host: a word of device memory copied to pinned memory behind each
// recorded iteration, with an event to wait for.
struct GmStatus {
  static constexpr int kSlots = 4;
  int* host = nullptr;  // kSlots words, then (from 8) the fields' iteration counts
  cudaEvent_t ev[kSlots] = {};
  GmStatus() = default;
  GmStatus(const GmStatus&) = delete;
  GmStatus& operator=(const GmStatus&) = delete;
  ~GmStatus() {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    if (host) cudaFreeHost(host);
  }
  nnpp_status init() {
    if (host) return NNPP_OK;
    if (cudaMallocHost(reinterpret_cast<void**>(&host), 64 * sizeof(int)) != cudaSuccess) {
      host = nullptr;
      cudaGetLastError();
      return set_error(NNPP_ERR_NOMEM, "implicit step: pinned status");
    }
    for (cudaEvent_t& e : ev) NNPP_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return NNPP_OK;
  }
  nnpp_status record(cudaStream_t st, int k, const int* word) {
    NNPP_CUDA(cudaMemcpyAsync(host + k % kSlots, word, sizeof(int), cudaMemcpyDeviceToHost, st));
    NNPP_CUDA(cudaEventRecord(ev[k % kSlots], st));
    return NNPP_OK;
  }
  nnpp_status wait(int k, int* word) {
    NNPP_CUDA(cudaEventSynchronize(ev[k % kSlots]));
    *word = *(volatile int*)(host + k % kSlots);
    return NNPP_OK;
  }
};

// The rows in slices of 32: offsets, columns, weights and the step's off-diagonals of every field.
struct Sliced {
  int n = 0;
  long long slots = 0;
  DBuf<int> off, col;
  DBuf<double> w, toff;
};
struct Work {
  int N = 0;
  DBuf<double> u0, u1, F, b, x, t, diag, V, part, red;
  Sliced sl;
  GmStatus status;
  DBuf<GmState> gm;
  DBuf<unsigned char> dir;
  DBuf<double> bc;
  DBuf<int> phase;
};

int grid_for(long long items, int per_block) {
  long long g = (items + per_block - 1) / per_block;
  return (int)std::max<long long>(1, std::min<long long>(g, 152 * 16));
}

// Slices below which four warps share a slice: with a warp each they fill half of the 152 SMs'
// 48 warps.  Measured, one field: 64k nodes (2,000 slices) 16.7 ms a four-species step split
// against 21.2 whole, 123 a ten-species step against 175; 8k nodes 4.81 against 7.05 and 17.2
// against 33.3; 176k (5,500 slices, above the line) 42.8 either way.
constexpr int kSplitSlices = 152 * 24;

template <int NA, int NS>
void apply_na(cudaStream_t st, const ImpCtxT<NS>& c, const double* v, double* out, const FieldList& fl,
              const double* scale) {
  constexpr int kStride = sizeof(GmField) / sizeof(double);
  auto go = [&](auto kern, int per) {
    const int grid = std::max(1, std::min((c.nslices + per - 1) / per, 152 * 64));
    kern<<<grid, 128, 0, st>>>(c.N, c.ptr, c.nslices, c.soff, c.scol, c.toff, c.slots, c.dinv, c.dir, v, out, fl, scale,
                                 kStride);
  };
  if (c.nslices < kSplitSlices)
    go(k_imp_apply<NA, 4>, 1);
  else
    go(k_imp_apply<NA, 1>, 4);
}

int fields_of(int mask, int nf, FieldList* fl) {
  int na = 0;
  for (int f = 0; f < nf; ++f)
    if ((mask >> f) & 1) fl->f[na++] = f;
  return na;
}

// the products of na fields
template <int NS>
nnpp_status apply(cudaStream_t st, const ImpCtxT<NS>& c, const double* v, double* out, const FieldList& fl, int na,
                  const double* scale) {
  switch (na) {
    case 0: return NNPP_OK;
    case 1: apply_na<1>(st, c, v, out, fl, scale); break;
    case 2: apply_na<2>(st, c, v, out, fl, scale); break;
    case 3: apply_na<3>(st, c, v, out, fl, scale); break;
    case 4: apply_na<4>(st, c, v, out, fl, scale); break;
    case 5: apply_na<5>(st, c, v, out, fl, scale); break;
    case 6: apply_na<6>(st, c, v, out, fl, scale); break;
    case 7: apply_na<7>(st, c, v, out, fl, scale); break;
    case 8: apply_na<8>(st, c, v, out, fl, scale); break;
    case 9: apply_na<9>(st, c, v, out, fl, scale); break;
    case 10: apply_na<10>(st, c, v, out, fl, scale); break;
    default: apply_na<11>(st, c, v, out, fl, scale);
  }
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// build_slices: asynchronous on st but for one read of the slot count
nnpp_status build_slices(cudaStream_t st, int N, const int* ptr, const int* col, const double* x, const double* y,
                         const double* z, double delta, double dx, double dV, Sliced& sl) {
  sl.n = (N + 31) / 32;
  DBuf<int> width;
  if (!width.alloc(sl.n) || !sl.off.alloc(sl.n + 1)) return set_error(NNPP_ERR_NOMEM, "implicit step: slices");
  k_imp_widths<<<grid_for((long long)sl.n * 32, kTB), kTB, 0, st>>>(N, ptr, sl.n, width.get());
  NNPP_CUDA(cudaGetLastError());
  long long cols = 0;
  NNPP_TRY(scan_ints(st, width.get(), sl.off.get(), sl.n, &cols));
  sl.slots = 32 * std::max<long long>(cols, 1);
  if (!sl.col.alloc(sl.slots) || !sl.w.alloc(sl.slots))
    return set_error(NNPP_ERR_NOMEM, "implicit step: slices");
  k_imp_weights<<<grid_for((long long)sl.n * 32, kTB), kTB, 0, st>>>(N, ptr, col, x, y, z, delta, dx, dV, sl.n,
                                                                     sl.off.get(), sl.col.get(), sl.w.get());
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// the arrays that only a step needs, the largest: the Arnoldi basis and the off-diagonals of nf fields
nnpp_status alloc_step(Work& wk, int nf) {
  if (!wk.V.alloc((size_t)(kRestart + 1) * nf * wk.N) || !wk.sl.toff.alloc((size_t)nf * wk.sl.slots))
    return set_error(NNPP_ERR_NOMEM, "implicit step: Arnoldi basis and off-diagonals");
  return NNPP_OK;
}

// Blocks of a product over N values when a launch forms `products` of them: 8 to 32 values a thread
// (a block's reduction costs as much FP64 as 8 values), the more the more products fill the chip.
int dot_blocks(int N, int products) {
  const int per = products >= 64 ? 32 : products >= 16 ? 16 : 8;
  return std::max(1, std::min(kDotBlocks, (N + kTB * per - 1) / (kTB * per)));
}

// NS + 1 independent GMRES solves K_f x_f = b_f (wk.b -> wk.x), as Eigen's; iterations summed.  The
// host launches iteration j while iteration j - kAhead may still run: it then knows which
// fields had finished by then, and leaves the others to the kernels' own test.
constexpr int kAhead = 2;
template <int NS>
nnpp_status gmres_fields(cudaStream_t st, const ImpCtxT<NS>& c, Work& wk, long long* iters_total) {
  constexpr int NF = NS + 1;
  const int N = wk.N;
  const size_t FN = (size_t)NF * N;
  double* V = wk.V.get();
  GmState* gs = wk.gm.get();
  double* part = wk.part.get();
  const int nb = dot_blocks(N, 1);
  // the combinations': one value a thread up to the partials' width
  const int nc = std::max(1, std::min((N + kTB - 1) / kTB, kDotBlocks));
  NNPP_TRY(wk.status.init());
  // x = b (GMRES.h:330-334); b = 0 gives x = 0
  NNPP_CUDA(cudaMemcpyAsync(wk.x.get(), wk.b.get(), sizeof(double) * FN, cudaMemcpyDeviceToDevice, st));
  int active = (1 << NF) - 1;
  bool first = true;
  while (active) {
    FieldList fl;
    int na = fields_of(active, NF, &fl);
    NNPP_TRY(apply(st, c, wk.x.get(), wk.t.get(), fl, na, nullptr));
    k_gm_start<<<dim3(nb, na), kTB, 0, st>>>(N, first ? 1 : 0, fl, wk.b.get(), c.dinv, wk.t.get(), V, gs, part);
    NNPP_CUDA(cudaGetLastError());
    const FieldList all = fl;
    const int nall = na;
    first = false;
    int k = 1;
    for (; k <= kRestart; ++k) {
      if (k > kAhead) {
        int cycle = 0;
        NNPP_TRY(wk.status.wait(k - kAhead, &cycle));
        if (!cycle) break;
        na = fields_of(cycle, NF, &fl);
      }
      NNPP_TRY(apply(st, c, V + (size_t)(k - 1) * FN, V + (size_t)k * FN, fl, na, &gs->f[0].s[k - 1]));
      const int nd = dot_blocks(N, k * na);
      k_gm_dots<<<dim3(nd, k, na), kTB, 0, st>>>(N, k, 0, fl, NF, V, gs, part);
      k_gm_combine<false><<<dim3(nc, na), kTB, 0, st>>>(N, k, fl, NF, V, gs, part);
      k_gm_dots<<<dim3(nd, k, na), kTB, 0, st>>>(N, k, 1, fl, NF, V, gs, part);
      k_gm_combine<true><<<dim3(nc, na), kTB, 0, st>>>(N, k, fl, NF, V, gs, part);
      NNPP_CUDA(cudaGetLastError());
      NNPP_TRY(wk.status.record(st, k, &gs->cycle));
    }
    k_gm_solution<<<dim3(nc, nall), kTB, 0, st>>>(N, all, NF, V, gs, wk.x.get());
    NNPP_CUDA(cudaGetLastError());
    // the fields that go on: those at their restart
    NNPP_TRY(wk.status.record(st, 0, &gs->restart));
    NNPP_CUDA(cudaMemsetAsync(&gs->restart, 0, sizeof(int), st));
    NNPP_TRY(wk.status.wait(0, &active));
  }
  for (int f = 0; f < NF; ++f)
    NNPP_CUDA(cudaMemcpyAsync(wk.status.host + 8 + f, &gs->f[f].it, sizeof(int), cudaMemcpyDeviceToHost, st));
  NNPP_CUDA(cudaStreamSynchronize(st));
  for (int f = 0; f < NF; ++f) *iters_total += wk.status.host[8 + f];
  return NNPP_OK;
}

// ||x_f||^2 of every field to the host
template <int NF>
nnpp_status norms(cudaStream_t st, Work& wk, double* h) {
  k_imp_norms<<<dim3(dot_blocks(wk.N, 1), NF), kTB, 0, st>>>(wk.N, wk.x.get(), wk.gm.get(), wk.part.get(), wk.red.get());
  NNPP_CUDA(cudaGetLastError());
  NNPP_CUDA(cudaMemcpyAsync(h, wk.red.get(), sizeof(double) * NF, cudaMemcpyDeviceToHost, st));
  NNPP_CUDA(cudaStreamSynchronize(st));
  return NNPP_OK;
}

// F = U - bc on the Dirichlet rows of every field (main.cpp:676-712)
template <int NF>
__global__ void k_imp_dirichlet(int N, const double* u1, const double* bc, const unsigned char* dir, double* F) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
    for (int f = 0; f < NF; ++f) {
      const size_t q = (size_t)f * N + i;
      if (dir[q]) F[q] = u1[q] - bc[q];
    }
}

__global__ void k_imp_negate(size_t n, const double* a, double* b) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = -a[i];
}

}  // namespace

// Bytes of a step's arrays (alloc_step) up to which nnpp_forward_implicit leaves them with the handle for
// its next call; larger ones (from some 85,000 nodes on; 3 GB at 512,000) are freed on return, since other
// runs and handles need the memory, and allocating them again is little of a step that long: 125k nodes
// 30.2 ms a call of one step against 29.5 with the arrays kept, 512k 136.0 against 134.1.
constexpr size_t kKeepStepBytes = (size_t)512 << 20;

// the four-species step's buffers
static nnpp_status make_work(Handle& h, Work& wk) {
  const nnpp_params& p = h.p;
  const int N = h.N;
  const size_t FN = (size_t)F5 * N;
  cudaStream_t st = h.st;
  wk.N = N;
  if (!wk.u0.alloc(FN) || !wk.u1.alloc(FN) || !wk.F.alloc(FN) ||
      !wk.b.alloc(FN) || !wk.x.alloc(FN) || !wk.t.alloc(FN) || !wk.diag.alloc(FN) ||
      !wk.part.alloc((size_t)kDotBlocks * (kRestart + 1) * F5) ||
      !wk.red.alloc(F5) || !wk.gm.alloc(1) || !wk.dir.alloc(FN) || !wk.bc.alloc(FN) || !wk.phase.alloc(N))
    return set_error(NNPP_ERR_NOMEM, "forward_implicit buffers");
  NNPP_CUDA(cudaMemsetAsync(wk.gm.get(), 0, sizeof(GmState), st));
  NNPP_TRY(build_slices(st, N, h.ref.ptr.get(), h.ref.col.get(), h.ux.get(), h.uy.get(), h.uz.get(), p.delta, p.dx,
                        p.dx * p.dy * p.dz, wk.sl));
  // Dirichlet flags and values in the reference's order (main.cpp:676-712)
  std::vector<unsigned char> dir(FN, 0);
  std::vector<double> bc(FN, 0.0);
  for (int f = 0; f <= S; ++f)
    for (int i = 0; i < N; ++i) {
      const double v = h.h_bcv[(size_t)f * N + i];
      if (h.h_bctypes[i] == 0 && v != -1) {
        dir[(size_t)f * N + i] = 1;
        bc[(size_t)f * N + i] = f < S ? v / p.CSolid : v;
      }
    }
  NNPP_CUDA(cudaMemcpyAsync(wk.dir.get(), dir.data(), FN, cudaMemcpyHostToDevice, st));
  NNPP_CUDA(cudaMemcpyAsync(wk.bc.get(), bc.data(), sizeof(double) * FN, cudaMemcpyHostToDevice, st));
  NNPP_CUDA(cudaStreamSynchronize(st));  // the sources are local
  return NNPP_OK;
}

extern "C" nnpp_status nnpp_forward_implicit(nnpp_handle* hp, int n_steps, int64_t* newton_iterations,
                                             int64_t* krylov_iterations) {
  nnpp::TraceRange trace_("nnpp_forward_implicit");
  clear_error();
  if (!hp) return set_error(NNPP_ERR_INVALID, "handle is NULL");
  Handle& h = hp->h;
  if (!h.built) return set_error(NNPP_ERR_STATE, "neighbour lists not built (call nnpp_build_neighbours)");
  if (n_steps < 0) return set_error(NNPP_ERR_INVALID, "forward_implicit: negative step count");
  NNPP_CUDA(cudaSetDevice(h.device));
  const nnpp_params& p = h.p;
  if (p.s_phi != 0.0) return set_error(NNPP_ERR_UNSUPPORTED, "forward_implicit: kernel exponent s must be 0");
  const int N = h.N;
  const size_t FN = (size_t)F5 * N;
  cudaStream_t st = h.st;
  // vectors, sliced rows with their weights and Dirichlet values (the reference's node order): made by
  // the first call, kept by the handle until its lists are rebuilt; a step's arrays as kKeepStepBytes says
  if (!h.implicit_work) {
    auto made = std::make_shared<Work>();
    NNPP_TRY(make_work(h, *made));
    h.implicit_work = made;
  }
  Work& wk = *std::static_pointer_cast<Work>(h.implicit_work);
  struct StepArrays {
    Work& wk;
    ~StepArrays() {
      if (wk.V.bytes() + wk.sl.toff.bytes() <= kKeepStepBytes) return;
      wk.V.reset();
      wk.sl.toff.reset();
    }
  } step_arrays{wk};
  NNPP_TRY(alloc_step(wk, F5));
  // the handle's state (FP64, user order)
  NNPP_TRY(store_state(h, wk.u0.get(), wk.u0.get() + (size_t)S * N, wk.phase.get()));
  DevState ds;
  NNPP_CUDA(cudaMemcpyAsync(&ds, h.dstate.get(), sizeof(DevState), cudaMemcpyDeviceToHost, st));
  NNPP_CUDA(cudaStreamSynchronize(st));
  ImpCtx c;
  std::memset(&c, 0, sizeof(c));
  c.N = N;
  c.ptr = h.ref.ptr.get();
  c.nslices = wk.sl.n;
  c.soff = wk.sl.off.get();
  c.scol = wk.sl.col.get();
  c.sw = wk.sl.w.get();
  c.slots = wk.sl.slots;
  c.dir = wk.dir.get();
  c.bc = wk.bc.get();
  c.phase = wk.phase.get();
  c.u0 = wk.u0.get();
  c.dinv = wk.diag.get();
  c.toff = wk.sl.toff.get();
  c.dt = p.dt;
  c.csat = p.CSat / p.CSolid;
  c.k_diss = p.k_diss;
  c.sw_width = p.switch_width;
  c.kphis = p.K_phi * p.sigma;
  c.lam = (1. / (p.K_phi * p.sigma)) * p.F * p.CSolid;
  double K2zF[S];
  for (int k = 0; k < S; ++k) {
    K2zF[k] = p.K2[k] * p.z[k] * p.F / (p.R * p.T);
    c.z[k] = p.z[k];
  }
  double voln1rel = ds.voln1rel;
  long long steps_done = ds.steps;
  long long newton_total = 0, krylov_total = 0;
  std::vector<double> res(F5), res_old(F5), part(kDotBlocks);
  for (int s = 0; s < n_steps; ++s) {
    set_coefficients(c, p.K1, K2zF, p.D_liquid, p.D_solid, std::pow(10., -p.vol_red * (1. - voln1rel)));  // utils.h:100-116
    // the tangents at U^n (main.cpp:657-662), U^{n+1} = U^n to start
    k_imp_diag<S><<<grid_for((long long)c.nslices * 32, 128), 128, 0, st>>>(c, wk.diag.get());
    k_imp_tangent<S><<<grid_for((long long)c.nslices * 32, 128), 128, 0, st>>>(c, wk.sl.toff.get());
    NNPP_CUDA(cudaMemcpyAsync(wk.u1.get(), wk.u0.get(), sizeof(double) * FN, cudaMemcpyDeviceToDevice, st));
    std::fill(res_old.begin(), res_old.end(), 0.0);
    int it = 0;
    for (it = 0; it < kMaxIter; ++it) {
      if (c.nslices < kSplitSlices)
        k_imp_residual<4><<<std::min(c.nslices, 152 * 64), 128, 0, st>>>(c, wk.u1.get(), wk.F.get());
      else
        k_imp_residual<1><<<std::min((c.nslices + 3) / 4, 152 * 64), 128, 0, st>>>(c, wk.u1.get(), wk.F.get());
      k_imp_negate<<<grid_for((long long)FN, kTB), kTB, 0, st>>>(FN, wk.F.get(), wk.b.get());
      NNPP_CUDA(cudaGetLastError());
      NNPP_TRY(gmres_fields<S>(st, c, wk, &krylov_total));
      NNPP_TRY(norms<F5>(st, wk, res.data()));
      k_imp_update<S><<<grid_for(N, kTB), kTB, 0, st>>>(N, wk.u1.get(), wk.x.get(), 1.0e-8 / p.CSolid, wk.phase.get());
      NNPP_CUDA(cudaGetLastError());
      double resMax = 0.0;
      for (int f = 0; f < F5; ++f) {
        res[f] = std::sqrt(res[f]);
        resMax = std::max(resMax, std::abs(res[f] - res_old[f]));
      }
      if (!std::isfinite(resMax)) return set_error(NNPP_ERR_NONFINITE, "forward_implicit: non-finite update");
      if (resMax < kEps) {
        ++it;
        break;
      }
      res_old = res;
    }
    newton_total += it;
    // flip, volume (main.cpp:914-922, 944-949)
    steps_done += 1;
    k_imp_flip<<<kDotBlocks, kTB, 0, st>>>(N, wk.u1.get(), wk.phase.get(), c.csat, (int)steps_done,
                                           h.lay.iperm.get(), h.flip_step.get(), wk.part.get());
    NNPP_CUDA(cudaGetLastError());
    NNPP_CUDA(cudaMemcpyAsync(part.data(), wk.part.get(), sizeof(double) * kDotBlocks, cudaMemcpyDeviceToHost, st));
    NNPP_CUDA(cudaStreamSynchronize(st));
    if (p.sub_step_no > 0 && steps_done % p.sub_step_no == 0) {
      double v = 0.0;
      for (double x : part) v += x;
      voln1rel = ds.vol0rel != 0.0 ? v / ds.vol0rel : 0.0;
    }
    // time-level swap (main.cpp:1002-1024)
    NNPP_CUDA(cudaMemcpyAsync(wk.u0.get(), wk.u1.get(), sizeof(double) * FN, cudaMemcpyDeviceToDevice, st));
  }
  // the result into the handle's state (FP64), its diagnostics and step count
  NNPP_TRY(load_state(h, wk.u0.get(), wk.u0.get() + (size_t)S * N, wk.phase.get(), NNPP_FP64, true));
  NNPP_TRY(init_diag(h, true));
  DevState d2;
  NNPP_CUDA(cudaMemcpyAsync(&d2, h.dstate.get(), sizeof(DevState), cudaMemcpyDeviceToHost, st));
  NNPP_CUDA(cudaStreamSynchronize(st));
  d2.steps = steps_done;
  d2.voln1rel = voln1rel;
  d2.BV = std::pow(10., -p.vol_red * (1. - voln1rel));
  NNPP_CUDA(cudaMemcpyAsync(h.dstate.get(), &d2, sizeof(DevState), cudaMemcpyHostToDevice, st));
  NNPP_CUDA(cudaStreamSynchronize(st));
  h.coarse.stale = true;
  h.nstep = 0;
  if (newton_iterations) *newton_iterations = newton_total;
  if (krylov_iterations) *krylov_iterations = krylov_total;
  return NNPP_OK;
}

// ---------------------------------------------------------------- the complete model -----
// The reference's time step with all eleven fields (main.cpp:640-922 as written: ten species
// and the potential).  The tangents of utils::NewtonMatrices (utils.h:846-1849) at U^n,
// applied matrix-free like the four-species step's (eleven fields in one pass over the bonds;
// the species' own constants, the linearised reaction terms on the diagonals), the residual
// of utils::Residuals (utils.h:29-842: nnpp_residuals_full_device) with the Dirichlet rows of
// main.cpp:676-712, eleven GMRES corrections advanced together, the clamp of
// main.cpp:805-837 (U10 on liquid nodes only), the update-norm test, the flip of
// main.cpp:914-922 and the relative volume every sub_step_no steps (main.cpp:944-949).
struct nnpp_chem {
  int N = 0, ml = 0, device = 0;
  long long nnz = 0;
  cudaStream_t st = nullptr;
  DBuf<double> xyz;
  DBuf<int> ptr, hz, hl;
  Work wk;
  std::vector<double> d2, dc, d11;
  double voln1rel = 0.0, vol0rel = 0.0;
  long long steps = 0;
  bool has_state = false;
  ~nnpp_chem() {
    if (st) cudaStreamDestroy(st);
  }
};

namespace {
constexpr int kChemNS = 10;
constexpr int kChemNF = 11;
constexpr int kChemSubSteps = 8;  // sub_step_no, main.cpp:39
}  // namespace

extern "C" nnpp_status nnpp_chem_create(nnpp_chem** out, int n_nodes, const double* nodes_colmajor,
                                        const int* clouds_colmajor, int max_node_no, const int* cloud_lengths,
                                        const int* bctypes, const double* bcvalues, const double* data2,
                                        const double* datac, const double* datac11) {
  clear_error();
  if (!out) return set_error(NNPP_ERR_INVALID, "chem_create: out is NULL");
  *out = nullptr;
  if (n_nodes <= 0 || max_node_no < 1 || !nodes_colmajor || !clouds_colmajor || !cloud_lengths || !bctypes ||
      !bcvalues || !data2 || !datac || !datac11)
    return set_error(NNPP_ERR_INVALID, "chem_create: bad argument");
  for (int k = 0; k < kChemNS; ++k)
    if (datac[7 * k + 3] != 0.0 || datac[7 * k + 4] != 0.0)
      return set_error(NNPP_ERR_UNSUPPORTED, "chem_create: the bond weights need the kernel exponents s = 0");
  if (datac11[2] != 0.0) return set_error(NNPP_ERR_UNSUPPORTED, "chem_create: the potential's exponent s must be 0");
  if (!(data2[2] != 0.0) || !(data2[3] > 0.0) || !(data2[7] > 0.0) || !(datac11[1] * datac11[3] != 0.0))
    return set_error(NNPP_ERR_INVALID, "chem_create: dt, dx, CSolid or K11prop1 sigma1 is zero");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return set_error(NNPP_ERR_CUDA, "chem_create: no CUDA device");
  }
  const int N = n_nodes;
  int ml = 1;
  long long nnz = 0;
  for (int i = 0; i < N; ++i) {
    const int l = cloud_lengths[i];
    if (l < 1 || l > max_node_no) return set_error(NNPP_ERR_INVALID, "chem_create: cloud length out of range");
    ml = std::max(ml, l);
    nnz += l - 1;
  }
  if (nnz > 0x7fffffffLL) return set_error(NNPP_ERR_UNSUPPORTED, "chem_create: more than 2^31 bonds");
  // CSR without the node itself (the tangents) and the padded clouds (the residual)
  std::vector<int> ptr(N + 1), col(std::max<long long>(nnz, 1));
  ptr[0] = 0;
  for (int i = 0; i < N; ++i) {
    int q = ptr[i];
    for (int j = 1; j < cloud_lengths[i]; ++j) {
      const int n = clouds_colmajor[(size_t)j * N + i];
      if (n < 0 || n >= N) return set_error(NNPP_ERR_INVALID, "chem_create: cloud index out of range");
      col[q++] = n;
    }
    ptr[i + 1] = q;
  }
  nnpp_chem* c = new nnpp_chem();
  c->N = N;
  c->ml = ml;
  c->nnz = nnz;
  cudaGetDevice(&c->device);
  c->d2.assign(data2, data2 + 51);
  c->dc.assign(datac, datac + 70);
  c->d11.assign(datac11, datac11 + 4);
  const size_t FN = (size_t)kChemNF * N;
  Work& wk = c->wk;
  wk.N = N;
  bool ok = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) == cudaSuccess;
  DBuf<int> dcol;
  ok = ok && c->xyz.alloc(3 * (size_t)N) && c->ptr.alloc(N + 1) &&
       dcol.alloc(col.size()) && c->hz.alloc((size_t)ml * N) && c->hl.alloc(N) && wk.u0.alloc(FN) &&
       wk.u1.alloc(FN) && wk.F.alloc(FN) && wk.b.alloc(FN) && wk.x.alloc(FN) && wk.t.alloc(FN) &&
       wk.diag.alloc(FN) &&
       wk.part.alloc((size_t)kDotBlocks * (kRestart + 1) * kChemNF) && wk.red.alloc(kChemNF) && wk.gm.alloc(1) &&
       wk.dir.alloc(FN) && wk.bc.alloc(FN) && wk.phase.alloc(N);
  if (!ok) {
    cudaGetLastError();
    delete c;
    return set_error(NNPP_ERR_NOMEM, "chem_create buffers");
  }
  cudaStream_t st = c->st;
  std::vector<unsigned char> dir(FN, 0);
  std::vector<double> bc(FN, 0.0);
  const double CSolid = data2[7];
  for (int f = 0; f < kChemNF; ++f)
    for (int i = 0; i < N; ++i) {
      const double v = bcvalues[(size_t)f * N + i];
      if (bctypes[i] == 0 && v != -1) {
        dir[(size_t)f * N + i] = 1;
        bc[(size_t)f * N + i] = f < kChemNS ? v / CSolid : v;
      }
    }
  nnpp_status rs = NNPP_OK;
  auto cp = [&](void* d, const void* h, size_t bytes) {
    if (rs == NNPP_OK && cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
      rs = set_error(NNPP_ERR_CUDA, "chem_create: copy");
  };
  cp(c->xyz.get(), nodes_colmajor, sizeof(double) * 3 * N);
  cp(c->ptr.get(), ptr.data(), sizeof(int) * (N + 1));
  cp(dcol.get(), col.data(), sizeof(int) * col.size());
  cp(c->hz.get(), clouds_colmajor, sizeof(int) * (size_t)ml * N);
  cp(c->hl.get(), cloud_lengths, sizeof(int) * N);
  cp(wk.dir.get(), dir.data(), FN);
  cp(wk.bc.get(), bc.data(), sizeof(double) * FN);
  if (rs == NNPP_OK && cudaMemsetAsync(wk.gm.get(), 0, sizeof(GmState), st) != cudaSuccess)
    rs = set_error(NNPP_ERR_CUDA, "chem_create: memset");
  if (rs == NNPP_OK) {
    const double dx = data2[3], dy = data2[4], dz = data2[5], delta = data2[6];
    rs = build_slices(st, N, c->ptr.get(), dcol.get(), c->xyz.get(), c->xyz.get() + N, c->xyz.get() + 2 * (size_t)N,
                      delta, dx, dx * dy * dz, wk.sl);
    if (rs == NNPP_OK) rs = alloc_step(wk, kChemNF);
    if (rs == NNPP_OK && cudaStreamSynchronize(st) != cudaSuccess) rs = set_error(NNPP_ERR_CUDA, "chem_create: weights");
  }
  if (rs != NNPP_OK) {
    delete c;
    return rs;
  }
  *out = c;
  return NNPP_OK;
}

extern "C" void nnpp_chem_destroy(nnpp_chem* c) { delete c; }

extern "C" nnpp_status nnpp_chem_set_state(nnpp_chem* c, const double* U, const int* phase, double voln1rel,
                                           double vol0rel) {
  clear_error();
  if (!c || !U || !phase) return set_error(NNPP_ERR_INVALID, "chem_set_state: NULL argument");
  const int N = c->N;
  NNPP_CUDA(cudaSetDevice(c->device));
  for (int i = 0; i < N; ++i)
    if (phase[i] != 0 && phase[i] != 1) return set_error(NNPP_ERR_INVALID, "chem_set_state: phase must be 0 or 1");
  if (!(vol0rel > 0.0)) {
    // the initial volume (main.cpp:472-480): the solid nodes' Mg above saturation
    const double csat = c->d2[8] / c->d2[7];
    double v = 0.0;
    for (int i = 0; i < N; ++i)
      if (phase[i] == 1) v += U[i] - csat;
    vol0rel = v;
  }
  NNPP_CUDA(cudaMemcpyAsync(c->wk.u0.get(), U, sizeof(double) * kChemNF * N, cudaMemcpyHostToDevice, c->st));
  NNPP_CUDA(cudaMemcpyAsync(c->wk.phase.get(), phase, sizeof(int) * N, cudaMemcpyHostToDevice, c->st));
  NNPP_CUDA(cudaStreamSynchronize(c->st));
  c->voln1rel = voln1rel;
  c->vol0rel = vol0rel;
  c->steps = 0;
  c->has_state = true;
  return NNPP_OK;
}

extern "C" nnpp_status nnpp_chem_get_state(nnpp_chem* c, double* U, int* phase, double* voln1rel) {
  clear_error();
  if (!c) return set_error(NNPP_ERR_INVALID, "chem_get_state: NULL handle");
  if (!c->has_state) return set_error(NNPP_ERR_STATE, "chem_get_state: no state (call nnpp_chem_set_state)");
  NNPP_CUDA(cudaSetDevice(c->device));
  const int N = c->N;
  if (U) NNPP_CUDA(cudaMemcpyAsync(U, c->wk.u0.get(), sizeof(double) * kChemNF * N, cudaMemcpyDeviceToHost, c->st));
  if (phase) NNPP_CUDA(cudaMemcpyAsync(phase, c->wk.phase.get(), sizeof(int) * N, cudaMemcpyDeviceToHost, c->st));
  NNPP_CUDA(cudaStreamSynchronize(c->st));
  if (voln1rel) *voln1rel = c->voln1rel;
  return NNPP_OK;
}

extern "C" nnpp_status nnpp_chem_step(nnpp_chem* c, int n_steps, int64_t* newton_iterations,
                                      int64_t* krylov_iterations) {
  nnpp::TraceRange trace_("nnpp_chem_step");
  clear_error();
  if (!c) return set_error(NNPP_ERR_INVALID, "chem_step: NULL handle");
  if (n_steps < 0) return set_error(NNPP_ERR_INVALID, "chem_step: negative step count");
  if (!c->has_state) return set_error(NNPP_ERR_STATE, "chem_step: no state (call nnpp_chem_set_state)");
  NNPP_CUDA(cudaSetDevice(c->device));
  const int N = c->N;
  const size_t FN = (size_t)kChemNF * N;
  const std::vector<double>& d2 = c->d2;
  const std::vector<double>& dc = c->dc;
  Work& wk = c->wk;
  cudaStream_t st = c->st;
  const double CSolid = d2[7], CSat = d2[8], T = d2[47], R = d2[48], Fc = d2[49], vol_red = d2[50];
  ImpCtxT<kChemNS> x;
  std::memset(&x, 0, sizeof(x));
  x.N = N;
  x.ptr = c->ptr.get();
  x.nslices = wk.sl.n;
  x.soff = wk.sl.off.get();
  x.scol = wk.sl.col.get();
  x.sw = wk.sl.w.get();
  x.slots = wk.sl.slots;
  x.dir = wk.dir.get();
  x.bc = wk.bc.get();
  x.phase = wk.phase.get();
  x.u0 = wk.u0.get();
  x.dinv = wk.diag.get();
  x.toff = wk.sl.toff.get();
  x.dt = d2[2];
  x.csat = CSat / CSolid;
  x.k7b = d2[41];
  x.k8b = d2[43];
  x.k9b = d2[45];
  double K1[kChemNS], K2zF[kChemNS], DL[kChemNS], DSo[kChemNS];
  for (int k = 0; k < kChemNS; ++k) {
    x.z[k] = dc[7 * k];
    DSo[k] = dc[7 * k + 1];
    DL[k] = dc[7 * k + 2];
    K1[k] = dc[7 * k + 5];
    K2zF[k] = dc[7 * k + 6] * dc[7 * k] * Fc / (R * T);
  }
  long long newton_total = 0, krylov_total = 0;
  std::vector<double> res(kChemNF), res_old(kChemNF), part(kDotBlocks);
  for (int s = 0; s < n_steps; ++s) {
    set_coefficients(x, K1, K2zF, DL, DSo, std::pow(10., -vol_red * (1. - c->voln1rel)));  // utils.h:100-116
    k_imp_diag<kChemNS><<<grid_for((long long)x.nslices * 32, 128), 128, 0, st>>>(x, wk.diag.get());
    k_imp_tangent<kChemNS><<<grid_for((long long)x.nslices * 32, 128), 128, 0, st>>>(x, wk.sl.toff.get());
    NNPP_CUDA(cudaMemcpyAsync(wk.u1.get(), wk.u0.get(), sizeof(double) * FN, cudaMemcpyDeviceToDevice, st));
    std::fill(res_old.begin(), res_old.end(), 0.0);
    int it = 0;
    for (it = 0; it < kMaxIter; ++it) {
      NNPP_TRY(nnpp_residuals_full_device(N, c->xyz.get(), c->hz.get(), c->hl.get(), wk.u1.get(), wk.u0.get(),
                                          wk.phase.get(), c->voln1rel, d2.data(), dc.data(), c->d11.data(),
                                          wk.F.get(), st));
      k_imp_dirichlet<kChemNF><<<grid_for(N, kTB), kTB, 0, st>>>(N, wk.u1.get(), wk.bc.get(), wk.dir.get(), wk.F.get());
      k_imp_negate<<<grid_for((long long)FN, kTB), kTB, 0, st>>>(FN, wk.F.get(), wk.b.get());
      NNPP_CUDA(cudaGetLastError());
      NNPP_TRY(gmres_fields<kChemNS>(st, x, wk, &krylov_total));
      NNPP_TRY(norms<kChemNF>(st, wk, res.data()));
      k_imp_update<kChemNS><<<grid_for(N, kTB), kTB, 0, st>>>(N, wk.u1.get(), wk.x.get(), 1.0e-8 / CSolid,
                                                             wk.phase.get());
      NNPP_CUDA(cudaGetLastError());
      double resMax = 0.0;
      for (int f = 0; f < kChemNF; ++f) {
        res[f] = std::sqrt(res[f]);
        resMax = std::max(resMax, std::abs(res[f] - res_old[f]));
      }
      if (!std::isfinite(resMax)) return set_error(NNPP_ERR_NONFINITE, "chem_step: non-finite update");
      if (resMax < kEps) {
        ++it;
        break;
      }
      res_old = res;
    }
    newton_total += it;
    c->steps += 1;
    k_imp_flip<<<kDotBlocks, kTB, 0, st>>>(N, wk.u1.get(), wk.phase.get(), x.csat, (int)c->steps, nullptr, nullptr,
                                           wk.part.get());
    NNPP_CUDA(cudaGetLastError());
    NNPP_CUDA(cudaMemcpyAsync(part.data(), wk.part.get(), sizeof(double) * kDotBlocks, cudaMemcpyDeviceToHost, st));
    NNPP_CUDA(cudaStreamSynchronize(st));
    if (c->steps % kChemSubSteps == 0) {
      double v = 0.0;
      for (double q : part) v += q;
      c->voln1rel = c->vol0rel != 0.0 ? v / c->vol0rel : 0.0;
    }
    NNPP_CUDA(cudaMemcpyAsync(wk.u0.get(), wk.u1.get(), sizeof(double) * FN, cudaMemcpyDeviceToDevice, st));
  }
  NNPP_CUDA(cudaStreamSynchronize(st));
  if (newton_iterations) *newton_iterations = newton_total;
  if (krylov_iterations) *krylov_iterations = krylov_total;
  return NNPP_OK;
}
