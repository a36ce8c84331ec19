// step.cu -- the explicit NNPP step on the GPU for one or many instances: potential solve
// (K11, utils.h:1794-1848 / F11, utils.h:798-841) and transport (bond sums utils.h:72-257,
// Dirichlet main.cpp:676-712, clamp main.cpp:805-837, phase flip main.cpp:914-922, volume
// main.cpp:944-949).
//
// Work is a list of slices of 32 rows (bond kernels), node chunks (vector kernels) or tiles (the
// residual entry and the FP64 adjoint) over all instances of a batch; each CTA loops over the list
// (persistent grid).  A slice streams its rows' bonds in quads of columns, weights and 16-bit codes;
// a tile kernel stages the tile's halo into shared memory and reaches every neighbour through a
// 16-bit slot.
//
// Precision:
//   FP64  : FP64 records and stored FP64 weights, FP64 CG.
//   mixed : transport in FP32 with stored FP32 weights (computed in FP64);
//           concentrations kept as compensated FP32 pairs (hi + lo), the saturation test on
//           hi + lo in FP64; potential: residual b - A phi in FP32 pairs (the FP64 weights as
//           pairs) into FP64, with FP32 CG corrections.
//
// Reductions: every work item writes one partial per value; the CTA that completes an
// instance's last item reduces that instance's partials in item order (deterministic), and
// the last instance to finish sets the graph's loop condition (any instance still active).  The
// one-launch inner solve (k_cg_sweep) instead has every CTA sum the CTAs' parts.
#include <cmath>
#include <cstring>

#include "engine.cuh"
#include "fp64_steps.cuh"
#include "tma.cuh"

namespace nnpp {

namespace {

constexpr int kBlock = 256;

// ---------------------------------------------------------------- work-item plumbing ----
struct TileSmem {
  int off[10];  // prefix offsets of the 9 halo rows, off[9] = halo size
  int hb[9];
  int flag;
};

__device__ __forceinline__ void load_tile(const TileDesc& t, TileSmem& ts) {
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int r = 0; r < 9; ++r) {
      ts.off[r] = acc;
      ts.hb[r] = t.hb[r];
      acc += t.hl[r];
    }
    ts.off[9] = acc;
  }
  __syncthreads();
}

__host__ __device__ __forceinline__ size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

// Copy the tile's bond slots [bond0, bond1) into shared memory with 16-byte loads (bond0 is
// a multiple of 8, the slot array is padded); bond j is then at dst[j - bond0].
__device__ __forceinline__ const unsigned short* stage_slots(const unsigned short* slot16,
                                                             const TileDesc& t, unsigned char* dst) {
  const int n = (t.bond1 - t.bond0 + 7) >> 3;
  const uint4* src = reinterpret_cast<const uint4*>(slot16 + t.bond0);
  uint4* d = reinterpret_cast<uint4*>(dst);
  for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = src[i];
  return reinterpret_cast<const unsigned short*>(dst);
}

// node of halo index s
__device__ __forceinline__ int halo_node(const TileSmem& ts, int s) {
  int r = 0;
#pragma unroll
  for (int q = 1; q < 9; ++q) r += (s >= ts.off[q]) ? 1 : 0;
  return ts.hb[r] + (s - ts.off[r]);
}

// Records that an item of an instance is done; true in the CTA that completed the
// instance's last one (all threads).  `count` = number of items of the instance.
__device__ __forceinline__ bool item_done(unsigned int* ticket, int count, int* s_flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int t = atomicAdd(ticket, 1u);
    *s_flag = (t == (unsigned int)(count - 1)) ? 1 : 0;
  }
  __syncthreads();
  const bool last = *s_flag != 0;
  if (last) __threadfence();
  return last;
}

// thread 0 of an instance's finishing CTA: reset its ticket, count the instance as done and,
// in the last instance, set the loop condition to "any instance active".
__device__ __forceinline__ void instance_finished(const EngineView& v, int inst, int which,
                                                  cudaGraphConditionalHandle hc) {
  v.ticket[inst] = 0;
  __threadfence();
  const unsigned int g = atomicAdd(&v.ticket[v.M], 1u);
  if (g == (unsigned int)(v.M - 1)) {
    __threadfence();
    v.ticket[v.M] = 0;
    int any = 0;
    for (int i = 0; i < v.M; ++i) {
      const DevState* ds = v.inst[i].ds;
      any |= (which == 0) ? *((volatile const int*)&ds->outer_active)
                          : *((volatile const int*)&ds->inner_active);
    }
    if (v.in_graph) cudaGraphSetConditional(hc, any ? 1u : 0u);
  }
}

// reduce NV partials of items [first, first+count) (layout partials[k*stride + item])
template <int NV>
__device__ __forceinline__ void reduce_items(const double* partials, int stride, int first, int count,
                                             double (&out)[NV], double* sm) {
  // eight independent accumulators per thread (loads in flight together), combined in a
  // fixed order: the sum does not depend on timing
  constexpr int U = 8;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const double* p = partials + (size_t)k * stride + first;
    double x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = 0.0;
    int b = threadIdx.x;
    for (; b + (U - 1) * kBlock < count; b += U * kBlock)
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] += p[b + u * kBlock];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (b + u * kBlock < count) x[u] += p[b + u * kBlock];
    out[k] = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  }
  block_sum<NV, kBlock>(out, sm);
}

template <int NV>
__device__ __forceinline__ void write_partials(const EngineView& v, int item, double (&part)[NV], double* sm) {
  block_sum<NV, kBlock>(part, sm);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) v.partials[(size_t)k * v.stride + item] = part[k];
}

// Pair partials: the FP32 path's item partials are FP32 pairs (hi, lo) stored in the 8-byte
// slots of the partials buffer, so that the last CTA sums them on the FP32 pipes (an FP64
// sum of the ~19k slice partials of a 512k-node pass would hold one SM's FP64 pipe for
// microseconds).
__device__ __forceinline__ void store_pair(double* partials, size_t idx, float hi, float lo) {
  reinterpret_cast<float2*>(partials)[idx] = make_float2(hi, lo);
}

// FP32 pair of an FP64 value x*x (x split into a pair, the square to ~2^-46 relative)
__device__ __forceinline__ void pair_square(double x, float& h, float& l) {
  float xh, xl;
  split_pair(x, xh, xl);
  h = xh * xh;
  l = fmaf(xh, xh, -h) + 2.0f * xh * xl;
}

// block sums of NV pairs per thread; thread 0 gets the FP64 values (sm: NV * BLK / 32
// doubles, used as pairs)
template <int NV, int BLK = kBlock>
__device__ __forceinline__ void block_pair_sum(float (&h)[NV], float (&l)[NV], double (&out)[NV], double* sm) {
  float2* smf = reinterpret_cast<float2*>(sm);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    pair_warp_sum(h[q], l[q]);
    if (lane == 0) smf[q * (BLK / 32) + wid] = make_float2(h[q], l[q]);
  }
  __syncthreads();
  if (wid == 0) {
    // value q ends in lane q, so that one conversion (the FP64 pipe) serves all of them
    static_assert(NV <= 32, "a value a lane");
    float mh = 0.0f, ml = 0.0f;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      float th = 0.0f, tl = 0.0f;
      if (lane < BLK / 32) {
        th = smf[q * (BLK / 32) + lane].x;
        tl = smf[q * (BLK / 32) + lane].y;
      }
      pair_warp_sum(th, tl);
      const float h0 = __shfl_sync(0xffffffffu, th, 0), l0 = __shfl_sync(0xffffffffu, tl, 0);
      if (lane == q) {
        mh = h0;
        ml = l0;
      }
    }
    const double d = (double)mh + (double)ml;
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = __shfl_sync(0xffffffffu, d, q);
  }
  __syncthreads();
}

// reduce NV pair partials of items [first, first+count) (layout partials[k*stride + item]);
// four independent pair accumulators per thread, combined in a fixed order
template <int NV, int BLK = kBlock>
__device__ __forceinline__ void reduce_pair_items(const double* partials, int stride, int first, int count,
                                                  double (&out)[NV], double* sm) {
  constexpr int U = 4;
  const float2* pp = reinterpret_cast<const float2*>(partials);
  float hh[NV], ll[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const float2* p = pp + (size_t)k * stride + first;
    float h[U], l[U];
#pragma unroll
    for (int u = 0; u < U; ++u) h[u] = l[u] = 0.0f;
    int b = threadIdx.x;
    for (; b + (U - 1) * BLK < count; b += U * BLK) {
      float2 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = p[b + u * BLK];
#pragma unroll
      for (int u = 0; u < U; ++u) pair_add(h[u], l[u], x[u].x, x[u].y);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (b + u * BLK < count) pair_add(h[u], l[u], p[b + u * BLK].x, p[b + u * BLK].y);
    pair_add(h[0], l[0], h[1], l[1]);
    pair_add(h[2], l[2], h[3], l[3]);
    pair_add(h[0], l[0], h[2], l[2]);
    hh[k] = h[0];
    ll[k] = l[0];
  }
  block_pair_sum<NV, BLK>(hh, ll, out, sm);
}

// the last CTA's reduction of items written by write_dot_partials
template <int NV, typename P>
__device__ __forceinline__ void reduce_dot_items(const double* partials, int stride, int first, int count,
                                                 double (&out)[NV], double* sm) {
  if constexpr (sizeof(P) == 8)
    reduce_items<NV>(partials, stride, first, count, out, sm);
  else
    reduce_pair_items<NV>(partials, stride, first, count, out, sm);
}

// FP64 slice partials: a warp stores its slice's values (lane 0 holds them) and the warp that
// completes a group of 32 of the instance's slices sums the group, so that the last CTA is
// left with a thirty-second of the FP64 additions (one SM's FP64 pipe takes microseconds for
// the slices of a 512k-node pass).  Groups are fixed, so the sums do not depend on timing.
// `first`, `count`: the instance's slices; group sums at partials[(NV + k) * stride + slot].
__device__ __forceinline__ int slice_group0(int first, int inst) { return (first >> 5) + inst; }
template <int NV>
__device__ __forceinline__ void slice_partials64(const EngineView& v, int inst, int first, int count, int sg,
                                                 const double (&val)[NV]) {
  const int lane = threadIdx.x & 31;
  const int gi = (sg - first) >> 5, members = min(32, count - 32 * gi);
  const int slot = slice_group0(first, inst) + gi;
  unsigned int t = 0;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v.partials[(size_t)k * v.stride + sg] = val[k];
    __threadfence();
    t = atomicAdd(&v.gcount[slot], 1u);
  }
  t = __shfl_sync(0xffffffffu, t, 0);
  if (t != (unsigned int)(members - 1)) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = lane < members ? __ldcg(&v.partials[(size_t)k * v.stride + first + 32 * gi + lane]) : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if (lane == 0) v.partials[(size_t)(NV + k) * v.stride + slot] = x;
  }
  if (lane == 0) v.gcount[slot] = 0;
}
// the last CTA's sum of an instance's groups
template <int NV>
__device__ __forceinline__ void reduce_slices64(const EngineView& v, int inst, int first, int count, double (&out)[NV],
                                                double* sm) {
  reduce_items<NV>(v.partials + (size_t)NV * v.stride, v.stride, slice_group0(first, inst), (count + 31) >> 5, out, sm);
}

// Item partials of per-thread dot accumulators: FP64 block sums on the FP64 path; on the
// FP32 path FP32-pair warp sums, then warp 0 sums the warps' pairs (sm: NV * kBlock / 32
// doubles, reused as pairs) and stores the pair partials (reduce_dot_items sums them).
template <int NV, typename P>
__device__ __forceinline__ void write_dot_partials(const EngineView& v, int item, DotAcc<P> (&acc)[NV], double* sm) {
  if constexpr (sizeof(P) == 8) {
    double part[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) part[q] = acc[q].s;
    write_partials<NV>(v, item, part, sm);
  } else {
    float2* smf = reinterpret_cast<float2*>(sm);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      acc[q].warp_sum();
      if (lane == 0) smf[q * (kBlock / 32) + wid] = make_float2(acc[q].hi, acc[q].lo);
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        DotAcc<float> t;
        if (lane < kBlock / 32) {
          t.hi = smf[q * (kBlock / 32) + lane].x;
          t.lo = smf[q * (kBlock / 32) + lane].y;
        }
        t.warp_sum();
        if (lane == 0) store_pair(v.partials, (size_t)q * v.stride + item, t.hi, t.lo);
      }
    }
    __syncthreads();
  }
}

template <typename P>
struct VecSel;
template <>
struct VecSel<float> {
  __device__ static float* rin(const KParams& k) { return k.rin32; }
  __device__ static float* z(const KParams& k) { return k.z32; }
  __device__ static float* p(const KParams& k) { return k.p32; }
  __device__ static float* q(const KParams& k) { return k.q32; }
  __device__ static float* e(const KParams& k) { return k.e32; }
  __device__ static const float* dinv(const KParams& k) { return k.dinv32; }
  __device__ static const float* d(const KParams& k) { return k.d32; }
};
template <>
struct VecSel<double> {
  __device__ static double* rin(const KParams& k) { return k.rin64; }
  __device__ static double* z(const KParams& k) { return k.z64; }
  __device__ static double* p(const KParams& k) { return k.p64; }
  __device__ static double* q(const KParams& k) { return k.q64; }
  __device__ static double* e(const KParams& k) { return k.e64; }
  __device__ static const double* dinv(const KParams& k) { return k.dinv64; }
  __device__ static const double* d(const KParams& k) { return k.dsum64; }
};

template <typename P>
__device__ __forceinline__ float phase_of(const KParams& k, int a);
template <>
__device__ __forceinline__ float phase_of<float>(const KParams& k, int a) {
  return k.rec32_cur[a].phase;
}
template <>
__device__ __forceinline__ float phase_of<double>(const KParams& k, int a) {
  return (float)k.rec64_cur[a].phase;
}

template <typename P>
__device__ __forceinline__ double conc_of(const KParams& k, int a, int s);
template <>
__device__ __forceinline__ double conc_of<float>(const KParams& k, int a, int s) {
  const float4 lo = k.clo[a];
  const float l = s == 0 ? lo.x : s == 1 ? lo.y : s == 2 ? lo.z : lo.w;
  return (double)k.rec32_cur[a].c[s] + (double)l;
}
template <>
__device__ __forceinline__ double conc_of<double>(const KParams& k, int a, int s) {
  return k.rec64_cur[a].c[s];
}

__device__ __forceinline__ void set_phi_rec(const KParams& k, int a, double phi, bool mixed) {
  if (mixed) {
    const float hi = (float)phi;
    k.rec32_cur[a].phi_hi = hi;
    k.rec32_cur[a].phi_lo = (float)(phi - (double)hi);
  } else {
    k.rec64_cur[a].phi = phi;
  }
}

__device__ __forceinline__ float sel4(const float4& v, int s) {
  return s == 0 ? v.x : s == 1 ? v.y : s == 2 ? v.z : v.w;
}

// sum of pairs over the W lanes of a node's segment (lane 0 of the segment holds it)
template <int WIDTH>
__device__ __forceinline__ double seg_reduce_pair(float h, float l) {
#pragma unroll
  for (int off = WIDTH / 2; off > 0; off >>= 1) {
    const float oh = __shfl_down_sync(0xffffffffu, h, off, WIDTH);
    const float ol = __shfl_down_sync(0xffffffffu, l, off, WIDTH);
    pair_add(h, l, oh, ol);
  }
  return (double)h + (double)l;
}

// ------------------------------------------------------------------- potential: F11 ------
// The reference's F11 (utils.h:798-841) for every node of one instance: the sum of liquid-liquid
// weights times the potential's differences against b = (1/(K sigma)) F CSolid sum_k z_k c_k,
// zero on nodes without such a bond.  CTA per tile, its halo staged in shared memory.
template <typename P, int W>
__global__ void __launch_bounds__(kBlock) k_f11(EngineView v, double* F11_out) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ TileSmem ts;
  const int sub = threadIdx.x % W, seg = threadIdx.x / W, nseg = kBlock / W;
  for (int item = blockIdx.x; item < v.ntiles; item += gridDim.x) {
    const TileDesc t = v.tiles[item];
    const KParams& k = v.inst[t.inst];
    load_tile(t, ts);
    constexpr bool kPair = sizeof(P) == 4;  // mixed path: FP32-pair arithmetic on the bonds
    double* sphi = reinterpret_cast<double*>(dsm);
    float2* sphi2 = reinterpret_cast<float2*>(dsm);
    unsigned char* sfl = dsm + sizeof(double) * (size_t)t.halo;
    const unsigned short* sslot = stage_slots(k.slot16, t, dsm + align16(sizeof(double) * (size_t)t.halo + t.halo));
    for (int s = threadIdx.x; s < t.halo; s += kBlock) {
      const int n = halo_node(ts, s);
      const double ph = k.phi64[n];
      if (kPair) {
        const float hi = (float)ph;
        sphi2[s] = make_float2(hi, (float)(ph - (double)hi));
      } else {
        sphi[s] = ph;
      }
      sfl[s] = phase_of<P>(k, n) == 0.0f ? 1 : 0;
    }
    __syncthreads();
    const int* row = k.row;
    const int own0 = ts.off[4] + (t.own_begin - t.hb[4]);
    for (int a0 = t.own_begin; a0 < t.own_end; a0 += nseg) {
      const int a = a0 + seg;
      const bool act = a < t.own_end;
      const int so = own0 + (a - t.own_begin);
      const bool scan = act && sfl[so];
      double dsum = 0.0, swphi = 0.0;
      int anyll = 0;
      if (kPair) {
        float dh = 0.f, dl = 0.f, sh = 0.f, sl = 0.f;
        if (scan)
          for (int j = row[a] + sub; j < row[a + 1]; j += W) {
            const int s = sslot[j - t.bond0];
            if (!sfl[s]) continue;
            const float wh = k.w32[j], wl = k.wlo32[j];
            const float2 ph = sphi2[s];
            float ph_, pl_;
            pair_mul(wh, wl, ph.x, ph.y, ph_, pl_);
            pair_add(dh, dl, wh, wl);
            pair_add(sh, sl, ph_, pl_);
            anyll = 1;
          }
        dsum = seg_reduce_pair<W>(dh, dl);
        swphi = seg_reduce_pair<W>(sh, sl);
      } else {
        if (scan)
          for (int j = row[a] + sub; j < row[a + 1]; j += W) {
            const int s = sslot[j - t.bond0];
            if (!sfl[s]) continue;
            const double w = k.w64[j];
            dsum += w;
            swphi += w * sphi[s];
            anyll = 1;
          }
        dsum = seg_reduce_d<W>(dsum);
        swphi = seg_reduce_d<W>(swphi);
      }
      anyll = seg_or<W>(anyll);
      if (act && sub == 0) {
        double R11 = 0.0;
        for (int s = 0; s < S; ++s) R11 += k.z[s] * conc_of<P>(k, a, s);
        const double b = k.b_override ? k.b_override[a] : k.lam * R11;
        const double pha = kPair ? (double)sphi2[so].x + (double)sphi2[so].y : sphi[so];
        F11_out[a] = anyll ? (dsum * pha - swphi) - b : 0.0;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------- potential: CG -------
// Inner PCG on A e = r (r: FP64 outer residual rounded to P).  Jacobi preconditioner
// (the reference's Eigen::DiagonalPreconditioner, main.cpp:714-768).
template <typename P>
__global__ void __launch_bounds__(kBlock) k_cg_init(EngineView v, cudaGraphConditionalHandle hc,
                                                    int fp64, int split) {
  __shared__ double sm[2 * kBlock / 32];
  __shared__ int s_last;
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const bool active = *((volatile int*)&k.ds->outer_active) != 0;
    DotAcc<P> part[2];
    if (split) {
      // two-level preconditioner: r, p, q, e here; z and the dots after the coarse solve
      if (active) {
        P* rin = VecSel<P>::rin(k);
        P* p = VecSel<P>::p(k);
        P* q = VecSel<P>::q(k);
        P* e = VecSel<P>::e(k);
        for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
          rin[a] = (P)k.r64[a];
          p[a] = P(0);
          q[a] = P(0);
          e[a] = P(0);
          if (sizeof(P) == 4) {  // the deflated solve's right-hand side and t = A e^
            k.r0_32[a] = (float)k.r64[a];
            k.t32[a] = 0.0f;
          }
        }
      }
      continue;
    }
    if (active) {
      P* rin = VecSel<P>::rin(k);
      P* z = VecSel<P>::z(k);
      P* p = VecSel<P>::p(k);
      P* q = VecSel<P>::q(k);
      P* e = VecSel<P>::e(k);
      const P* dinv = VecSel<P>::dinv(k);
      for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
        const P r = (P)k.r64[a];
        const P zz = r * dinv[a];
        rin[a] = r;
        z[a] = zz;
        p[a] = P(0);
        q[a] = P(0);
        e[a] = P(0);
        part[0].add(r, zz);
        part[1].add(r, r);
      }
    }
    write_dot_partials<2, P>(v, item, part, sm);
    if (item_done(&v.ticket[c.inst], v.chunk_count[c.inst], &s_last)) {
      double tot[2];
      reduce_dot_items<2, P>(v.partials, v.stride, v.chunk_first[c.inst], v.chunk_count[c.inst], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = k.ds;
        if (ds->outer_active) {
          ds->rz = tot[0];
          ds->rr = tot[1];
          ds->beta = 0.0;
          ds->alpha = 0.0;
          ds->inner_it = 0;
          // FP64: solve to the final tolerance in one sweep; mixed: reduce by inner_rel, but
          // not below what the outer tolerance needs (0.3 tol: the last sweep stops early)
          const double target = fp64 ? 0.25 * ds->tol * ds->tol * ds->bnorm2
                                     : fmax(ds->inner_rel * ds->inner_rel * tot[1],
                                            0.09 * ds->tol * ds->tol * ds->bnorm2);
          ds->inner_target = target;
          ds->inner_active = (tot[1] > target && ds->max_iter > 0) ? 1 : 0;
        } else {
          ds->inner_active = 0;
        }
        instance_finished(v, c.inst, 1, hc);
      }
    }
    __syncthreads();
  }
}

// Work split of the slice list: warp gw of nw takes the contiguous range [s0, s1), so the
// warps of one CTA walk neighbouring slices and share their neighbours in L1.
__device__ __forceinline__ void warp_slices(const EngineView& v, int* s0, int* s1) {
  const long long nw = (long long)gridDim.x * (kBlock / 32);
  const long long gw = (long long)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  *s0 = (int)(((long long)v.nslices * gw) / nw);
  *s1 = (int)(((long long)v.nslices * (gw + 1)) / nw);
}

// the next slice of a kernel whose warps claim slices one at a time from the grid-wide
// counter ticket[M + 2] (reset by the kernel's last CTA); lane 0 claims, the warp shares it
__device__ __forceinline__ int claim_slice(const EngineView& v, int lane) {
  int s = 0;
  if (lane == 0) s = (int)atomicAdd(&v.ticket[v.M + 2], 1u);
  return __shfl_sync(0xffffffffu, s, 0);
}

__device__ __forceinline__ double warp_sum_d(double x) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
  return x;
}


// Interleaved sliced operator: a quad of bond columns of a slice holds, per lane, the four FP32
// weights of its row's bonds (32 x 16 bytes), then per lane their four 16-bit slot codes (32 x 8
// bytes): one 16-byte and one 8-byte load a lane bring four bonds, and one contiguous copy
// moves both.  A column takes 48 floats (192 bytes) on average; widths are padded to quads.
constexpr int kSellW = 48;              // floats a column
constexpr int kQuadW = 4 * kSellW;      // floats a quad
__device__ __forceinline__ const float* sell_w(const KParams& k, const SliceDesc& d) {
  return k.sell + (size_t)(d.off >> 5) * kSellW;
}

// the CG operator's compacted copy (same layout and offsets; columns in use: cg_width)
__device__ __forceinline__ const float* sell_cg_w(const KParams& k, const SliceDesc& d) {
  return k.sell_cg + (size_t)(d.off >> 5) * kSellW;
}

// the inner-loop flag of a slice's instance (constant while the operator runs)
__device__ __forceinline__ bool slice_active(const EngineView& v, int sg) {
  return __ldg(&v.inst[__ldg(&v.slices[sg].inst)].ds->inner_active) != 0;
}

// node of a slot code: window row start (per-warp table of the slice's lo[]) + offset
// streamed operator loads: no L1 allocation (L1 stays with the gathered vectors) and L2
// evict-first (the operator is read once per pass; the vectors and the coarse inverse the
// other kernels of the iteration read stay in L2)
__device__ __forceinline__ uint64_t stream_policy() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p), "l"(stream_policy()));
  return v;
}
__device__ __forceinline__ uint2 ld_stream(const uint2* p) {
  uint2 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
      : "=r"(v.x), "=r"(v.y)
      : "l"(p), "l"(stream_policy()));
  return v;
}
// a lane's view of a slice's operator: quad q's weights and codes
struct QuadPtr {
  const float4* w;
  const uint2* c;
  __device__ __forceinline__ QuadPtr(const float* base, int lane)
      : w(reinterpret_cast<const float4*>(base) + lane), c(reinterpret_cast<const uint2*>(base + 128) + lane) {}
  __device__ __forceinline__ float4 weights(int q) const { return ld_stream(w + (kQuadW / 4) * q); }
  __device__ __forceinline__ uint2 codes(int q) const { return ld_stream(c + (kQuadW / 2) * q); }
};
// the FP64 weights of a quad: 32 bytes a lane
__device__ __forceinline__ void ld_stream_d4(const double* p, double (&w)[4]) {
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f64 {%0, %1, %2, %3}, [%4], %5;"
      : "=d"(w[0]), "=d"(w[1]), "=d"(w[2]), "=d"(w[3])
      : "l"(p), "l"(stream_policy()));
}
__device__ __forceinline__ float quad_weight(const float4& w, int u) { return u == 0 ? w.x : u == 1 ? w.y : u == 2 ? w.z : w.w; }
__device__ __forceinline__ unsigned int quad_code(const uint2& c, int u) {
  const unsigned int v = u < 2 ? c.x : c.y;
  return u & 1 ? v >> 16 : v & 0xffffu;
}

__device__ __forceinline__ int code_node(const int* hb, unsigned int code) {
  return hb[code >> 12] + (int)(code & 4095u);
}

// q = A z + beta q, p = z + beta p (so that q = A p), partial p.q -> alpha.
// FP32, on the CG operator's slices (32 of a bin row's nodes without a potential Dirichlet
// value; each row holds only its bonds to possible unknowns, in bond order, zero-padded to
// the slice's longest, in quads of bond columns: a 16-byte and an 8-byte load a lane bring four
// bonds), one lane per row.  WIN: the warp first copies the slice's window (the z values of its 9 window rows)
// into its shared-memory buffer with asynchronous 16-byte copies and gathers from there (the
// code's low 12 bits are the position in the window); otherwise it gathers from L1/L2.
// PF > 0: lane 0 keeps bulk L2 prefetches of the warp's operator stream PF batches ahead of
// the batch being read (the warp's slices are contiguous in the sliced array), so that the
// batch loads hit L2.  Slice partials are reduced per instance by the last CTA.
template <int W, bool WIN, int B, bool PIPE, int MINB, int PF = 0>
__global__ void __launch_bounds__(kBlock, MINB) k_cg_spmv32(EngineView v) {
  extern __shared__ __align__(16) float zwin[];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // PF == 0: warps claim slices one at a time (slices of solid nodes and narrow ones cost
  // less than full ones, and a static split leaves warps idle at the end of the single
  // wave); PF > 0 keeps each warp's contiguous range for its prefetch stream
  constexpr bool kClaim = PF == 0;
  const int ns = v.ncslices;
  int s0, s1;
  if (kClaim) {
    s0 = claim_slice(v, lane);
    s1 = ns;
  } else {
    const long long nw = (long long)gridDim.x * (kBlock / 32);
    const long long gw = (long long)blockIdx.x * (kBlock / 32) + warp;
    s0 = (int)(((long long)ns * gw) / nw);
    s1 = (int)(((long long)ns * (gw + 1)) / nw);
  }
  float* zw = zwin + (WIN ? (size_t)warp * kWinCap : 0);
  // prefetch window of the operator stream: [pf_next, pf_end) of the warp's byte range
  const char* pf_next = nullptr;
  const char* pf_end = nullptr;
  if (PF > 0 && s0 < s1) {
    const SliceDesc& da = v.cslices[s0];
    const SliceDesc& db = v.cslices[s1 - 1];
    pf_next = reinterpret_cast<const char*>(sell_cg_w(v.inst[da.inst], da));
    pf_end = reinterpret_cast<const char*>(sell_cg_w(v.inst[db.inst], db)) + (size_t)db.width * kSellW * 4;
    if (da.inst != db.inst) pf_end = pf_next;  // the range spans instances: no prefetch
    if (lane == 0) {
      const char* stop = pf_next + (size_t)PF * B * kSellW * 4;
      if (stop > pf_end) stop = pf_end;
      for (; pf_next < stop; pf_next += B * kSellW * 4)
        bulk_prefetch_l2(pf_next, (unsigned)min((size_t)B * kSellW * 4, (size_t)(pf_end - pf_next)));
    }
  }
  for (int sg = s0; sg < s1; sg = kClaim ? claim_slice(v, lane) : sg + 1) {
    const SliceDesc& d = v.cslices[sg];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    DotAcc<float> part;
    if (__ldg(&k.ds->inner_active) != 0) {
      const int cs = sg - __ldg(&v.cslice_first[inst]);
      const int width = k.cg_width[cs];
      const int a = k.cg_rows[__ldg(&d.row0) + lane];
      const bool live = a >= 0 && k.freem[a];
      if (WIN && width > 0) {
        // the window (z of the 9 window rows, 16-byte aligned row segments) by 16-byte
        // cp.async, all copies in flight before the one wait
        const float* zg = k.z32;
#pragma unroll 1
        for (int r = 0; r < 9; ++r) {
          const int n = d.wlen[r], lo = d.lo[r], wo = d.woff[r];
          for (int i = 4 * lane; i < n; i += 128)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(zw + wo + i)), "l"(zg + lo + i)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      } else if (lane < 9) {
        s_hb[warp][lane] = d.gbase[lane];
      }
      __syncwarp();
      if (PF > 0 && lane == 0) {
        // keep the prefetches at least PF batches ahead of this slice's first column
        const char* target = reinterpret_cast<const char*>(sell_cg_w(k, d)) + (size_t)PF * B * kSellW * 4;
        if (target > pf_end) target = pf_end;
        for (; pf_next < target; pf_next += B * kSellW * 4)
          bulk_prefetch_l2(pf_next, (unsigned)min((size_t)B * kSellW * 4, (size_t)(pf_end - pf_next)));
      }
      // every lane of a slice with a live row runs the slice's columns (the shorter rows hold
      // code 0, weight 0), so that lane 0 can issue the prefetches
      if (PF > 0 ? __any_sync(0xffffffffu, live) : live) {
        const int* hb = s_hb[warp];
        const QuadPtr op(sell_cg_w(k, d), lane);
        const float* z = k.z32;
        // QB quads (B columns) per batch; PIPE: the next batch of streamed quads is in flight
        // while the current batch's neighbour values are gathered (more registers, fewer warps).
        // The last batch's missing quads take weight 0 and code 0 (a valid node).
        constexpr int QB = B / 4;
        const int nq = (width + 3) >> 2;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float4 w[QB];
        uint2 code[QB];
        auto load = [&](int q0) {
#pragma unroll
          for (int u = 0; u < QB; ++u) {
            w[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            code[u] = make_uint2(0u, 0u);
            if (q0 + u < nq) {
              w[u] = op.weights(q0 + u);
              code[u] = op.codes(q0 + u);
            }
          }
        };
        if (PIPE) load(0);
        for (int q0 = 0; q0 < nq; q0 += QB) {
          if (PF > 0 && lane == 0 && pf_next < pf_end) {
            bulk_prefetch_l2(pf_next, (unsigned)min((size_t)B * kSellW * 4, (size_t)(pf_end - pf_next)));
            pf_next += B * kSellW * 4;
          }
          if (!PIPE) load(q0);
          float zv[B];
#pragma unroll
          for (int u = 0; u < B; ++u) {
            const unsigned int cd = quad_code(code[u >> 2], u & 3);
            zv[u] = WIN ? zw[cd & 4095u] : __ldg(z + code_node(hb, cd));
          }
          float4 wc[QB];
#pragma unroll
          for (int u = 0; u < QB; ++u) wc[u] = w[u];
          if (PIPE && q0 + QB < nq) load(q0 + QB);
#pragma unroll
          for (int u = 0; u < B; ++u) acc[u & 3] = fmaf(quad_weight(wc[u >> 2], u & 3), zv[u], acc[u & 3]);
        }
        if (live) {
          const float za = z[a];
          const float sa = k.d32[a] * za - ((acc[0] + acc[1]) + (acc[2] + acc[3]));
          const float beta = (float)k.ds->beta;
          const float qn = sa + beta * k.q32[a];
          const float pn = za + beta * k.p32[a];
          k.q32[a] = qn;
          k.p32[a] = pn;
          part.add(pn, qn);
        }
      }
      __syncwarp();
    }
    part.warp_sum();
    if (lane == 0) store_pair(v.partials, sg, part.hi, part.lo);
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = v.inst[i].ds;
        if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      }
    }
    if (threadIdx.x == 0) {
      v.ticket[v.M + 1] = 0;
      v.ticket[v.M + 2] = 0;
    }
  }
}

// The warp's share of a slice that K warps of a CTA split: part p of K takes the quads p, p + K,
// ...; the parts' sums meet in shared memory and part 0 finishes the row.  For sizes at which a
// warp a slice leaves most of the chip's warps empty and a pass is one slice's chain of loads
// (8,000 nodes: 110 slices of unknowns on 152 SMs).
template <int K>
struct SplitSlice {
  static constexpr int kSlices = (kBlock / 32) / K;  // slices of a CTA at a time
  int sg, part;
  __device__ __forceinline__ SplitSlice(int base) : sg(base + (threadIdx.x >> 5) / K), part((threadIdx.x >> 5) % K) {}
};
// the parts' sums of NV values a lane: part 0 gets the totals, in part order (sm: kBlock * NV).  With as
// many values as parts each part adds a share of them (16 FP64 values of eight parts are 112 additions
// of 64 cycles in part 0 alone).
template <int K, int NV, typename T>
__device__ __forceinline__ void split_sum(T (&v)[NV], T* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (NV >= K && K > 1) {
    const int part = warp % K;
    T* own = sm + (size_t)(warp - part) * NV * 32 + lane;  // part 0's values, the next part's NV * 32 on
#pragma unroll
    for (int q = 0; q < NV; ++q) own[(part * NV + q) * 32] = v[q];
    __syncthreads();
    for (int q = part; q < NV; q += K) {
      T t = own[q * 32];
#pragma unroll
      for (int h = 1; h < K; ++h) t += own[(h * NV + q) * 32];
      own[q * 32] = t;
    }
    __syncthreads();
    if (part == 0)
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] = own[q * 32];
    return;
  }
  if (warp % K)
#pragma unroll
    for (int q = 0; q < NV; ++q) sm[(warp * NV + q) * 32 + lane] = v[q];
  __syncthreads();
  if (warp % K == 0)
#pragma unroll
    for (int h = 1; h < K; ++h)
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] += sm[((warp + h) * NV + q) * 32 + lane];
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_cg_spmv32k(EngineView v) {
  constexpr int QB = 4;
  __shared__ float s_acc[kBlock];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.ncslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.cslices[have ? ss.sg : 0];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    const bool run = have && __ldg(&k.ds->inner_active) != 0;
    float sum[1] = {0.0f};
    int a = -1;
    bool live = false;
    if (run) {
      const int width = k.cg_width[ss.sg - __ldg(&v.cslice_first[inst])];
      a = k.cg_rows[__ldg(&d.row0) + lane];
      live = a >= 0 && k.freem[a];
      if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
      __syncwarp();
      const int* hb = s_hb[warp];
      const QuadPtr op(sell_cg_w(k, d), lane);
      const float* z = k.z32;
      const int nq = (width + 3) >> 2;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (live)
        for (int q0 = ss.part; q0 < nq; q0 += QB * K) {
          float4 w[QB];
          uint2 code[QB];
#pragma unroll
          for (int u = 0; u < QB; ++u) {
            w[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            code[u] = make_uint2(0u, 0u);
            if (q0 + u * K < nq) {
              w[u] = op.weights(q0 + u * K);
              code[u] = op.codes(q0 + u * K);
            }
          }
          float zv[4 * QB];
#pragma unroll
          for (int u = 0; u < 4 * QB; ++u) zv[u] = __ldg(z + code_node(hb, quad_code(code[u >> 2], u & 3)));
#pragma unroll
          for (int u = 0; u < 4 * QB; ++u) acc[u & 3] = fmaf(quad_weight(w[u >> 2], u & 3), zv[u], acc[u & 3]);
        }
      sum[0] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    split_sum<K, 1>(sum, s_acc);
    if (have && ss.part == 0) {
      DotAcc<float> part;
      if (live) {
        const float za = k.z32[a];
        const float sa = k.d32[a] * za - sum[0];
        const float beta = (float)k.ds->beta;
        const float qn = sa + beta * k.q32[a];
        const float pn = za + beta * k.p32[a];
        k.q32[a] = qn;
        k.p32[a] = pn;
        part.add(pn, qn);
      }
      part.warp_sum();
      if (lane == 0) store_pair(v.partials, ss.sg, part.hi, part.lo);
    }
    __syncthreads();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = v.inst[i].ds;
        if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      }
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// Halo-staged FP32 CG operator with recomputed weights (variant 8): the product of
// k_cg_spmv32 (q = A z + beta q, p = z + beta p, partial p.q) over the rows and columns that
// can be unknowns of the potential solve (no Dirichlet value of the potential; the other
// columns hold z = 0).  A CTA claims tiles one at a time; for each it
//   - starts one bulk copy of the tile's code block into shared memory (an mbarrier wait,
//     bounded: a timeout is recorded in the instance's state and reported as NNPP_ERR_CUDA),
//   - stages the tile's halo as float4 {X, Y, Z, z}: the node's position in units of the bin
//     side, relative to the centre of the halo's box (|X| <= T/2 + 1, |Y|, |Z| <= 1.5, so
//     FP32 keeps it to ~1e-7 of a bin), and the CG vector z,
//   - then its warps take the tile's quads (longest first, from a shared counter); eight
//     lanes per row walk the row's codes (halo slots) and recompute each bond's weight
//     beta(xi) dV / xi^3 (utils.h:17-25, s = 0) from the two staged positions.
// HBM sees the 2-byte codes; positions and z of the halo come through L2.
constexpr unsigned kHaloWaitPolls = 1u << 22;  // polls of the tile copies' mbarrier
// z staging of a halo of hal_cap - 1 nodes: every row rounded out to 16-byte boundaries
__host__ __device__ constexpr int halo_zcap(int hal_cap) { return ((hal_cap - 1 + 9 * 8) + 3) & ~3; }

__device__ __forceinline__ float halo_bond(const float4& pa, const float4& pb, float hc0, float hc1) {
  const float dx = pb.x - pa.x, dy = pb.y - pa.y, dz = pb.z - pa.z;
  const float x2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float ri = rsqrtf(x2);
  const float be = fminf(1.0f, fmaf(-hc1, x2 * ri, hc0));
  return be * (ri * ri) * ri * pb.w;
}

// CHECK (nnpp_set_checks): every quad, row and code is checked against its bounds before
// it indexes an array (a bad one is recorded in bounds_error and replaced by the padding
// slot or an empty row), and with NNPP_CHECK_WAIT_PROBE the kernel also waits, bounded, on a
// barrier that nothing completes after each tile's copies have landed -- the timeout path
// without a copy in flight.
template <bool CHECK>
__global__ void __launch_bounds__(kBlock, 3) k_cg_spmv32h(EngineView v, int hal_cap, int quad_cap) {
  extern __shared__ __align__(16) float4 hal[];
  // after the halo: the z rows (each from a 16-byte aligned node, kHaloZPad floats of slack
  // per row), then the code block
  float* zst = reinterpret_cast<float*>(hal + hal_cap);
  // per quad of the tile: its rows' p.q as an FP32 pair (reduced in quad order, so that the
  // sum does not depend on which warp took which quad)
  float2* qpart = reinterpret_cast<float2*>(zst + halo_zcap(hal_cap));
  unsigned short* cod = reinterpret_cast<unsigned short*>(qpart + quad_cap);
  __shared__ __align__(8) uint64_t bar, probe_bar;
  __shared__ int s_tile, s_quad, s_last, s_stop;
  __shared__ int s_hb[9], s_pre[10], s_zb[9];
  __shared__ double sm[kBlock / 32];
  const int lane = threadIdx.x & 31;
  const int g = lane >> 3, j = lane & 7;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    if (CHECK) mbar_init(&probe_bar, 1);  // one arrival expected, none ever made
    fence_mbar_init();
    s_stop = 0;
  }
  __syncthreads();
  unsigned phase = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      s_tile = s_stop ? v.ntiles : (int)atomicAdd(&v.ticket[v.M + 2], 1u);
      s_quad = 0;
    }
    __syncthreads();
    const int t = s_tile;
    if (t >= v.ntiles) break;
    const int inst = v.tiles[t].inst;
    const KParams& k = v.inst[inst];
    const HTile ht = v.htiles[t];
    const bool run = ht.nq > 0 && __ldg(&k.ds->inner_active) != 0;
    if (run) {
      if (threadIdx.x == 0) {
        // every row of the halo by bulk copies on one mbarrier: the position records (16
        // bytes a node, rows start 16-byte aligned) into their slots, the row's z values
        // from the 16-byte boundary at or below its first node (z is padded past N), and the
        // tile's code block
        int acc = 0, zacc = 0;
        unsigned bytes = (unsigned)ht.clen16 * 16u;
        for (int r = 0; r < 9; ++r) {
          const int hb = v.tiles[t].hb[r], hl = v.tiles[t].hl[r];
          s_hb[r] = hb;
          s_pre[r] = acc;
          const int a0 = hb & ~3;
          s_zb[r] = zacc - a0;  // z of node n of row r at zst[s_zb[r] + n]
          if (hl > 0) {
            bytes += (unsigned)hl * 16u + (unsigned)(((hb + hl + 3) & ~3) - a0) * 4u;
            zacc += ((hb + hl + 3) & ~3) - a0;
          }
          acc += hl;
        }
        s_pre[9] = acc;
        // the previous tile's reads and writes of these buffers come before the copies
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bar, bytes);
        for (int r = 0; r < 9; ++r) {
          const int hb = s_hb[r], hl = s_pre[r + 1] - s_pre[r];
          if (hl <= 0) continue;
          const int a0 = hb & ~3;
          bulk_g2s(hal + s_pre[r], k.posrec + hb, (unsigned)hl * 16u, &bar);
          bulk_g2s(zst + s_zb[r] + a0, k.z32 + a0, (unsigned)(((hb + hl + 3) & ~3) - a0) * 4u, &bar);
        }
        if (ht.clen16 > 0) bulk_g2s(cod, k.hcode + (size_t)ht.cstart16 * 8, (unsigned)ht.clen16 * 16u, &bar);
      }
      __syncthreads();
      if (!mbar_wait_bounded(&bar, phase, kHaloWaitPolls)) {
        k.ds->wait_timeout = 1;
        s_stop = 1;
      }
      phase ^= 1u;
      if (CHECK && (k.checks & NNPP_CHECK_WAIT_PROBE) && !mbar_wait_bounded(&probe_bar, 0, 1u << 10)) {
        k.ds->wait_timeout = 1;
        s_stop = 1;
      }
      // the records as float4 {X, Y, Z, z} in the halo's frame, in place
      const float hinv = k.hinv;
      const float xoff = 0.5f * (float)ht.T;
      const int halo = s_pre[9];
      for (int i = threadIdx.x; i < halo; i += kBlock) {
        int r = 0;
#pragma unroll
        for (int q = 1; q < 9; ++q) r += i >= s_pre[q] ? 1 : 0;
        const float4 pr = hal[i];
        const int pb = __float_as_int(pr.w);
        float4 o;
        o.x = fmaf(pr.x, hinv, (float)((pb & 1023) - ht.bx0) - xoff);
        o.y = fmaf(pr.y, hinv, (float)(((pb >> 10) & 1023) - ht.by) - 0.5f);
        o.z = fmaf(pr.z, hinv, (float)(((pb >> 20) & 1023) - ht.bz) - 0.5f);
        o.w = zst[s_zb[r] + s_hb[r] + (i - s_pre[r])];
        hal[i] = o;
      }
      // the padding slot: far away (weight 0) and z = 0
      if (threadIdx.x == 0) hal[halo] = make_float4(1e18f, 0.0f, 0.0f, 0.0f);
      __syncthreads();
      const int own = s_pre[4] - s_hb[4];  // slot of own node a: own + a
      const float hc0 = k.hc0, hc1 = k.hc1, hsw = k.hsw;
      const float beta = (float)k.ds->beta;
      for (;;) {
        int qi = 0;
        if (lane == 0) qi = atomicAdd(&s_quad, 1);
        qi = __shfl_sync(0xffffffffu, qi, 0);
        if (qi >= ht.nq) break;
        if (CHECK && (ht.q0 + qi < 0 || ht.q0 + qi >= k.hquad_n)) {
          if (lane == 0) k.ds->bounds_error = 1;
          break;
        }
        const HQuad* qd = k.hquad + ht.q0 + qi;
        int a = __ldg(&qd->rows[g]);
        int npass = __ldg(&qd->npass);
        if (CHECK) {
          const TileDesc& td = v.tiles[t];
          const int coff = __ldg(&qd->coff_rel);
          const bool bad_row = a != -1 && (a < td.own_begin || a >= td.own_end);
          const bool bad_codes = npass < 0 || coff < 0 || coff + 32 * npass > 8 * ht.clen16;
          if (bad_row || bad_codes) k.ds->bounds_error = 1;
          if (bad_row) a = -1;
          if (__any_sync(0xffffffffu, bad_codes)) npass = 0;
        }
        const bool live = a >= 0 && k.freem[a] != 0;
        if (!__any_sync(0xffffffffu, live)) {
          if (lane == 0) qpart[qi] = make_float2(0.0f, 0.0f);
          continue;
        }
        const float4 pa = a >= 0 ? hal[own + a] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const unsigned short* cq = cod + __ldg(&qd->coff_rel) + lane;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        int p = 0;
        for (; p + 4 <= npass; p += 4) {
          unsigned sl[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) sl[u] = cq[32 * (p + u)];
          if (CHECK)
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (sl[u] > (unsigned)halo) {
                k.ds->bounds_error = 1;
                sl[u] = (unsigned)halo;
              }
          float4 pb[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) pb[u] = hal[sl[u]];
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[u] += halo_bond(pa, pb[u], hc0, hc1);
        }
        for (; p < npass; ++p) {
          unsigned sl = cq[32 * p];
          if (CHECK && sl > (unsigned)halo) {
            k.ds->bounds_error = 1;
            sl = (unsigned)halo;
          }
          acc[0] += halo_bond(pa, hal[sl], hc0, hc1);
        }
        float sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        float ph = 0.0f, pl = 0.0f;  // this row's p.q, TwoProd
        if (j == 0 && live) {
          const float za = pa.w;
          const float sa = __ldg(k.d32 + a) * za - hsw * sum;
          const float qn = sa + beta * k.q32[a];
          const float pn = za + beta * k.p32[a];
          k.q32[a] = qn;
          k.p32[a] = pn;
          ph = pn * qn;
          pl = fmaf(pn, qn, -ph);
        }
        // the quad's sum, rows in order
        float qh = __shfl_sync(0xffffffffu, ph, 0), ql = __shfl_sync(0xffffffffu, pl, 0);
#pragma unroll
        for (int r = 1; r < 4; ++r)
          pair_add(qh, ql, __shfl_sync(0xffffffffu, ph, 8 * r), __shfl_sync(0xffffffffu, pl, 8 * r));
        if (lane == 0) qpart[qi] = make_float2(qh, ql);
      }
    }
    __syncthreads();
    // the tile's partial: its quads' sums in quad order (lane l takes quads l, l + 32, ...,
    // then a fixed shuffle tree)
    if (threadIdx.x < 32) {
      float th = 0.0f, tl = 0.0f;
      if (run)
        for (int q = lane; q < ht.nq; q += 32) pair_add(th, tl, qpart[q].x, qpart[q].y);
      pair_warp_sum(th, tl);
      if (lane == 0) store_pair(v.partials, t, th, tl);
    }
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.tile_first[i], v.tile_count[i], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = v.inst[i].ds;
        if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      }
    }
    if (threadIdx.x == 0) {
      v.ticket[v.M + 1] = 0;
      v.ticket[v.M + 2] = 0;
    }
  }
}

// Staged FP32 CG operator (the same product as k_cg_spmv32, same work split).  Every warp
// owns, in shared memory,
//   - a ring of kTmaStages stages of kTmaCol interleaved bond columns of its slices (one
//     cp.async.bulk per stage, completed on an mbarrier), refilled by lane 0 as soon as the
//     warp has consumed the stage, and
//   - two window buffers: the z values of the current slice's 9 window rows (the only nodes
//     its bonds reach) and, in flight, the next slice's, copied by the lanes with 16-byte
//     cp.async.
// The gathers are shared-memory loads; HBM only sees the streamed operator.  Waits are
// bounded: a timeout is recorded in the instance's state (reported as NNPP_ERR_CUDA).
constexpr int kTmaCol = 32;
constexpr int kTmaStages = 2;
constexpr int kStageBytes = kTmaCol * kSellW * 4;  // 6 KB
constexpr int kWarpsCta = kBlock / 32;
constexpr size_t kTmaRingBytes = (size_t)kWarpsCta * kTmaStages * kStageBytes;
constexpr size_t kTmaWinBytes = (size_t)kWarpsCta * 2 * kWinCap * sizeof(float);
constexpr size_t kTmaBarBytes = (size_t)kWarpsCta * kTmaStages * sizeof(uint64_t);
constexpr unsigned kWaitPolls = 1u << 22;

__device__ __forceinline__ int tma_chunks(int width) { return width > 0 ? (width + kTmaCol - 1) / kTmaCol : 1; }

// a warp's operator producer (lane 0): position in its slice range and the current slice's
// descriptors, loaded once per slice so that issuing a chunk costs no dependent loads
struct TmaCursor {
  int sg, ch;
  int loaded;  // slice whose fields below are valid (-1: none)
  int width, nch;
  const float* base;
};

// lane 0: issue the cursor's chunk into `stage` and advance; false when the range is done
__device__ __forceinline__ bool tma_produce(const EngineView& v, TmaCursor& c, int s1, int warp, int stage,
                                            unsigned char* ring, uint64_t* bars, uint64_t pol) {
  if (c.loaded != c.sg) {
    while (c.sg < s1 && !slice_active(v, c.sg)) {
      ++c.sg;  // inactive instance: the consumer skips its slices too
      c.ch = 0;
    }
    if (c.sg >= s1) return false;
    const SliceDesc& d = v.slices[c.sg];
    c.width = d.width;
    c.nch = tma_chunks(c.width);
    c.base = sell_w(v.inst[d.inst], d);
    c.loaded = c.sg;
  }
  const int c0 = c.ch * kTmaCol;
  const int cc = min(kTmaCol, max(c.width - c0, 0));
  unsigned char* buf = ring + (size_t)(warp * kTmaStages + stage) * kStageBytes;
  uint64_t* bar = bars + warp * kTmaStages + stage;
  fence_proxy_async_smem();
  mbar_arrive_expect_tx(bar, (unsigned)(cc * kSellW * 4));
  if (cc > 0) bulk_g2s_hint(buf, c.base + (size_t)c0 * kSellW, (unsigned)(cc * kSellW * 4), bar, pol);
  if (++c.ch >= c.nch) {
    c.ch = 0;
    ++c.sg;
  }
  return true;
}

// all lanes: 16-byte cp.async copies of the window of the next active slice at or after *ws
// into zw, then one commit group (empty when no slice is left); advances *ws past it
__device__ __forceinline__ void win_copy(const EngineView& v, int* ws, int s1, float* zw, int lane) {
  while (*ws < s1 && !slice_active(v, *ws)) ++*ws;
  if (*ws < s1) {
    const SliceDesc& d = v.slices[*ws];
    const float* z = v.inst[d.inst].z32;
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
      const int n = d.wlen[r], lo = d.lo[r], wo = d.woff[r];
      for (int i = 4 * lane; i < n; i += 128)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(zw + wo + i)), "l"(z + lo + i)
                     : "memory");
    }
    ++*ws;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// quad q of a staged chunk (shared memory) times the window values
__device__ __forceinline__ void staged_quad(const float* stage, int q, int lane, const float* zw, float (&acc)[4]) {
  const float4 w = reinterpret_cast<const float4*>(stage + kQuadW * q)[lane];
  const uint2 c = reinterpret_cast<const uint2*>(stage + kQuadW * q + 128)[lane];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u] = fmaf(quad_weight(w, u), zw[quad_code(c, u) & 4095u], acc[u]);
}

template <int W>
__global__ void __launch_bounds__(kBlock, 1) k_cg_spmv32t(EngineView v) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* ring = dsm;
  float* wins = reinterpret_cast<float*>(dsm + kTmaRingBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(dsm + kTmaRingBytes + kTmaWinBytes);
  if (threadIdx.x < kWarpsCta * kTmaStages) mbar_init(bars + threadIdx.x, 1);
  fence_mbar_init();
  __syncthreads();
  int s0, s1;
  warp_slices(v, &s0, &s1);
  float* mywin = wins + (size_t)warp * 2 * kWinCap;
  TmaCursor pc{s0, 0, -1, 0, 0, nullptr};
  int wsrc = s0;  // next slice whose window is to be copied
  const uint64_t pol = l2_evict_first_policy();  // the operator is read once per launch
  if (lane == 0)
    for (int st = 0; st < kTmaStages; ++st)
      if (!tma_produce(v, pc, s1, warp, st, ring, bars, pol)) break;
  win_copy(v, &wsrc, s1, mywin, lane);
  int stage = 0, wb = 0;
  unsigned phases = 0u;
  int timed_out = -1;  // instance whose wait gave up
  for (int sg = s0; sg < s1; ++sg) {
    const SliceDesc& d = v.slices[sg];
    const KParams& k = v.inst[d.inst];
    DotAcc<float> part;
    if (slice_active(v, sg)) {
      // the next slice's window goes to the other buffer (free: its slice is done), then
      // this slice's window (the older commit group) is waited for
      win_copy(v, &wsrc, s1, mywin + (wb ^ 1) * kWinCap, lane);
      const int width = d.width;
      const int a = d.row0 + lane;
      const bool live = lane < d.nrows && k.freem[a];
      float za = 0.0f, da = 0.0f, qa = 0.0f, pa = 0.0f;
      if (live) {
        za = k.z32[a];
        da = k.d32[a];
        qa = k.q32[a];
        pa = k.p32[a];
      }
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const float* zw = mywin + wb * kWinCap;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      const int nch = tma_chunks(width);
      for (int ch = 0; ch < nch; ++ch) {
        uint64_t* bar = bars + warp * kTmaStages + stage;
        if (!mbar_wait_bounded(bar, (phases >> stage) & 1u, kWaitPolls)) timed_out = d.inst;
        phases ^= 1u << stage;
        const float* sw = reinterpret_cast<const float*>(ring + (size_t)(warp * kTmaStages + stage) * kStageBytes);
        const int cc = min(kTmaCol, width - ch * kTmaCol);  // a multiple of 4
        if (cc == kTmaCol) {
#pragma unroll 2
          for (int q = 0; q < kTmaCol / 4; ++q) staged_quad(sw, q, lane, zw, acc);
        } else {
          for (int q = 0; q < cc / 4; ++q) staged_quad(sw, q, lane, zw, acc);
        }
        __syncwarp();
        if (lane == 0) tma_produce(v, pc, s1, warp, stage, ring, bars, pol);
        stage = stage + 1 == kTmaStages ? 0 : stage + 1;
      }
      if (live) {
        const float sa = da * za - ((acc[0] + acc[1]) + (acc[2] + acc[3]));
        const float beta = (float)k.ds->beta;
        const float qn = sa + beta * qa;
        const float pn = za + beta * pa;
        k.q32[a] = qn;
        k.p32[a] = pn;
        part.add(pn, qn);
      }
      __syncwarp();
      wb ^= 1;
    }
    part.warp_sum();
    if (lane == 0) store_pair(v.partials, sg, part.hi, part.lo);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (timed_out >= 0 && lane == 0) v.inst[timed_out].ds->wait_timeout = 1;
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.slice_first[i], v.slice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = v.inst[i].ds;
        if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      }
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// Streamed FP32 CG operator for single-instance engines (the same product and work split as
// k_cg_spmv32).  A warp's slices are consecutive in the sliced array, so its whole share of
// the operator is one contiguous byte range: lane 0 streams it through a ring of `stages`
// shared-memory stages of kTmaCol bond columns with cp.async.bulk (completed on mbarriers,
// refilled as soon as a stage is consumed), independently of the slice boundaries.  The
// lanes consume the columns slice by slice and gather from double-buffered slice windows.
// Nothing on a slice's path waits on a dependent global load: the slice descriptors arrive
// by cp.async three slices ahead into a shared-memory ring of four, and each slice's window
// one slice ahead (one cp.async group per slice: the window of slice s + 1 and the
// descriptor of slice s + 3).
// Dynamic shared memory: ring [warps][stages][kStageBytes], windows [warps][2][win_cap]
// floats, barriers [warps][stages], descriptors [warps][4].  Waits are bounded (timeout
// recorded in the state).
constexpr int kDescRing = 4;

// lanes 0..11: 16-byte cp.async copies of slice sg's descriptor into dst (no-op past s1)
__device__ __forceinline__ void desc_copy(const EngineView& v, int sg, int s1, SliceDesc* dst, int lane) {
  static_assert(sizeof(SliceDesc) % 16 == 0, "slice descriptor copied in 16-byte pieces");
  if (sg < s1 && lane < (int)(sizeof(SliceDesc) / 16))
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(reinterpret_cast<char*>(dst) + 16 * lane)),
                 "l"(reinterpret_cast<const char*>(v.slices + sg) + 16 * lane)
                 : "memory");
}

// all lanes: 16-byte cp.async copies of the window of the slice described by d into zw
__device__ __forceinline__ void win_copy_desc(const SliceDesc& d, const float* z, float* zw, int lane) {
#pragma unroll 1
  for (int r = 0; r < 9; ++r) {
    const int n = d.wlen[r], lo = d.lo[r], wo = d.woff[r];
    for (int i = 4 * lane; i < n; i += 128)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(zw + wo + i)), "l"(z + lo + i)
                   : "memory");
  }
}

template <int W, int COL>
__global__ void __launch_bounds__(kBlock, 1) k_cg_spmv32s(EngineView v, int stages, int win_cap) {
  constexpr int SB = COL * kSellW * 4;  // bytes of a stage
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t ring_bytes = (size_t)kWarpsCta * stages * SB;
  const size_t win_bytes = (size_t)kWarpsCta * 2 * win_cap * sizeof(float);
  unsigned char* ring = dsm;
  float* wins = reinterpret_cast<float*>(dsm + ring_bytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(dsm + ring_bytes + win_bytes);
  SliceDesc* descs = reinterpret_cast<SliceDesc*>(dsm + ring_bytes + win_bytes +
                                                  (size_t)kWarpsCta * stages * sizeof(uint64_t));
  if (threadIdx.x < kWarpsCta * stages) mbar_init(bars + threadIdx.x, 1);
  fence_mbar_init();
  __syncthreads();
  int s0, s1;
  warp_slices(v, &s0, &s1);
  const KParams& k = v.inst[0];
  int timed_out = 0;
  if (s0 < s1 && slice_active(v, s0)) {
    const SliceDesc& da = v.slices[s0];
    const SliceDesc& db = v.slices[s1 - 1];
    const char* base = reinterpret_cast<const char*>(sell_w(k, da));
    const size_t total = ((size_t)((db.off - da.off) >> 5) + (size_t)db.width) * kSellW * 4;
    const uint64_t pol = l2_evict_first_policy();  // the operator is read once per launch
    unsigned char* myring = ring + (size_t)warp * stages * SB;
    uint64_t* mybars = bars + warp * stages;
    SliceDesc* mydesc = descs + warp * kDescRing;
    size_t pos = 0;  // lane 0: bytes of the range issued so far
    if (lane == 0)
      for (int st = 0; st < stages && pos < total; ++st) {
        const unsigned bytes = (unsigned)min((size_t)SB, total - pos);
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(mybars + st, bytes);
        bulk_g2s_hint(myring + (size_t)st * SB, base + pos, bytes, mybars + st, pol);
        pos += bytes;
      }
    const float* zg = k.z32;
    float* mywin = wins + (size_t)warp * 2 * win_cap;
    // descriptors of s0 and s0 + 1 now; then the window of s0 with the descriptor of s0 + 2
    desc_copy(v, s0, s1, mydesc, lane);
    desc_copy(v, s0 + 1, s1, mydesc + 1, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    win_copy_desc(mydesc[0], zg, mywin, lane);
    desc_copy(v, s0 + 2, s1, mydesc + 2, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    int stage = 0, wb = 0;
    unsigned phases = 0u;
    bool ready = false;
    int cis = 0;  // column within the current stage
    for (int sg = s0; sg < s1; ++sg) {
      const int j = sg - s0;
      // this slice's window and the descriptors up to sg + 2 are in
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      const SliceDesc& d = mydesc[j & (kDescRing - 1)];
      if (sg + 1 < s1) win_copy_desc(mydesc[(j + 1) & (kDescRing - 1)], zg, mywin + (wb ^ 1) * win_cap, lane);
      desc_copy(v, sg + 3, s1, mydesc + ((j + 3) & (kDescRing - 1)), lane);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const int width = d.width;
      const int a = d.row0 + lane;
      const bool row = lane < d.nrows;
      bool live = false;
      float za = 0.0f, dd = 0.0f, qa = 0.0f, pa = 0.0f;
      if (row) {
        live = k.freem[a] != 0;
        za = k.z32[a];
        dd = k.d32[a];
        qa = k.q32[a];
        pa = k.p32[a];
      }
      const float* zw = mywin + wb * win_cap;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      int c = 0;
      while (c < width) {
        if (!ready) {
          if (!mbar_wait_bounded(mybars + stage, (phases >> stage) & 1u, kWaitPolls)) timed_out = 1;
          phases ^= 1u << stage;
          ready = true;
        }
        const float* sw = reinterpret_cast<const float*>(myring + (size_t)stage * SB);
        const int n = min(COL - cis, width - c);  // widths, and so cis and n, are multiples of 4
        if (n == COL) {
#pragma unroll 2
          for (int q = 0; q < COL / 4; ++q) staged_quad(sw, q, lane, zw, acc);
        } else {
          for (int q = cis / 4; q < (cis + n) / 4; ++q) staged_quad(sw, q, lane, zw, acc);
        }
        c += n;
        cis += n;
        if (cis == COL) {
          // stage consumed: refill it with the range's next chunk
          __syncwarp();
          if (lane == 0 && pos < total) {
            const unsigned bytes = (unsigned)min((size_t)SB, total - pos);
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(mybars + stage, bytes);
            bulk_g2s_hint(myring + (size_t)stage * SB, base + pos, bytes, mybars + stage, pol);
            pos += bytes;
          }
          stage = stage + 1 == stages ? 0 : stage + 1;
          ready = false;
          cis = 0;
        }
      }
      DotAcc<float> part;
      if (live) {
        const float sa = dd * za - ((acc[0] + acc[1]) + (acc[2] + acc[3]));
        const float beta = (float)k.ds->beta;
        const float qn = sa + beta * qa;
        const float pn = za + beta * pa;
        k.q32[a] = qn;
        k.p32[a] = pn;
        part.add(pn, qn);
      }
      __syncwarp();
      wb ^= 1;
      part.warp_sum();
      if (lane == 0) store_pair(v.partials, sg, part.hi, part.lo);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (int sg = s0; sg < s1; ++sg)
      if (lane == 0) store_pair(v.partials, sg, 0.0f, 0.0f);
  }
  if (timed_out && lane == 0) k.ds->wait_timeout = 1;
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    double tot[1];
    reduce_pair_items<1>(v.partials, v.stride, v.slice_first[0], v.slice_count[0], tot, sm);
    if (threadIdx.x == 0) {
      DevState* ds = k.ds;
      if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      v.ticket[v.M + 1] = 0;
    }
  }
}

// The FP64 operator's row sums on the CG slices: sum over this part's quads of w x[node] (FP64
// weights, 32 bytes a lane and quad, next to the codes of the FP32 operator), two quads in flight.
// CONST: x does not change while the kernel runs.
template <int K, bool CONST = true>
__device__ __forceinline__ double cg_row64(const KParams& k, int off, int nq, int lane, int part, const int* hb,
                                           const double* x) {
  constexpr int QB = 2;
  const double* w64 = k.sell_cg64 + (size_t)(off >> 5) * 32 + 4 * lane;
  const QuadPtr op(k.sell_cg + (size_t)(off >> 5) * kSellW, lane);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  int q0 = part;
  for (; q0 + (QB - 1) * K < nq; q0 += QB * K) {
    double w[QB][4], xv[QB][4];
    uint2 code[QB];
#pragma unroll
    for (int u = 0; u < QB; ++u) {
      code[u] = op.codes(q0 + u * K);
      ld_stream_d4(w64 + 128 * (size_t)(q0 + u * K), w[u]);
    }
#pragma unroll
    for (int u = 0; u < QB; ++u)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const double* xp = x + code_node(hb, quad_code(code[u], t));
        xv[u][t] = CONST ? __ldg(xp) : *xp;
      }
#pragma unroll
    for (int u = 0; u < QB; ++u)
#pragma unroll
      for (int t = 0; t < 4; ++t) acc[t] = fma(w[u][t], xv[u][t], acc[t]);
  }
  for (; q0 < nq; q0 += K) {
    double w[4];
    const uint2 code = op.codes(q0);
    ld_stream_d4(w64 + 128 * (size_t)q0, w);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double* xp = x + code_node(hb, quad_code(code, t));
      acc[t] = fma(w[t], CONST ? __ldg(xp) : *xp, acc[t]);
    }
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// FP64 operator on the CG slices (q = A z + beta q, p = z + beta p, p.q), one lane a row, K warps
// a slice: bound by the stream (10 bytes a slot).  512k nodes: 0.1146 ms, against 0.2085
// for FP64 weights per bond with halo tiles in shared memory (the tile form it replaces).
template <int K>
__global__ void __launch_bounds__(kBlock, 4) k_cg_spmv64(EngineView v) {
  __shared__ double s_acc[K > 1 ? kBlock : 1];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.ncslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.cslices[have ? ss.sg : 0];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    const int first = __ldg(&v.cslice_first[inst]);
    double sum[1] = {0.0};
    int a = -1;
    bool live = false;
    if (have && __ldg(&k.ds->inner_active) != 0) {
      a = k.cg_rows[__ldg(&d.row0) + lane];
      live = a >= 0 && k.freem[a];
      if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
      __syncwarp();
      if (live) sum[0] = cg_row64<K>(k, d.off, (k.cg_width[ss.sg - first] + 3) >> 2, lane, ss.part, s_hb[warp], k.z64);
    }
    if (K > 1) split_sum<K, 1>(sum, s_acc);
    if (have && ss.part == 0) {
      double part[1] = {0.0};
      if (live) {
        const double za = k.z64[a];
        const double beta = k.ds->beta;
        const double qn = fma(beta, k.q64[a], fma(k.dsum64[a], za, -sum[0]));
        const double pn = fma(beta, k.p64[a], za);
        k.q64[a] = qn;
        k.p64[a] = pn;
        part[0] = pn * qn;
      }
      part[0] = warp_sum_d(part[0]);
      slice_partials64<1>(v, inst, first, __ldg(&v.cslice_count[inst]), ss.sg, part);
    }
    if (K > 1) __syncthreads();
    else __syncwarp();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_slices64<1>(v, i, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = v.inst[i].ds;
        if (ds->inner_active) {
          ds->alpha = (tot[0] > 0.0 && isfinite(tot[0])) ? ds->rz / tot[0] : 0.0;
          ds->pq = tot[0];
        }
      }
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// e += alpha p, r -= alpha q, z = D^-1 r, partial r.z and r.r -> beta, stop test
template <typename P>
__global__ void __launch_bounds__(kBlock) k_cg_update(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ double sm[2 * kBlock / 32];
  __shared__ int s_last;
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const bool active = *((volatile int*)&k.ds->inner_active) != 0;
    DotAcc<P> part[2];
    if (active) {
      P* rin = VecSel<P>::rin(k);
      P* z = VecSel<P>::z(k);
      const P* p = VecSel<P>::p(k);
      const P* q = VecSel<P>::q(k);
      P* e = VecSel<P>::e(k);
      const P* dinv = VecSel<P>::dinv(k);
      const P alpha = (P)k.ds->alpha;
      for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
        const P di = dinv[a];
        if (di == P(0)) continue;
        const P ee = e[a] + alpha * p[a];
        const P r = rin[a] - alpha * q[a];
        const P zz = r * di;
        e[a] = ee;
        rin[a] = r;
        z[a] = zz;
        part[0].add(r, zz);
        part[1].add(r, r);
      }
    }
    write_dot_partials<2, P>(v, item, part, sm);
    if (item_done(&v.ticket[c.inst], v.chunk_count[c.inst], &s_last)) {
      double tot[2];
      reduce_dot_items<2, P>(v.partials, v.stride, v.chunk_first[c.inst], v.chunk_count[c.inst], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = k.ds;
        if (ds->inner_active) {
          const double alpha_d = ds->alpha;
          ds->beta = ds->rz != 0.0 ? tot[0] / ds->rz : 0.0;
          ds->rz = tot[0];
          ds->rr = tot[1];
          ds->inner_it += 1;
          ds->solve_iters += 1;
          ds->cg_iters += 1;
          const bool go = alpha_d != 0.0 && isfinite(tot[1]) && tot[1] > ds->inner_target &&
                          ds->inner_it < ds->max_iter && ds->solve_iters < ds->max_iter;
          ds->inner_active = go ? 1 : 0;
        }
        instance_finished(v, c.inst, 1, hc);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ two-level preconditioner ----
// Applied as z = D^-1 r + P A_c^-1 P^T r per instance (block diagonal over an ensemble; the
// coarse spaces and their inverses come from coarse.cu): the restriction sums r over each
// aggregate, the coarse solve is one product with the dense inverse, and k_cg_zdots forms z
// with the CG's dots and decisions.  Instances without a coarse space (k.coarse == 0) take
// z = D^-1 r.  All reductions run in a fixed order (reproducible iterates).
__device__ __forceinline__ bool coarse_active(const KParams& k, int which) {
  return (which ? *((volatile int*)&k.ds->inner_active) : *((volatile int*)&k.ds->outer_active)) != 0;
}

// The mixed inner CG runs deflated (DEF1: CG on P_d A e^ = P_d r with P_d = I - A Q,
// Q = P A_c^-1 P^T, e = Q r + e^ - Q A e^) while the coarse operator and A P match the
// phases; otherwise it takes the additive coarse correction.
template <typename P>
__device__ __forceinline__ bool deflating(const KParams& k) {
  return sizeof(P) == 4 && k.coarse && k.defl_ok && *((volatile const int*)&k.ds->defl) != 0;
}

// (A P x_c)_i of an unknown i: its diagonal term from the CG operator's diagonal, the rest
// from the stored rows.  Eight slots at a time (with aggregates two or more bins wide, a
// node's bonds reach at most 8 aggregates): their loads and gathers are in flight together,
// the sum runs in slot order.
// xc: x_c, in global or shared memory.
__device__ __forceinline__ float ap_apply(const KParams& k, int i, const float* xc) {
  float s = __ldg(k.d32 + i) * xc[__ldg(k.agg + i)];
  const size_t N = (size_t)k.N;
  int q = 0;
  for (; q + 8 <= k.ap_k; q += 8) {
    int col[8];
    float val[8], xv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      col[u] = __ldg(k.ap_col + (size_t)(q + u) * N + i);
      val[u] = __ldg(k.ap_val + (size_t)(q + u) * N + i);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) xv[u] = xc[col[u]];
#pragma unroll
    for (int u = 0; u < 8; ++u) s = fmaf(val[u], xv[u], s);
  }
  for (; q < k.ap_k; ++q) {
    const size_t o = (size_t)q * N + i;
    s = fmaf(__ldg(k.ap_val + o), xc[__ldg(k.ap_col + o)], s);
  }
  return s;
}

// The coarse kernels' work: kBlock / 32 aggregates (a warp each) of one instance a tile, the instances'
// tiles in one list, so that an ensemble's small coarse spaces run side by side (eight members of
// 20,000 to 195,000 nodes: restriction 29 us and product 22 us with every warp on one instance after
// another).  False past the last tile.
constexpr int kAggTile = kBlock / 32;
__device__ __forceinline__ bool agg_tile(const EngineView& v, int t, int* inst, int* first) {
  for (int i = 0; i < v.M; ++i) {
    const int n = v.inst[i].coarse ? (v.inst[i].cn + kAggTile - 1) / kAggTile : 0;
    if (t < n) {
      *inst = i;
      *first = t * kAggTile;
      return true;
    }
    t -= n;
  }
  return false;
}

// warp per aggregate
template <typename P>
__global__ void __launch_bounds__(kBlock) k_coarse_restrict(EngineView v, int which) {
  const int lane = threadIdx.x & 31;
  int inst, first;
  for (int t = blockIdx.x; agg_tile(v, t, &inst, &first); t += gridDim.x) {
    const KParams& k = v.inst[inst];
    if (!coarse_active(k, which == 2 ? 0 : which)) continue;
    if (which == 2 && !deflating<P>(k)) continue;  // the deflated solve's final correction only
    const P* r = VecSel<P>::rin(k);
    const int I = first + (threadIdx.x >> 5);
    if (I < k.cn) {
      const int ax = I % k.cna0, ay = (I / k.cna0) % k.cna1, az = I / (k.cna0 * k.cna1);
      const int bx0 = ax * k.cf, bx1 = min(bx0 + k.cf, k.nb0);
      float acc = 0.0f;
      for (int bz = az * k.cf; bz < min(az * k.cf + k.cf, k.nb2); ++bz)
        for (int by = ay * k.cf; by < min(ay * k.cf + k.cf, k.nb1); ++by) {
          // the aggregate's bins along x are one contiguous node range
          const int b0 = bx0 + k.nb0 * (by + k.nb1 * bz);
          const int i0 = k.bin_start[b0], i1 = k.bin_start[b0 + (bx1 - bx0)];
          for (int i = i0 + lane; i < i1; i += 32) acc += (float)r[i];
        }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
      if (lane == 0) k.rc[I] = acc;
    }
  }
}

// The CG update of the split (two-level) iteration fused with the restriction: e += alpha p,
// r -= alpha q on the unknowns, with a warp per aggregate walking its bins' node ranges, so
// that the new residual is summed into r_c[I] as it is written, with the aggregate's parts
// of r.D^-1 r and r.r.
template <typename P>
__global__ void __launch_bounds__(kBlock) k_cg_update_restrict(EngineView v) {
  __shared__ int2 s_runs[kBlock / 32][32];
  const int lane = threadIdx.x & 31;
  int inst, first;
  for (int t = blockIdx.x; agg_tile(v, t, &inst, &first); t += gridDim.x) {
    const KParams& k = v.inst[inst];
    if (!coarse_active(k, 1)) continue;
    P* rin = VecSel<P>::rin(k);
    const P* p = VecSel<P>::p(k);
    const P* q = VecSel<P>::q(k);
    P* e = VecSel<P>::e(k);
    const P* dinv = VecSel<P>::dinv(k);
    const P alpha = (P)k.ds->alpha;
    const bool def = deflating<P>(k);
    const int I = first + (threadIdx.x >> 5);
    if (I < k.cn) {
      const int ax = I % k.cna0, ay = (I / k.cna0) % k.cna1, az = I / (k.cna0 * k.cna1);
      const int bx0 = ax * k.cf, bx1 = min(bx0 + k.cf, k.nb0);
      if (def) {
        // deflated iteration: restrict q = A p (the update follows the coarse product)
        float acc = 0.0f;
        const int y0 = ay * k.cf, ny = min(y0 + k.cf, k.nb1) - y0;
        const int z0 = az * k.cf, nr = ny * (min(z0 + k.cf, k.nb2) - z0);
        if (nr <= 32) {
          // the aggregate's runs (cf bins along x each): their bounds loaded one run a lane,
          // then the warp walks the runs' concatenation, eight elements a lane in flight
          int lo = 0, len = 0;
          if (lane < nr) {
            const int b0 = bx0 + k.nb0 * ((y0 + lane % ny) + k.nb1 * (z0 + lane / ny));
            lo = k.bin_start[b0];
            len = k.bin_start[b0 + (bx1 - bx0)] - lo;
          }
          int pre = len;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, pre, off);
            if (lane >= off) pre += t;
          }
          const int total = __shfl_sync(0xffffffffu, pre, 31);
          int2* runs = s_runs[(threadIdx.x >> 5)];
          __syncwarp();
          if (lane < nr) runs[lane] = make_int2(pre - len, lo);  // (first position, first node)
          __syncwarp();
          for (int base = 0; base < total; base += 32 * 8) {
            P qv[8], dv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int idx = base + lane + 32 * u;
              qv[u] = dv[u] = P(0);
              if (idx < total) {
                int node = 0;
                for (int r = 0; r < nr; ++r) {
                  const int2 ru = runs[r];
                  if (idx >= ru.x) node = ru.y + (idx - ru.x);
                }
                dv[u] = dinv[node];
                qv[u] = q[node];
              }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) acc += (float)(dv[u] != P(0) ? qv[u] : P(0));
          }
        } else {
          for (int bz = z0; bz < min(z0 + k.cf, k.nb2); ++bz)
            for (int by = y0; by < y0 + ny; ++by) {
              const int b0 = bx0 + k.nb0 * (by + k.nb1 * bz);
              const int i0 = k.bin_start[b0], i1 = k.bin_start[b0 + (bx1 - bx0)];
              for (int i = i0 + lane; i < i1; i += 32) acc += (float)(dinv[i] != P(0) ? q[i] : P(0));
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) k.rc[I] = acc;
        continue;
      }
      float acc = 0.0f;
      DotAcc<P> rzf, rr;  // r.D^-1 r and r.r of the aggregate's nodes
      for (int bz = az * k.cf; bz < min(az * k.cf + k.cf, k.nb2); ++bz)
        for (int by = ay * k.cf; by < min(ay * k.cf + k.cf, k.nb1); ++by) {
          // the aggregate's bins along x are one contiguous node range
          const int b0 = bx0 + k.nb0 * (by + k.nb1 * bz);
          const int i0 = k.bin_start[b0], i1 = k.bin_start[b0 + (bx1 - bx0)];
          // two nodes per lane per round (their loads in flight together), summed in order
          for (int i = i0 + lane; i < i1; i += 64) {
            const bool two = i + 32 < i1;
            P r0 = rin[i], r1 = two ? rin[i + 32] : P(0);
            const P d0 = dinv[i], d1 = two ? dinv[i + 32] : P(0);
            const P p0 = p[i], p1 = two ? p[i + 32] : P(0);
            const P q0 = q[i], q1 = two ? q[i + 32] : P(0);
            const P e0 = e[i], e1 = two ? e[i + 32] : P(0);
            if (d0 != P(0)) {
              e[i] = e0 + alpha * p0;
              r0 = r0 - alpha * q0;
              rin[i] = r0;
              rzf.add(r0, r0 * d0);
              rr.add(r0, r0);
            }
            acc += (float)r0;
            if (d1 != P(0)) {
              e[i + 32] = e1 + alpha * p1;
              r1 = r1 - alpha * q1;
              rin[i + 32] = r1;
              rzf.add(r1, r1 * d1);
              rr.add(r1, r1);
            }
            acc += (float)r1;
          }
        }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
      rzf.warp_sum();
      rr.warp_sum();
      if (lane == 0) {
        k.rc[I] = acc;
        k.cdots[I] = rzf.value();
        k.cdots[k.cn + I] = rr.value();
      }
    }
  }
}

// warp per row of an instance's inverse: x_c = A_c^-1 r_c (r_c in shared memory, 16-byte
// row loads, four accumulators combined in a fixed order).  With dots (the CG update of the
// split iteration), also r_c[I] x_c[I] = (P^T r).(x_c) per row, and the last CTA forms
// r.z = r.D^-1 r + r_c.x_c and r.r from the per-aggregate parts and makes the CG decisions.
// 16-byte loads per lane in flight (8 x 32 x 4 = 1024 floats a round); with at most 80
// registers three CTAs fit an SM, so the 343 CTAs of the 512k workload run in one wave
constexpr int kGemvU = 8;
__global__ void __launch_bounds__(kBlock, 3) k_coarse_gemv(EngineView v, int which, cudaGraphConditionalHandle hc,
                                                        int dots, int def_mixed) {
  extern __shared__ __align__(16) float srv[];
  __shared__ double sm[3 * kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31;
  int inst, first;
  for (int t = blockIdx.x; agg_tile(v, t, &inst, &first); t += gridDim.x) {
    const KParams& k = v.inst[inst];
    if (!coarse_active(k, which == 2 ? 0 : which)) continue;
    if (which == 2 && !deflating<float>(k)) continue;  // the deflated solve's final correction only
    const int n = k.cn, ld = k.cld;
    const bool dm = def_mixed && k.defl_ok && *((volatile const int*)&k.ds->defl) != 0;
    __syncthreads();
    {
      // r_c into shared memory: 16-byte loads, four per thread in flight (rc holds ld
      // floats, its padding zero)
      const float4* rc4 = reinterpret_cast<const float4*>(k.rc);
      float4* sv4 = reinterpret_cast<float4*>(srv);
      const int nq = ld >> 2;
      for (int i0 = threadIdx.x; i0 < nq; i0 += 4 * kBlock) {
        float4 t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 + u * kBlock < nq) t[u] = rc4[i0 + u * kBlock];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 + u * kBlock < nq) sv4[i0 + u * kBlock] = t[u];
      }
    }
    __syncthreads();
    const float4* sr4 = reinterpret_cast<const float4*>(srv);
    const int nq = ld >> 2;  // 16-byte groups per row
    const int I = first + (threadIdx.x >> 5);
    if (I < n) {
      const float4* row = reinterpret_cast<const float4*>(k.cinv + (size_t)I * ld);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      // rounds of kGemvU 16-byte loads per lane, all in flight before their products
      for (int j0 = lane; j0 < nq; j0 += 32 * kGemvU) {
        float4 a[kGemvU];
#pragma unroll
        for (int u = 0; u < kGemvU; ++u)
          if (j0 + 32 * u < nq) a[u] = __ldg(row + j0 + 32 * u);
#pragma unroll
        for (int u = 0; u < kGemvU; ++u)
          if (j0 + 32 * u < nq) {
            const float4 b = sr4[j0 + 32 * u];
            acc[0] = fmaf(a[u].x, b.x, acc[0]);
            acc[1] = fmaf(a[u].y, b.y, acc[1]);
            acc[2] = fmaf(a[u].z, b.z, acc[2]);
            acc[3] = fmaf(a[u].w, b.w, acc[3]);
          }
      }
      float x = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
      if (lane == 0) {
        k.xc[I] = x;
        if (dots) {
          if (dm) {
            // deflated (FP32 path): r_c[I] x_c[I] as an exact FP32 pair
            const float pr = srv[I] * x;
            store_pair(k.cdots, 2 * (size_t)n + I, pr, fmaf(srv[I], x, -pr));
          } else {
            k.cdots[2 * n + I] = (double)srv[I] * (double)x;
          }
        }
      }
    }
  }
  if (!dots) return;
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      const KParams& k = v.inst[i];
      double tot[3] = {0.0, 0.0, 0.0};
      // the deflated iteration needs only r_c.x_c (the update kernel forms the dots)
      const bool dm = def_mixed && k.coarse && k.defl_ok && *((volatile const int*)&k.ds->defl) != 0;
      if (dm) {
        double t2[1];
        reduce_pair_items<1>(k.cdots + 2 * (size_t)k.cn, k.cn, 0, k.cn, t2, sm);
        tot[2] = t2[0];
      } else if (k.coarse) {
        reduce_items<3>(k.cdots, k.cn, 0, k.cn, tot, sm);
      }
      if (threadIdx.x == 0) {
        DevState* ds = k.ds;
        if (dm) {
          // deflated step length: p.P_d A p = p.q - r_c.x_c (r_c = P^T q); the update kernel
          // makes the decisions and drives the loop
          if (ds->inner_active) {
            const double pw = ds->pq - tot[2];
            ds->alpha = (pw > 0.0 && isfinite(pw)) ? ds->rz / pw : 0.0;
          }
        } else {
          if (!k.coarse) {
            ds->inner_active = 0;  // not reached: split engines have a coarse space per member
          } else if (ds->inner_active) {
            const double rz = tot[0] + tot[2];
            const double alpha_d = ds->alpha;
            ds->beta = ds->rz != 0.0 ? rz / ds->rz : 0.0;
            ds->rz = rz;
            ds->rr = tot[1];
            ds->inner_it += 1;
            ds->solve_iters += 1;
            ds->cg_iters += 1;
            const bool go = alpha_d != 0.0 && isfinite(tot[1]) && tot[1] > ds->inner_target &&
                            ds->inner_it < ds->max_iter && ds->solve_iters < ds->max_iter;
            ds->inner_active = go ? 1 : 0;
          }
          instance_finished(v, i, 1, hc);
        }
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// Additive form: z = D^-1 r + x_c[agg] on the unknowns (after the decisions of
// k_coarse_gemv).  Deflated form: w = q - A P x_c, e^ += alpha p, r^ -= alpha w, t += alpha q,
// z = D^-1 r^, with the dots and the CG decisions (last chunk of the instance).
template <typename P>
__global__ void __launch_bounds__(kBlock) k_z_form(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ double sm[2 * kBlock / 32];
  __shared__ int s_last;
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const bool active = coarse_active(k, 1);
    P* rin = VecSel<P>::rin(k);
    P* z = VecSel<P>::z(k);
    const P* dinv = VecSel<P>::dinv(k);
    if (!deflating<P>(k)) {
      if (!active) continue;
      for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
        const P di = dinv[a];
        z[a] = di == P(0) ? P(0) : rin[a] * di + (P)k.xc[k.agg[a]];
      }
      continue;
    }
    DotAcc<float> part[2];
    if constexpr (sizeof(P) == 4) {
      if (active) {
        const float* p = k.p32;
        const float* q = k.q32;
        float* e = k.e32;
        float* t = k.t32;
        const float alpha = (float)k.ds->alpha;
        for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
          const float di = dinv[a];
          if (di == 0.0f) continue;
          // every load before the first store (loads are not moved across the stores)
          const float qa = __ldg(q + a);
          const float pa = __ldg(p + a);
          const float ea = e[a];
          const float ra = rin[a];
          const float ta = t[a];
          const float w = qa - ap_apply(k, a, k.xc);
          e[a] = ea + alpha * pa;
          const float r = ra - alpha * w;
          rin[a] = r;
          t[a] = ta + alpha * qa;
          const float zz = r * di;
          z[a] = zz;
          part[0].add(r, zz);
          part[1].add(r, r);
        }
      }
    }
    write_dot_partials<2, float>(v, item, part, sm);
    if (item_done(&v.ticket[c.inst], v.chunk_count[c.inst], &s_last)) {
      double tot[2];
      reduce_dot_items<2, float>(v.partials, v.stride, v.chunk_first[c.inst], v.chunk_count[c.inst], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = k.ds;
        if (ds->inner_active) {
          const double alpha_d = ds->alpha;
          ds->beta = ds->rz != 0.0 ? tot[0] / ds->rz : 0.0;
          ds->rz = tot[0];
          ds->rr = tot[1];
          ds->inner_it += 1;
          ds->solve_iters += 1;
          ds->cg_iters += 1;
          const bool go = alpha_d != 0.0 && isfinite(tot[1]) && tot[1] > ds->inner_target &&
                          ds->inner_it < ds->max_iter && ds->solve_iters < ds->max_iter;
          ds->inner_active = go ? 1 : 0;
        }
        instance_finished(v, c.inst, 1, hc);
      }
    }
    __syncthreads();
  }
}

// Deflated solve, after the inner loop: e = e^ + Q (r0 - t).  Step 1 writes r0 - t into r
// (restricted and solved next), step 2 adds P x_c.
__global__ void __launch_bounds__(kBlock) k_def_final(EngineView v, int step) {
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    if (!deflating<float>(k) || !coarse_active(k, 0)) continue;
    for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
      const bool unk = k.dinv32[a] != 0.0f;
      if (step == 1)
        k.rin32[a] = unk ? k.r0_32[a] - k.t32[a] : 0.0f;
      else if (unk)
        k.e32[a] = k.e32[a] + k.xc[k.agg[a]];
    }
  }
}

template <typename P>
__global__ void __launch_bounds__(kBlock) k_cg_zdots(EngineView v, cudaGraphConditionalHandle hc, int init,
                                                     int fp64) {
  __shared__ double sm[3 * kBlock / 32];
  __shared__ int s_last;
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const bool active = coarse_active(k, init ? 0 : 1);
    DotAcc<P> part[3];
    if (active) {
      P* rin = VecSel<P>::rin(k);
      P* z = VecSel<P>::z(k);
      const P* dinv = VecSel<P>::dinv(k);
      // deflated start (mixed, operator fresh): r^ = r - A P x_c, z = D^-1 r^
      const bool def = init && deflating<P>(k);
      for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
        const P di = dinv[a];
        P r = rin[a];
        part[2].add(r, r);
        P zz;
        if (def) {
          if (di != P(0)) {
            r = r - (P)ap_apply(k, a, k.xc);
            rin[a] = r;
          }
          zz = r * di;
        } else {
          zz = di == P(0) ? P(0) : (k.coarse ? r * di + (P)k.xc[k.agg[a]] : r * di);
        }
        z[a] = zz;
        part[0].add(r, zz);
        part[1].add(r, r);
      }
    }
    write_dot_partials<3, P>(v, item, part, sm);
    if (item_done(&v.ticket[c.inst], v.chunk_count[c.inst], &s_last)) {
      double tot[3];
      reduce_dot_items<3, P>(v.partials, v.stride, v.chunk_first[c.inst], v.chunk_count[c.inst], tot, sm);
      if (threadIdx.x == 0) {
        DevState* ds = k.ds;
        if (init) {
          if (ds->outer_active) {
            ds->rz = tot[0];
            ds->rr = tot[1];
            ds->beta = 0.0;
            ds->alpha = 0.0;
            ds->inner_it = 0;
            // the reduction is relative to the correction equation's residual r (before
            // the deflation), the stop test on the (deflated) iterated residual
            const double target = fp64 ? 0.25 * ds->tol * ds->tol * ds->bnorm2
                                       : fmax(ds->inner_rel * ds->inner_rel * tot[2],
                                              0.09 * ds->tol * ds->tol * ds->bnorm2);
            ds->inner_target = target;
            ds->inner_active = (tot[1] > target && ds->max_iter > 0) ? 1 : 0;
          } else {
            ds->inner_active = 0;
          }
        } else if (ds->inner_active) {
          const double alpha_d = ds->alpha;
          ds->beta = ds->rz != 0.0 ? tot[0] / ds->rz : 0.0;
          ds->rz = tot[0];
          ds->rr = tot[1];
          ds->inner_it += 1;
          ds->solve_iters += 1;
          ds->cg_iters += 1;
          const bool go = alpha_d != 0.0 && isfinite(tot[1]) && tot[1] > ds->inner_target &&
                          ds->inner_it < ds->max_iter && ds->solve_iters < ds->max_iter;
          ds->inner_active = go ? 1 : 0;
        }
        instance_finished(v, c.inst, 1, hc);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------- the inner solve in one launch ---
// One refinement sweep's correction solve of a single instance with the two-level preconditioner,
// start to end, in one cooperative launch: the CG's right-hand side and first z, every iteration, and
// the deflated form's final correction (the same steps as the kernels above, which ensembles, the
// Jacobi preconditioner and the other operators take).  An iteration has four passes -- operator,
// restriction, coarse product, update -- of a few us each up to a few hundred thousand nodes, so as
// launches they are bound by the gaps, the ramps and the last CTAs' reductions; here a CTA an SM stays
// for the whole solve and meets the others between passes.  The dots are block partials that every
// CTA sums again in the same order after it has met the others, so each takes the loop's decisions
// itself, with the same bits.  A meeting takes 1.3 us, one that sums two values 3 to 4 (its chain of
// FP64 instructions, 64 cycles each, is what was left of 10: hence the FP32 pairs, the values side by
// side and the division while waiting).  A step, this against the launches (ms): 8k nodes 0.251 against
// 0.358 mixed and 0.304 against 0.402 FP64, 64k 0.471 against 0.628, 262k 1.27 against 1.60, 512k 2.42
// against 2.71 and 7.05 against 7.43, 2M 18.2 against 21.2.
// NW: warps a CTA, see k_cg_sweep.
template <typename P>
struct SweepState {
  P alpha_p, beta_p;              // alpha and beta as the passes use them
  double alpha, beta, rz, rr, pq, target;
  double irz;                     // 1 / rz
  double tol, inner_rel, bnorm2;  // the solve's settings
  int it, solve_it, go, max_iter;
};

// The sums' parts: FP64, or FP32 pairs on the FP32 path (an FP64 instruction holds the pipe for 64 cycles,
// and the chain of a reduction is what a meeting waits for)
template <typename P>
struct SweepSum;
template <>
struct SweepSum<double> {
  double s;
  __device__ __forceinline__ void add(const SweepSum& o) { s += o.s; }
  __device__ __forceinline__ void shfl_add(int off) { s += __shfl_xor_sync(0xffffffffu, s, off); }
  __device__ __forceinline__ double value() const { return s; }
  __device__ __forceinline__ static SweepSum of(const DotAcc<double>& d) { return {d.s}; }
  __device__ __forceinline__ static SweepSum of(double d) { return {d}; }
};
template <>
struct SweepSum<float> {
  float hi, lo;
  __device__ __forceinline__ void add(const SweepSum& o) { pair_add(hi, lo, o.hi, o.lo); }
  __device__ __forceinline__ void shfl_add(int off) {
    const float h = __shfl_xor_sync(0xffffffffu, hi, off), l = __shfl_xor_sync(0xffffffffu, lo, off);
    pair_add(hi, lo, h, l);
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
  __device__ __forceinline__ static SweepSum of(const DotAcc<float>& d) { return {d.hi, d.lo}; }
};
template <typename P>
__device__ __forceinline__ SweepSum<P> sweep_load(const double* p) {
  const double d = __ldcg(p);
  if constexpr (sizeof(P) == 8) {
    return {d};
  } else {
    const long long b = __double_as_longlong(d);
    return {__int_as_float((int)(b & 0xffffffffll)), __int_as_float((int)(b >> 32))};
  }
}
template <typename P>
__device__ __forceinline__ void sweep_store(double* p, const SweepSum<P>& x) {
  if constexpr (sizeof(P) == 8)
    __stcg(p, x.s);
  else
    __stcg(p, __longlong_as_double((long long)((unsigned long long)(unsigned)__float_as_int(x.lo) << 32 |
                                               (unsigned)__float_as_int(x.hi))));
}
// comparisons by the bits (an FP64 comparison takes the FP64 pipe)
__device__ __forceinline__ bool sweep_finite(double x) {
  return ((__double_as_longlong(x) >> 52) & 0x7ff) != 0x7ff;
}
__device__ __forceinline__ bool sweep_nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }
// x > 0, finite or infinite (a NaN fails sweep_finite, which goes with it)
__device__ __forceinline__ bool sweep_positive(double x) { return __double_as_longlong(x) > 0; }
// a > b for finite a and b >= 0
__device__ __forceinline__ bool sweep_above(double a, double b) { return __double_as_longlong(a) > __double_as_longlong(b); }

template <int NW, typename P>
struct SweepSmem {
  SweepSum<P> red[3 * NW];
  SweepState<P> st;
  int fail;
  int hb[NW][12];       // gather bases of the warp's slice
  int off[NW], nq[NW];  // the planned slice: quad offset base and quads (0: none)
  int2 runs[NW][32];
};
// A pass, inlined with 16 warps a CTA (128 registers), a function of its own with 32 (64 registers: one
// body with all of them spills)
#define NNPP_SWEEP_PASS(name, ...) (NW <= 16 ? name<__VA_ARGS__> : name##_fn<__VA_ARGS__>)

// Every CTA of the launch meets here: what the others wrote before is visible after.  The warps' sums
// of NV values (part, lane 0) come back as totals in decide(tot), which thread 0 runs before the CTA
// goes on; waiting() is its work while the others come.  partials has two halves, used in turn (half): a CTA can be a meeting ahead of the last
// one's reads, not two.  False when the wait gave up.
template <int NV, int NW, typename P, typename F, typename H>
__device__ __forceinline__ bool sweep_meet(const EngineView& v, SweepSmem<NW, P>& sm, unsigned int& target, int& half,
                                           const SweepSum<P> (&part)[NV > 0 ? NV : 1], F&& decide, H&& waiting) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (NV > 0 && lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) sm.red[q * NW + warp] = part[q];
  __syncthreads();
  if (warp == 0) {
    // two values: half a warp each, so that their chains run at once
    constexpr int kSeg = NV == 2 ? 16 : 32, kRounds = NV == 2 ? 1 : NV;
    const int sub = lane % kSeg, G = gridDim.x;
    double* buf = v.partials + (size_t)half * 3 * G;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int q = NV == 2 ? lane / 16 : r;
      SweepSum<P> x{};
#pragma unroll
      for (int w = 0; w < NW; w += kSeg)
        if (w + sub < NW) x.add(sm.red[q * NW + w + sub]);
#pragma unroll
      for (int off = kSeg / 2; off > 0; off >>= 1) x.shfl_add(off);
      if (sub == 0) sweep_store<P>(buf + q * G + blockIdx.x, x);
    }
    unsigned int* count = v.ticket + v.M + 4;
    target += G;
    int ok = 1;
    __syncwarp();
    if (lane == 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      waiting();
      unsigned int seen, polls = 0;
      do {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
      } while ((int)(seen - target) < 0 && ++polls < kWaitPolls);
      ok = (int)(seen - target) >= 0 ? 1 : 0;
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    double tot[NV > 0 ? NV : 1];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int q = NV == 2 ? lane / 16 : r;
      constexpr int kU = 160 / kSeg;  // a lane's parts all in flight (160 CTAs a round)
      SweepSum<P> x{};
      for (int i0 = sub; i0 < G; i0 += 160) {
        SweepSum<P> y[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          y[u] = SweepSum<P>{};
          if (i0 + kSeg * u < G) y[u] = sweep_load<P>(buf + q * G + i0 + kSeg * u);
        }
#pragma unroll
        for (int d = 1; d < kU; d *= 2)
#pragma unroll
          for (int u = 0; u + d < kU; u += 2 * d) y[u].add(y[u + d]);
        x.add(y[0]);
      }
#pragma unroll
      for (int off = kSeg / 2; off > 0; off >>= 1) x.shfl_add(off);
      const double t = x.value();
      if (NV == 2) {
        tot[0] = __shfl_sync(0xffffffffu, t, 0);
        tot[NV - 1] = __shfl_sync(0xffffffffu, t, 16);
      } else {
        tot[r] = t;
      }
    }
    if (lane == 0) {
      sm.fail = ok ? 0 : 1;
      decide(tot);
    }
  }
  half ^= 1;
  __syncthreads();
  return sm.fail == 0;
}

// The warp walks an aggregate's nodes: f(nodes) with U nodes a lane (-1: none), in a fixed order.  The
// aggregate's bins along x are one contiguous node range; their bounds are loaded one run a lane and
// the warp walks the runs' concatenation.
template <int U, typename F>
__device__ __forceinline__ void walk_aggregate(const KParams& k, int I, int lane, int2* runs, F&& f) {
  const int ax = I % k.cna0, ay = (I / k.cna0) % k.cna1, az = I / (k.cna0 * k.cna1);
  const int bx0 = ax * k.cf, nx = min(bx0 + k.cf, k.nb0) - bx0;
  const int y0 = ay * k.cf, ny = min(y0 + k.cf, k.nb1) - y0;
  const int z0 = az * k.cf, rows = ny * (min(z0 + k.cf, k.nb2) - z0);
#pragma unroll 1
  for (int g = 0; g < rows; g += 32) {
    const int nr = min(32, rows - g);
    int lo = 0, len = 0;
    if (lane < nr) {
      const int b0 = bx0 + k.nb0 * ((y0 + (g + lane) % ny) + k.nb1 * (z0 + (g + lane) / ny));
      lo = __ldg(k.bin_start + b0);
      len = __ldg(k.bin_start + b0 + nx) - lo;
    }
    int pre = len;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pre, off);
      if (lane >= off) pre += t;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    __syncwarp();
    if (lane < nr) runs[lane] = make_int2(pre - len, lo);  // (first position, first node)
    __syncwarp();
#pragma unroll 1
    for (int base = 0; base < total; base += 32 * U) {
      int node[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = base + lane + 32 * u;
        node[u] = -1;
        if (idx < total)
#pragma unroll 1
          for (int r = 0; r < nr; ++r) {
            const int2 ru = runs[r];
            if (idx >= ru.x) node[u] = ru.y + (idx - ru.x);
          }
      }
      f(node);
    }
  }
}

// x_c = A_c^-1 r_c, a warp a row; the warp's sum of r_c[I] x_c[I] (lane 0)
template <typename P, int NW>
__device__ __forceinline__ SweepSum<P> sweep_coarse(const KParams& k, float* srv) {
  const int lane = threadIdx.x & 31;
  const int nq = k.cld >> 2;
  float4* sv4 = reinterpret_cast<float4*>(srv);
  for (int i = threadIdx.x; i < nq; i += 32 * NW) sv4[i] = reinterpret_cast<const float4*>(k.rc)[i];
  __syncthreads();
  constexpr int kU = NW <= 16 ? kGemvU : kGemvU / 2;
  DotAcc<P> dot;
#pragma unroll 1
  for (int I = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; I < k.cn; I += gridDim.x * NW) {
    const float4* row = reinterpret_cast<const float4*>(k.cinv + (size_t)I * k.cld);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int j0 = lane; j0 < nq; j0 += 32 * kU) {
      float4 a[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (j0 + 32 * u < nq) a[u] = __ldg(row + j0 + 32 * u);
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (j0 + 32 * u < nq) {
          const float4 b = sv4[j0 + 32 * u];
          acc[0] = fmaf(a[u].x, b.x, acc[0]);
          acc[1] = fmaf(a[u].y, b.y, acc[1]);
          acc[2] = fmaf(a[u].z, b.z, acc[2]);
          acc[3] = fmaf(a[u].w, b.w, acc[3]);
        }
    }
    float x = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if (lane == 0) {
      k.xc[I] = x;
      dot.add(srv[I], x);
    }
  }
  return SweepSum<P>::of(dot);
}

// A part of a slice's row sums: sum of w x[node] over the quads part, part + K, ..., QB quads a batch, the
// next batch's loads in flight
template <int K, int QB>
__device__ __forceinline__ float sweep_row(const KParams& k, int off, int nq, int lane, int part, const int* hb,
                                           bool live) {
  const QuadPtr op(k.sell_cg + (size_t)(off >> 5) * kSellW, lane);
  const float* z = k.z32;
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  float4 w[QB];
  uint2 code[QB];
  auto load = [&](int q0) {
#pragma unroll
    for (int u = 0; u < QB; ++u) {
      w[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      code[u] = make_uint2(0u, 0u);
      if (q0 + u * K < nq) {
        w[u] = op.weights(q0 + u * K);
        code[u] = op.codes(q0 + u * K);
      }
    }
  };
  if (!live) return 0.0f;
  load(part);
#pragma unroll 1
  for (int q0 = part; q0 < nq; q0 += QB * K) {
    float zv[4 * QB];
#pragma unroll
    for (int u = 0; u < 4 * QB; ++u) zv[u] = z[code_node(hb, quad_code(code[u >> 2], u & 3))];
    float4 wc[QB];
#pragma unroll
    for (int u = 0; u < QB; ++u) wc[u] = w[u];
    if (q0 + QB * K < nq) load(q0 + QB * K);
#pragma unroll
    for (int u = 0; u < 4 * QB; ++u) acc[u & 3] = fmaf(quad_weight(wc[u >> 2], u & 3), zv[u], acc[u & 3]);
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}
template <int K>
__device__ __forceinline__ double sweep_row64(const KParams& k, int off, int nq, int lane, int part, const int* hb,
                                              bool live) {
  return live ? cg_row64<K, false>(k, off, nq, lane, part, hb, k.z64) : 0.0;
}

// q = A z + beta q, p = z + beta p on a slice that K warps share (lane's row a, -1: none); adds p.q.  Every
// warp of the CTA calls it.  EARLY: the row's own values are loaded before its sum (four registers
// more; a slice's chain of loads is shorter).
template <bool EARLY, typename P, int K, int NW>
__device__ __forceinline__ void sweep_slice(const KParams& k, SweepSmem<NW, P>& sm, P* s_acc, int off, int nq, int a, P beta,
                                            DotAcc<P>& dot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % K;
  const bool live = a >= 0, owner = live && part == 0;
  P *p = VecSel<P>::p(k), *q = VecSel<P>::q(k);
  P za = P(0), da = P(0), qa = P(0), pa = P(0);
  auto own = [&] {
    za = VecSel<P>::z(k)[a];
    da = __ldg(VecSel<P>::d(k) + a);
    qa = q[a];
    pa = p[a];
  };
  if (EARLY && owner) own();
  P sum;
  if constexpr (sizeof(P) == 4)
    sum = sweep_row<K, EARLY && NW <= 16 ? 4 : 2>(k, off, nq, lane, part, sm.hb[warp], live);
  else
    sum = sweep_row64<K>(k, off, nq, lane, part, sm.hb[warp], live);
  if (K > 1) {
    if (part) s_acc[threadIdx.x] = sum;
    __syncthreads();
    if (!part)
#pragma unroll
      for (int h = 1; h < K; ++h) sum += s_acc[threadIdx.x + 32 * h];
  }
  if (owner) {
    if (!EARLY) own();
    const P qn = da * za - sum + beta * qa;
    const P pn = za + beta * pa;
    q[a] = qn;
    p[a] = pn;
    dot.add(pn, qn);
  }
  if (K > 1)
    __syncthreads();
  else
    __syncwarp();
}

// The slice's gather bases into the warp's table; the lane's row (-1: not an unknown) and the slice's place
template <typename P, int NW>
__device__ __forceinline__ int sweep_take(const KParams& k, SweepSmem<NW, P>& sm, const SliceDesc* slices, int sg, int* off,
                                          int* nq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SliceDesc& d = slices[sg];
  const int row0 = __ldg(&d.row0), width = __ldg(k.cg_width + sg);
  *off = __ldg(&d.off);
  *nq = (width + 3) >> 2;
  if (lane < 9) sm.hb[warp][lane] = __ldg(&d.gbase[lane]);
  __syncwarp();
  const int a = __ldg(k.cg_rows + row0 + lane);
  return a >= 0 && __ldg(k.freem + a) ? a : -1;
}

// the slices [s0, s1), K warps each
template <typename P, int K, int NW>
__device__ __forceinline__ SweepSum<P> sweep_slices(const KParams& k, SweepSmem<NW, P>& sm, P* s_acc, const SliceDesc* slices,
                                               int s0, int s1, P beta) {
  constexpr int kGroup = NW / K;  // slices of a CTA at a time
  DotAcc<P> dot;
#pragma unroll 1
  for (int base = s0 + blockIdx.x * kGroup; base < s1; base += gridDim.x * kGroup) {
    const int sg = base + (threadIdx.x >> 5) / K;
    int off = 0, nq = 0, a = -1;
    if (sg < s1) a = sweep_take<P, NW>(k, sm, slices, sg, &off, &nq);
    sweep_slice<false, P, K>(k, sm, s_acc, off, nq, a, beta, dot);
  }
  dot.warp_sum();
  return SweepSum<P>::of(dot);
}
template <typename P, int K, int NW>
__device__ __noinline__ SweepSum<P> sweep_slices_fn(const KParams& k, SweepSmem<NW, P>& sm, P* s_acc, const SliceDesc* slices,
                                               int s0, int s1, P beta) {
  return sweep_slices<P, K, NW>(k, sm, s_acc, slices, s0, s1, beta);
}

// the passes of the solve
__device__ __forceinline__ int sweep_agg0() { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }  // one an SM first
__device__ __forceinline__ int sweep_aggs() { return gridDim.x * (blockDim.x >> 5); }
__device__ __forceinline__ int sweep_node0() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int sweep_nodes() { return gridDim.x * blockDim.x; }
// x_c into shared memory (after the coarse product's meeting)
__device__ __forceinline__ void sweep_stage(const KParams& k, float* srv) {
  for (int i = threadIdx.x; i < k.cn; i += blockDim.x) srv[i] = k.xc[i];
  __syncthreads();
}
__device__ __forceinline__ void sweep_store_rc(const KParams& k, int I, float acc) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) k.rc[I] = acc;
}

// the right-hand side and its restriction
template <typename P, int NW>
__device__ __forceinline__ void sweep_rhs(const KParams& k, SweepSmem<NW, P>& sm) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int I = sweep_agg0(); I < k.cn; I += sweep_aggs()) {
    float acc = 0.0f;
    walk_aggregate<4>(k, I, lane, sm.runs[threadIdx.x >> 5], [&](const int (&node)[4]) {
      P* rin = VecSel<P>::rin(k);
      P* p = VecSel<P>::p(k);
      P* q = VecSel<P>::q(k);
      P* e = VecSel<P>::e(k);
      double r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) r[u] = node[u] >= 0 ? k.r64[node[u]] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (node[u] >= 0) {
          const int a = node[u];
          rin[a] = (P)r[u];
          p[a] = q[a] = e[a] = P(0);
          if (sizeof(P) == 4) {  // the deflated solve's right-hand side and t = A e^
            k.r0_32[a] = (float)r[u];
            k.t32[a] = 0.0f;
          }
          acc += (float)(P)r[u];
        }
    });
    sweep_store_rc(k, I, acc);
  }
}

// z = M^-1 r; deflated: r^ = r - A P x_c, z = D^-1 r^.  The warp's r.z, r.r and the undeflated r.r
template <typename P>
struct Dots3 {
  SweepSum<P> rz, rr, r0;
};
template <typename P>
struct Dots2 {
  SweepSum<P> a, b;
};
template <typename P, int NW>
__device__ __forceinline__ Dots3<P> sweep_first_z(const KParams& k, float* srv, bool def) {
  sweep_stage(k, srv);
  P* rin = VecSel<P>::rin(k);
  P* z = VecSel<P>::z(k);
  const P* dinv = VecSel<P>::dinv(k);
  DotAcc<P> part[3];
#pragma unroll 1
  for (int a = sweep_node0(); a < k.N; a += sweep_nodes()) {
    const P di = dinv[a];
    P r = rin[a];
    part[2].add(r, r);
    P zz = P(0);
    if (di != P(0)) {
      if (def) {
        r = r - (P)ap_apply(k, a, srv);
        rin[a] = r;
        zz = r * di;
      } else {
        zz = r * di + (P)srv[__ldg(k.agg + a)];
      }
    }
    z[a] = zz;
    part[0].add(r, zz);
    part[1].add(r, r);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) part[i].warp_sum();
  return Dots3<P>{SweepSum<P>::of(part[0]), SweepSum<P>::of(part[1]), SweepSum<P>::of(part[2])};
}

// deflated iteration: r_c = P^T q (q is 0 off the unknowns)
template <int NW>
__device__ __forceinline__ void sweep_restrict_q(const KParams& k, SweepSmem<NW, float>& sm) {
  const int lane = threadIdx.x & 31;
  const float* q = k.q32;
#pragma unroll 1
  for (int I = sweep_agg0(); I < k.cn; I += sweep_aggs()) {
    float acc = 0.0f;
    walk_aggregate<8>(k, I, lane, sm.runs[threadIdx.x >> 5], [&](const int (&node)[8]) {
      float x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = node[u] >= 0 ? q[node[u]] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc += x[u];
    });
    sweep_store_rc(k, I, acc);
  }
}

// deflated iteration: w = q - A P x_c, e^ += alpha p, r^ -= alpha w, t += alpha q, z = D^-1 r^; the
// warp's r.z and r.r
template <int NW>
__device__ __forceinline__ Dots2<float> sweep_update(const KParams& k, float* srv, float alpha) {
  sweep_stage(k, srv);
  const float *dinv = k.dinv32, *q = k.q32, *p = k.p32;
  float *e = k.e32, *rin = k.rin32, *t = k.t32, *z = k.z32;
  DotAcc<float> rz, rr;
#pragma unroll 1
  for (int a = sweep_node0(); a < k.N; a += sweep_nodes()) {
    const float di = dinv[a];
    if (di == 0.0f) continue;
    const float qa = q[a], pa = p[a], ea = e[a], ra = rin[a], ta = t[a];
    const float w = qa - ap_apply(k, a, srv);
    e[a] = ea + alpha * pa;
    const float r = ra - alpha * w;
    rin[a] = r;
    t[a] = ta + alpha * qa;
    const float zz = r * di;
    z[a] = zz;
    rz.add(r, zz);
    rr.add(r, r);
  }
  rz.warp_sum();
  rr.warp_sum();
  return Dots2<float>{SweepSum<float>::of(rz), SweepSum<float>::of(rr)};
}

// additive iteration: e += alpha p, r -= alpha q with the restriction of r; the warp's r.D^-1 r and r.r
template <typename P, int NW>
__device__ __forceinline__ Dots2<P> sweep_update_restrict(const KParams& k, SweepSmem<NW, P>& sm, P alpha) {
  const int lane = threadIdx.x & 31;
  DotAcc<P> rzf, rr;
#pragma unroll 1
  for (int I = sweep_agg0(); I < k.cn; I += sweep_aggs()) {
    float acc = 0.0f;
    walk_aggregate<2>(k, I, lane, sm.runs[threadIdx.x >> 5], [&](const int (&node)[2]) {
      P* rin = VecSel<P>::rin(k);
      P* p = VecSel<P>::p(k);
      P* q = VecSel<P>::q(k);
      P* e = VecSel<P>::e(k);
      const P* dinv = VecSel<P>::dinv(k);
      P r[2], d[2], pv[2], qv[2], ev[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        r[u] = d[u] = pv[u] = qv[u] = ev[u] = P(0);
        if (node[u] >= 0) {
          r[u] = rin[node[u]];
          d[u] = dinv[node[u]];
          pv[u] = p[node[u]];
          qv[u] = q[node[u]];
          ev[u] = e[node[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (d[u] != P(0)) {
          e[node[u]] = ev[u] + alpha * pv[u];
          r[u] = r[u] - alpha * qv[u];
          rin[node[u]] = r[u];
          rzf.add(r[u], r[u] * d[u]);
          rr.add(r[u], r[u]);
        }
        acc += (float)r[u];
      }
    });
    sweep_store_rc(k, I, acc);
  }
  rzf.warp_sum();
  rr.warp_sum();
  return Dots2<P>{SweepSum<P>::of(rzf), SweepSum<P>::of(rr)};
}

// additive iteration: z = D^-1 r + P x_c
template <typename P, int NW>
__device__ __forceinline__ void sweep_z(const KParams& k, float* srv) {
  sweep_stage(k, srv);
  P* rin = VecSel<P>::rin(k);
  P* z = VecSel<P>::z(k);
  const P* dinv = VecSel<P>::dinv(k);
  for (int a = sweep_node0(); a < k.N; a += sweep_nodes()) {
    const P di = dinv[a];
    z[a] = di == P(0) ? P(0) : rin[a] * di + (P)srv[__ldg(k.agg + a)];
  }
}

// the deflated solve's end, e = e^ + Q (r0 - t): the restriction, then the correction
template <int NW>
__device__ __forceinline__ void sweep_last_restrict(const KParams& k, SweepSmem<NW, float>& sm) {
  const int lane = threadIdx.x & 31;
  const float *dinv = k.dinv32, *r0 = k.r0_32, *t = k.t32;
#pragma unroll 1
  for (int I = sweep_agg0(); I < k.cn; I += sweep_aggs()) {
    float acc = 0.0f;
    walk_aggregate<4>(k, I, lane, sm.runs[threadIdx.x >> 5], [&](const int (&node)[4]) {
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        x[u] = node[u] >= 0 && dinv[node[u]] != 0.0f ? r0[node[u]] - t[node[u]] : 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) acc += x[u];
    });
    sweep_store_rc(k, I, acc);
  }
}
template <int NW>
__device__ __forceinline__ void sweep_last_add(const KParams& k, float* srv) {
  sweep_stage(k, srv);
  const float* dinv = k.dinv32;
  float* e = k.e32;
  for (int a = sweep_node0(); a < k.N; a += sweep_nodes())
    if (dinv[a] != 0.0f) e[a] = e[a] + srv[__ldg(k.agg + a)];
}

// the same passes as functions (NNPP_SWEEP_PASS)
template <typename P, int NW>
__device__ __noinline__ SweepSum<P> sweep_coarse_fn(const KParams& k, float* srv) {
  return sweep_coarse<P, NW>(k, srv);
}
template <typename P, int NW>
__device__ __noinline__ void sweep_rhs_fn(const KParams& k, SweepSmem<NW, P>& sm) {
  sweep_rhs<P, NW>(k, sm);
}
template <typename P, int NW>
__device__ __noinline__ Dots3<P> sweep_first_z_fn(const KParams& k, float* srv, bool def) {
  return sweep_first_z<P, NW>(k, srv, def);
}
template <int NW>
__device__ __noinline__ void sweep_restrict_q_fn(const KParams& k, SweepSmem<NW, float>& sm) {
  sweep_restrict_q<NW>(k, sm);
}
template <int NW>
__device__ __noinline__ Dots2<float> sweep_update_fn(const KParams& k, float* srv, float alpha) {
  return sweep_update<NW>(k, srv, alpha);
}
template <typename P, int NW>
__device__ __noinline__ Dots2<P> sweep_update_restrict_fn(const KParams& k, SweepSmem<NW, P>& sm, P alpha) {
  return sweep_update_restrict<P, NW>(k, sm, alpha);
}
template <typename P, int NW>
__device__ __noinline__ void sweep_z_fn(const KParams& k, float* srv) {
  sweep_z<P, NW>(k, srv);
}
template <int NW>
__device__ __noinline__ void sweep_last_restrict_fn(const KParams& k, SweepSmem<NW, float>& sm) {
  sweep_last_restrict<NW>(k, sm);
}
template <int NW>
__device__ __noinline__ void sweep_last_add_fn(const KParams& k, float* srv) {
  sweep_last_add<NW>(k, srv);
}

template <typename P, int NW>
__global__ void __launch_bounds__(32 * NW, 1) k_cg_sweep(EngineView v) {
  extern __shared__ __align__(16) float srv[];  // cld floats: r_c, then x_c
  __shared__ SweepSmem<NW, P> sm;
  __shared__ P s_acc[32 * NW];
  // the parameters in shared memory: a meeting empties the L1, and every pass would fetch its
  // pointers again
  __shared__ KParams k;
  for (int i = threadIdx.x; i < (int)(sizeof(KParams) / 4); i += 32 * NW)
    reinterpret_cast<int*>(&k)[i] = reinterpret_cast<const int*>(v.inst)[i];
  __syncthreads();
  DevState* ds = k.ds;
  if (threadIdx.x == 0) {
    sm.st.tol = ds->tol;
    sm.st.inner_rel = ds->inner_rel;
    sm.st.bnorm2 = ds->bnorm2;
    sm.st.max_iter = ds->max_iter;
    sm.st.solve_it = ds->solve_iters;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (*((volatile int*)&ds->outer_active) == 0) return;  // every CTA alike: only the loop around sets it
  const bool def = deflating<P>(k);
  unsigned int target = 0;
  int half = 0;
  auto none = [](const double*) {};
  auto idle = [] {};
  auto meet = [&] {
    const SweepSum<P> no[1] = {};
    return sweep_meet<0, NW, P>(v, sm, target, half, no, none, idle);
  };
  // restriction done: the coarse product
  auto coarse = [&] {
    if (!meet()) return false;
    NNPP_SWEEP_PASS(sweep_coarse, P, NW)(k, srv);
    return meet();
  };
  auto next = [&](double rz, double rr) {
    SweepState<P>& s = sm.st;
    s.beta = sweep_nonzero(s.rz) ? rz * s.irz : 0.0;
    s.beta_p = (P)s.beta;
    s.rz = rz;
    s.rr = rr;
    s.it += 1;
    s.solve_it += 1;
    s.go = sweep_nonzero(s.alpha) && sweep_finite(rr) && sweep_above(rr, s.target) && s.it < s.max_iter && s.solve_it < s.max_iter;
  };
  // The slices over the warps: a warp each for the rounds that fill every warp, and the last round's
  // shared by as many warps as there are for each.  Where all of them make one such round (small cases),
  // a warp keeps its slice: its place and the lane's row are fetched once.
  const int all = gridDim.x * NW;
  const int whole = v.ncslices / all * all;
  int split = 1;
  while (split < 8 && (v.ncslices - whole) * 2 * split <= all) split *= 2;
  int row = -1;
  if (whole == 0) {
    const int sg = blockIdx.x * (NW / split) + warp / split;
    int off = 0, nq = 0;
    if (sg < v.ncslices) row = sweep_take<P, NW>(k, sm, v.cslices, sg, &off, &nq);
    if (lane == 0) {
      sm.off[warp] = off;
      sm.nq[warp] = nq;
    }
    __syncwarp();
  }
  auto shared_slices = [&](auto kc, P beta) {
    constexpr int K = decltype(kc)::value;
    if (whole) return NNPP_SWEEP_PASS(sweep_slices, P, K, NW)(k, sm, s_acc, v.cslices, whole, v.ncslices, beta);
    DotAcc<P> dot;
    sweep_slice<true, P, K>(k, sm, s_acc, sm.off[warp], sm.nq[warp], row, beta, dot);
    dot.warp_sum();
    return SweepSum<P>::of(dot);
  };
  auto apply = [&](P beta) {
    SweepSum<P> dot{};
    if (whole) dot = NNPP_SWEEP_PASS(sweep_slices, P, 1, NW)(k, sm, s_acc, v.cslices, 0, whole, beta);
    if (split == 8)
      dot.add(shared_slices(std::integral_constant<int, 8>(), beta));
    else if (split == 4)
      dot.add(shared_slices(std::integral_constant<int, 4>(), beta));
    else if (split == 2)
      dot.add(shared_slices(std::integral_constant<int, 2>(), beta));
    else
      dot.add(shared_slices(std::integral_constant<int, 1>(), beta));
    return dot;
  };
  NNPP_SWEEP_PASS(sweep_rhs, P, NW)(k, sm);
  bool ok = coarse();
  if (ok) {
    const Dots3<P> d = NNPP_SWEEP_PASS(sweep_first_z, P, NW)(k, srv, def);
    const SweepSum<P> t[3] = {d.rz, d.rr, d.r0};
    ok = sweep_meet<3, NW, P>(v, sm, target, half, t, [&](const double* tot) {
      SweepState<P>& s = sm.st;
      s.rz = tot[0];
      s.rr = tot[1];
      s.beta = s.alpha = s.pq = 0.0;
      s.beta_p = s.alpha_p = P(0);
      s.it = 0;
      // FP64: to the final tolerance in one sweep; mixed: by inner_rel of the correction equation's
      // residual (before the deflation), not below what the outer tolerance needs
      const double tb = s.tol * s.tol * s.bnorm2;
      s.target = sizeof(P) == 4 ? fmax(s.inner_rel * s.inner_rel * tot[2], 0.09 * tb) : 0.25 * tb;
      s.go = tot[1] > s.target && s.max_iter > 0;
    }, idle);
  }
  while (ok && sm.st.go) {
    const SweepSum<P> pq = apply(sm.st.beta_p);
    auto inverse = [&] { sm.st.irz = div_newton(1.0, sm.st.rz); };  // next()'s division, ahead
    if (def) {
      if constexpr (sizeof(P) == 4) {
        const SweepSum<P> no[1] = {};
        if (!(ok = sweep_meet<0, NW, P>(v, sm, target, half, no, none, inverse))) break;
        NNPP_SWEEP_PASS(sweep_restrict_q, NW)(k, sm);
        if (!(ok = meet())) break;
        const SweepSum<P> d[2] = {pq, NNPP_SWEEP_PASS(sweep_coarse, P, NW)(k, srv)};
        ok = sweep_meet<2, NW, P>(v, sm, target, half, d, [&](const double* tot) {
          SweepState<P>& s = sm.st;  // p.P_d A p = p.q - r_c.x_c
          s.pq = tot[0];
          const double pw = tot[0] - tot[1];
          s.alpha = (sweep_positive(tot[0]) && sweep_positive(pw) && sweep_finite(pw)) ? div_newton(s.rz, pw) : 0.0;
          s.alpha_p = (P)s.alpha;
        }, idle);
        if (!ok) break;
        const Dots2<P> u = NNPP_SWEEP_PASS(sweep_update, NW)(k, srv, sm.st.alpha_p);
        const SweepSum<P> t[2] = {u.a, u.b};
        ok = sweep_meet<2, NW, P>(v, sm, target, half, t, [&](const double* tot) { next(tot[0], tot[1]); }, idle);
      }
    } else {
      const SweepSum<P> d[1] = {pq};
      ok = sweep_meet<1, NW, P>(v, sm, target, half, d, [&](const double* tot) {
        SweepState<P>& s = sm.st;
        s.pq = tot[0];
        s.alpha = (sweep_positive(tot[0]) && sweep_finite(tot[0])) ? div_newton(s.rz, tot[0]) : 0.0;
        s.alpha_p = (P)s.alpha;
      }, inverse);
      if (!ok) break;
      const Dots2<P> u = NNPP_SWEEP_PASS(sweep_update_restrict, P, NW)(k, sm, sm.st.alpha_p);
      if (!(ok = meet())) break;
      SweepSum<P> t[2] = {u.a, u.b};
      t[0].add(NNPP_SWEEP_PASS(sweep_coarse, P, NW)(k, srv));  // r.D^-1 r + r_c.x_c
      ok = sweep_meet<2, NW, P>(v, sm, target, half, t, [&](const double* tot) { next(tot[0], tot[1]); }, idle);
      if (!ok) break;
      NNPP_SWEEP_PASS(sweep_z, P, NW)(k, srv);
      ok = meet();
    }
  }
  if constexpr (sizeof(P) == 4)
    if (ok && def) {
      NNPP_SWEEP_PASS(sweep_last_restrict, NW)(k, sm);
      ok = coarse();
      if (ok) NNPP_SWEEP_PASS(sweep_last_add, NW)(k, srv);
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!ok) {
      ds->wait_timeout = 1;
    } else if (blockIdx.x == 0) {
      const SweepState<P>& s = sm.st;
      ds->rz = s.rz;
      ds->rr = s.rr;
      ds->alpha = s.alpha;
      ds->beta = s.beta;
      ds->pq = s.pq;
      ds->inner_target = s.target;
      ds->inner_it = s.it;
      ds->solve_iters = s.solve_it;
      ds->cg_iters += s.it;
      ds->inner_active = 0;
    }
    // the last CTA out sets the meeting's counters back
    __threadfence();
    if (atomicAdd(&v.ticket[v.M + 5], 1u) == gridDim.x - 1) {
      v.ticket[v.M + 4] = 0;
      v.ticket[v.M + 5] = 0;
    }
  }
}
#undef NNPP_SWEEP_PASS

// ------------------------------------------------------------------- warm start ---------
// Initial guess of the potential solve from the last H solutions x_n, ..., x_{n-H+1} and
// their images A x (the ring xh, bh; bh = b - r at the end of each solve):
//   x0 = x_n + sum_l a_l D^l x_n,   D^l: l-th backward difference at the newest solution,
// with the coefficients minimising the A-norm error of x0 over that affine space
// (Galerkin condition  (D^i x)^T A (D^j x) a_j = (D^i x)^T (b_new - A x_n)); A D^l x is the
// same difference of bh.  The differences are the well-conditioned basis of the span of
// the history; the linear extrapolation 2 x_n - x_{n-1} is the member a = (1, 0, ...).
constexpr int kWarmD = kHistMax - 1;                         // differences
constexpr int kWarmSlots = kWarmD * (kWarmD + 1) / 2 + kWarmD + 1;  // G (upper), rhs, x.Ax
static_assert(kWarmSlots <= kReduceSlots, "warm-start partials exceed the reduction buffer");

__device__ __forceinline__ int warm_history(const KParams& k) {
  if (k.hist_m < 3 || !k.extrapolate) return 0;
  const int n = k.ds->hist_n;
  return n < k.hist_m ? n : k.hist_m;
}

// Solve the scaled Galerkin system by Cholesky; differences whose pivot falls below 1e-12
// (near-dependent) or whose A-norm is below 1e-12 of the solution's (rounding level) end
// the basis.  One warp: lane 5 i + j holds the scaled entry (i, j), lane 25 + i the right-hand side's i,
// which takes the same steps as a sixth column.  (Thread 0 alone took 45 us, a chain of some 45 divisions
// and roots of 25 FP64 instructions that each hold the pipe for 64 cycles.)
__device__ void warm_solve(const double* tot, int nd, DevState* ds) {
  static_assert(kWarmD * (kWarmD + 1) <= 32, "an entry a lane");
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int D = kWarmD, kRhs = D * D, kTri = D * (D + 1) / 2;
  const int lane = threadIdx.x & 31;
  const bool entry = lane < kRhs, rhs = lane >= kRhs && lane < kRhs + D;
  const int i = entry ? lane / D : rhs ? lane - kRhs : 0, j = entry ? lane % D : D;
  auto tri = [&](int p, int q) { return p * D - p * (p - 1) / 2 + (q - p); };  // p <= q
  double c = entry ? tot[tri(min(i, j), max(i, j))] : rhs ? tot[kTri + i] : 0.0;
  const double gd = tot[tri(lane < D ? lane : 0, lane < D ? lane : 0)];  // lanes < D: the diagonal
  const bool use = lane < nd && lane < D && gd > 1e-24 * tot[kTri + D] && isfinite(gd);
  const int n = __ffs(~__ballot_sync(kAll, use)) - 1;
  const double dinv = use ? rsqrt_newton(gd) : 1.0;
  c *= __shfl_sync(kAll, dinv, i);
  const double dj = __shfl_sync(kAll, dinv, entry ? j : 0);
  if (entry) c *= dj;
  int m = 0;
  double inv = 0.0;  // lane q: 1 / L(q, q)
  for (int q = 0; q < n; ++q) {
    const double sq = __shfl_sync(kAll, c, q * D + q);
    if (!(sq > 1e-12)) break;
    const double iv = rsqrt_newton(sq);
    if ((entry && j == q) || (rhs && i == q)) c *= iv;
    const double li = __shfl_sync(kAll, c, i * D + q);
    const double lj = __shfl_sync(kAll, c, entry ? j * D + q : kRhs + q);
    if ((entry || rhs) && i > q && j > q) c = fma(-li, lj, c);
    if (lane == q) inv = iv;
    m = q + 1;
  }
  for (int q = m - 1; q >= 0; --q) {
    const double y = __shfl_sync(kAll, c, kRhs + q) * __shfl_sync(kAll, inv, q);
    const double l = __shfl_sync(kAll, c, q * D + i);  // L(q, i)
    if (rhs && i == q) c = y;
    if (rhs && i < q) c = fma(-l, y, c);
  }
  const bool ok = m > 0 && __all_sync(kAll, !(rhs && i < m) || isfinite(c));
  const double di = __shfl_sync(kAll, dinv, i);
  if (rhs) ds->warm_coef[i] = ok && i < m ? c * di : 0.0;
  if (lane == 0) ds->warm_nd = ok ? m : 0;
}

// backward differences D^1..D^{H-1} of the FP32 pairs t[0..H-1] (newest first) into d;
// t is consumed
__device__ __forceinline__ void pair_warm_diffs(float (&th)[kHistMax], float (&tl)[kHistMax], int H,
                                                float (&dh)[kWarmD], float (&dl)[kWarmD]) {
#pragma unroll
  for (int l = 1; l < kHistMax; ++l) {
#pragma unroll
    for (int j = 0; j + 1 < kHistMax; ++j)
      if (j + l < H) pair_sub(th[j], tl[j], th[j + 1], tl[j + 1], th[j], tl[j]);
    dh[l - 1] = l < H ? th[0] : 0.0f;
    dl[l - 1] = l < H ? tl[0] : 0.0f;
  }
}

// the history of node a as FP32 pairs, newest first (zero beyond H)
__device__ __forceinline__ void load_history_pairs(const double* ring, const int (&slot)[kHistMax], int H,
                                                   size_t N, int a, float (&th)[kHistMax], float (&tl)[kHistMax]) {
#pragma unroll
  for (int j = 0; j < kHistMax; ++j) {
    th[j] = tl[j] = 0.0f;
    if (j < H) split_pair(ring[(size_t)slot[j] * N + a], th[j], tl[j]);
  }
}

// A warp's sums of its lanes' 32 values, value q in lane q: at each step the lanes of a pair keep half of
// the values each (31 pair sums instead of five a value)
__device__ __forceinline__ void pair_warp_transpose_sum(float (&h)[32], float (&l)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int q = 0; q < off; ++q) {
      const float sh = up ? h[q] : h[q + off], sl = up ? l[q] : l[q + off];
      float kh = up ? h[q + off] : h[q], kl = up ? l[q + off] : l[q];
      pair_add(kh, kl, __shfl_xor_sync(0xffffffffu, sh, off), __shfl_xor_sync(0xffffffffu, sl, off));
      h[q] = kh;
      l[q] = kl;
    }
  }
}

// The Galerkin system's dot products, on FP32 pairs (the FP64 rate of the GB300 would
// bound this pass): the history is split into pairs, differenced and multiplied with the
// pair operations, ~2^-46 relative per operation.  Up to 64k nodes it is the chain of the sums and of the
// small solve: a value a lane in every stage of the sums, a warp in the solve.  A step of 8k nodes 0.251 ms
// with 21 sums one after another and the solve in one thread, 0.215
// so.
template <typename P>
__global__ void __launch_bounds__(kBlock, 2) k_warm_dots(EngineView v) {
  constexpr int kW = kBlock / 32;
  static_assert(kWarmSlots <= 32 && kWarmSlots <= kReduceSlots, "a value a lane");
  __shared__ float2 s_sum[kW][32];
  __shared__ double s_tot[32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* parts = reinterpret_cast<float2*>(v.partials);  // item i: kReduceSlots pairs
  // the warps' pairs summed by lane (of warp 0)
  auto across = [&](float& th, float& tl) {
    __syncthreads();
    th = tl = 0.0f;
    if (warp == 0)
#pragma unroll
      for (int w = 0; w < kW; ++w) pair_add(th, tl, s_sum[w][lane].x, s_sum[w][lane].y);
  };
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const int H = warm_history(k);
    DotAcc<float> part[kWarmSlots];
    if (H >= 3) {
      const int head = k.ds->hist_head, m = k.hist_m;
      const size_t N = (size_t)k.N;
      int slot[kHistMax];
#pragma unroll
      for (int j = 0; j < kHistMax; ++j) slot[j] = (head - j + 2 * m) % m;
      float lamh, laml, zh[S], zl[S];
      split_pair(k.lam, lamh, laml);
#pragma unroll
      for (int s2 = 0; s2 < S; ++s2) split_pair(k.z[s2], zh[s2], zl[s2]);
      for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
        if (!k.freem[a]) continue;
        float xh[kHistMax], xl[kHistMax], bh[kHistMax], bl[kHistMax];
        load_history_pairs(k.xh, slot, H, N, a, xh, xl);
        load_history_pairs(k.bh, slot, H, N, a, bh, bl);
        float bnh, bnl;
        if (k.b_override) {
          split_pair(k.b_override[a], bnh, bnl);  // adjoint solves: the given right-hand side
        } else {
          // b = lam sum_s z_s c_s
          float rh = 0.0f, rl = 0.0f;
#pragma unroll
          for (int s2 = 0; s2 < S; ++s2) {
            float ch, cl, ph, pl;
            if constexpr (sizeof(P) == 4) {
              const float4 lo4 = k.clo[a];
              ch = k.rec32_cur[a].c[s2];
              cl = sel4(lo4, s2);
            } else {
              split_pair(k.rec64_cur[a].c[s2], ch, cl);
            }
            pair_mul(zh[s2], zl[s2], ch, cl, ph, pl);
            pair_add(rh, rl, ph, pl);
          }
          pair_mul(lamh, laml, rh, rl, bnh, bnl);
        }
        float gh, gl;
        pair_sub(bnh, bnl, bh[0], bl[0], gh, gl);
        const float x0h = xh[0], x0l = xl[0], b0h = bh[0], b0l = bl[0];
        float dxh[kWarmD], dxl[kWarmD], dbh[kWarmD], dbl[kWarmD];
        pair_warm_diffs(xh, xl, H, dxh, dxl);
        pair_warm_diffs(bh, bl, H, dbh, dbl);
        int q = 0;
#pragma unroll
        for (int i = 0; i < kWarmD; ++i)
#pragma unroll
          for (int j = i; j < kWarmD; ++j) part[q++].add_pair(dxh[i], dxl[i], dbh[j], dbl[j]);
#pragma unroll
        for (int i = 0; i < kWarmD; ++i) part[q++].add_pair(dxh[i], dxl[i], gh, gl);
        part[q].add_pair(x0h, x0l, b0h, b0l);
      }
    }
    float sh[32], sl[32], th, tl;
#pragma unroll
    for (int q = 0; q < 32; ++q) {
      sh[q] = q < kWarmSlots ? part[q < kWarmSlots ? q : 0].hi : 0.0f;
      sl[q] = q < kWarmSlots ? part[q < kWarmSlots ? q : 0].lo : 0.0f;
    }
    pair_warp_transpose_sum(sh, sl);
    s_sum[warp][lane] = make_float2(sh[0], sl[0]);
    across(th, tl);
    if (warp == 0 && lane < kWarmSlots) parts[(size_t)item * kReduceSlots + lane] = make_float2(th, tl);
    const int first = v.chunk_first[c.inst], count = v.chunk_count[c.inst];
    if (item_done(&v.ticket[c.inst], count, &s_last)) {
      // the last CTA: a warp takes every kW-th item, its lanes a value each
      constexpr int U = 8;
      float ah = 0.0f, al = 0.0f;
      for (int i = warp; i < count; i += U * kW) {
        float2 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          x[u] = make_float2(0.0f, 0.0f);
          if (i + u * kW < count && lane < kWarmSlots) x[u] = __ldcg(parts + (size_t)(first + i + u * kW) * kReduceSlots + lane);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) pair_add(ah, al, x[u].x, x[u].y);
      }
      s_sum[warp][lane] = make_float2(ah, al);
      across(th, tl);
      if (warp == 0) {
        s_tot[lane] = (double)th + (double)tl;
        if (lane == 0) {
          k.ds->warm_nd = 0;
          v.ticket[c.inst] = 0;
        }
        __syncwarp();
        if (H >= 3) warm_solve(s_tot, H - 1, k.ds);
      }
    }
    __syncthreads();
  }
}

// the solution of a solve run outside a step (adjoint) and A x = b - r into ring slot `slot`
__global__ void k_record_solve(KParams k, int slot) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    const size_t o = (size_t)slot * k.N + a;
    k.xh[o] = k.phi64[a];
    k.bh[o] = k.freem[a] ? k.b64[a] - k.r64[a] : 0.0;
  }
}

// x0 = x_n + sum_l a_l D^l x_n on the unknowns, into phi64 and the state's potential
// (FP32-pair arithmetic as k_warm_dots; x0 is exact in FP64 as the sum of its pair)
template <typename P>
__global__ void __launch_bounds__(kBlock) k_warm_apply(EngineView v) {
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    const int H = warm_history(k);
    if (H < 3) continue;
    const int nd = k.ds->warm_nd;
    if (nd <= 0) continue;
    float ch[kWarmD], cl[kWarmD];
#pragma unroll
    for (int i = 0; i < kWarmD; ++i) split_pair(k.ds->warm_coef[i], ch[i], cl[i]);
    const int head = k.ds->hist_head, m = k.hist_m;
    const size_t N = (size_t)k.N;
    int slot[kHistMax];
#pragma unroll
    for (int j = 0; j < kHistMax; ++j) slot[j] = (head - j + 2 * m) % m;
    for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
      if (!k.freem[a]) continue;
      float th[kHistMax], tl[kHistMax];
      load_history_pairs(k.xh, slot, H, N, a, th, tl);
      const float xh0 = th[0], xl0 = tl[0];
      float dh[kWarmD], dl[kWarmD];
      pair_warm_diffs(th, tl, H, dh, dl);
      float sh = 0.0f, sl = 0.0f;
#pragma unroll
      for (int i = 0; i < kWarmD; ++i) {
        float ph, pl;
        pair_mul(ch[i], cl[i], dh[i], dl[i], ph, pl);
        pair_add(sh, sl, ph, pl);
      }
      pair_add(sh, sl, xh0, xl0);
      // normalised pair: hi the FP32 rounding of the sum, lo its exact remainder
      const float hi = sh + sl;
      const float lo = sl - (hi - sh);
      k.phi64[a] = (double)hi + (double)lo;
      if constexpr (sizeof(P) == 4) {
        k.rec32_cur[a].phi_hi = hi;
        k.rec32_cur[a].phi_lo = lo;
      } else {
        k.rec64_cur[a].phi = (double)hi + (double)lo;
      }
    }
  }
}

// ---------------------------------------------------- potential residuals on the slices ----
// Mixed path: the prep and the refinement residual as slice kernels over the sliced operator
// (one lane per row, two quads of bond columns a batch, neighbour values gathered through
// L1/L2), with the FP64 weight carried as the FP32 pair (sell, sell_lo) and FP32-pair
// arithmetic (TwoProd, TwoSum) along each row.  Slice partials, one global ticket; the last
// CTA makes every instance's decisions.
constexpr int kResB = 8;

__device__ __forceinline__ const float* sell_lo_col(const KParams& k, const SliceDesc& d) {
  return k.sell_lo + (size_t)(d.off >> 5) * 32;
}

// A lane's row of the CG operator as the preps write it: bonds are collected four at a time and
// stored as a quad (one 16- or 32-byte and one 8-byte store instead of scattered words).  W: float
// with low words, or double.
template <typename W>
struct CgRowWriter {
  float* sell;            // the slice's interleaved array (weights unless W is double, codes)
  float* lo;              // the weights' low words (W = float)
  double* w64;            // the FP64 weights (W = double)
  int lane, n;
  W w[4];
  float l[4];
  unsigned int c[4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      w[u] = W(0);
      l[u] = 0.0f;
      c[u] = 0u;
    }
  }
  __device__ __forceinline__ void flush(int q) {
    float* base = sell + (size_t)q * kQuadW;
    reinterpret_cast<uint2*>(base + 128)[lane] = make_uint2(c[0] | c[1] << 16, c[2] | c[3] << 16);
    if constexpr (sizeof(W) == 4) {
      reinterpret_cast<float4*>(base)[lane] = make_float4(w[0], w[1], w[2], w[3]);
      reinterpret_cast<float4*>(lo + (size_t)q * 128)[lane] = make_float4(l[0], l[1], l[2], l[3]);
    } else {
      double2* o = reinterpret_cast<double2*>(w64 + (size_t)q * 128 + 4 * lane);
      o[0] = make_double2(w[0], w[1]);
      o[1] = make_double2(w[2], w[3]);
    }
    clear();
  }
  __device__ __forceinline__ void add(W weight, float low, unsigned int code) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if ((n & 3) == u) {
        w[u] = weight;
        l[u] = low;
        c[u] = code;
      }
    if ((++n & 3) == 0) flush((n >> 2) - 1);
  }
  // the last quad and zero quads up to the slice's capacity (columns, a multiple of 4)
  __device__ __forceinline__ void finish(int capacity) {
    for (int q = n >> 2; q < capacity >> 2; ++q) flush(q);
  }
};

// an instance's decision after the prep from ||b||^2 and ||r||^2 (one thread)
__device__ __forceinline__ void prep_decide(DevState* ds, double bb, double rr) {
  ds->op_valid = 1;
  const double bn = bb > 0.0 ? bb : 1.0;
  ds->bnorm2 = bn;
  ds->rnorm2 = rr;
  ds->outer_it = 0;
  ds->solve_iters = 0;
  const bool go = rr > ds->tol * ds->tol * bn && ds->max_outer > 0;
  if (!go) {
    ds->cg_solves += 1;
    ds->last_relres = sqrt(rr / bn);
  }
  ds->outer_active = go ? 1 : 0;
  ds->inner_active = 0;
}

// bond columns c0 .. c0 + nc - 1 (whole quads) of the slice: weights as FP32 pairs, codes
__device__ __forceinline__ void load_residual_quads(const QuadPtr& op, const float4* lo, int c0, int nc,
                                                    float (&w)[kResB], float (&wl)[kResB],
                                                    unsigned int (&code)[kResB]) {
#pragma unroll
  for (int q = 0; q < kResB / 4; ++q)
    if (4 * q < nc) {
      const float4 wq = op.weights((c0 >> 2) + q), lq = ld_stream(lo + 32 * ((c0 >> 2) + q));
      const uint2 cq = op.codes((c0 >> 2) + q);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        w[4 * q + u] = quad_weight(wq, u);
        wl[4 * q + u] = quad_weight(lq, u);
        code[4 * q + u] = quad_code(cq, u);
      }
    }
}

// per node {phi_hi, phi_lo} (zero on solid nodes), liquid flag, potential-Dirichlet flag; the FP64
// path's preps read the potential from z64 instead
template <typename P>
__global__ void __launch_bounds__(kBlock) k_phi4(EngineView v) {
  // a prep that forms the mask sums rewrites the CG operator's rows: their slices' longest
  // rows start from zero
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < v.ncslices; g += gridDim.x * blockDim.x) {
    const int inst = v.cslices[g].inst;
    const KParams& k = v.inst[inst];
    if (k.ds->op_valid == 0) k.cg_width[g - v.cslice_first[inst]] = 0;
  }
  for (int item = blockIdx.x; item < v.nchunks; item += gridDim.x) {
    const Chunk c = v.chunks[item];
    const KParams& k = v.inst[c.inst];
    for (int a = c.begin + threadIdx.x; a < c.end; a += kBlock) {
      const bool liq = phase_of<P>(k, a) == 0.0f;
      const double ph = k.phi64[a];
      if (sizeof(P) == 8) k.z64[a] = liq ? ph : 0.0;
      const float hi = (float)ph;
      const float lo = (float)(ph - (double)hi);
      k.phi4[a] = make_float4(liq ? hi : 0.0f, liq ? lo : 0.0f, liq ? 1.0f : 0.0f,
                              ((k.dirmask[a] >> S) & 1) ? 1.0f : 0.0f);
    }
  }
}

// prep: b, the FP64 residual r = b - A phi and the norms; the mask-only sums (diagonal,
// Dirichlet coupling, unknown flag) are formed only when the phases changed (op_valid == 0), by
// k_prep_masks, for the instances that need them; k_prep_slices serves the others and takes every
// instance's decision.  (One kernel for both had the mask pass's 128 registers: the usual pass, which
// only sums phi, took 0.22 ms at 512k nodes, 0.17 and 0.003 for the other's launch alone.)  K warps share
// a slice where a warp each leaves the chip's warps empty (see SplitSlice); the mask pass, a warp a
// slice, adds the K parts as they do, so that a step repeated from a restored state gives the same bits.

// a row's b, residual and norms from its sums (mixed path); the slice's partials
__device__ __forceinline__ void prep_row(const EngineView& v, const KParams& k, int sg, int lane, int a, bool rowok,
                                         bool fr, double dsum, double cpl, double swphi, double pha) {
  float b2h = 0.0f, b2l = 0.0f, r2h = 0.0f, r2l = 0.0f;  // b.b and r.r as FP32 pairs
  if (rowok) {
    double b;
    if (k.b_override) {
      b = k.b_override[a];
    } else {
      double R11 = 0.0;
      for (int s = 0; s < S; ++s) R11 += k.z[s] * conc_of<float>(k, a, s);
      b = k.lam * R11;
    }
    const double bb = fr ? b : 0.0;
    const double r = fr ? bb - (dsum * pha - swphi) : 0.0;
    k.b64[a] = bb;
    k.r64[a] = r;
    const double be = bb + (fr ? cpl : 0.0);
    pair_square(be, b2h, b2l);
    pair_square(r, r2h, r2l);
  }
  pair_warp_sum(b2h, b2l);
  pair_warp_sum(r2h, r2l);
  if (lane == 0) {
    store_pair(v.partials, sg, b2h, b2l);
    store_pair(v.partials, (size_t)v.stride + sg, r2h, r2l);
  }
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_prep_masks(EngineView v) {
  __shared__ int s_hb[kBlock / 32][12];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int any = 0;
  for (int i = threadIdx.x; i < v.M; i += kBlock) any |= v.inst[i].ds->op_valid == 0;
  if (!__syncthreads_or(any)) return;
  for (int sg = blockIdx.x * (kBlock / 32) + warp; sg < v.nslices; sg += gridDim.x * (kBlock / 32)) {
    const SliceDesc& d = v.slices[sg];
    const KParams& k = v.inst[d.inst];
    if (k.ds->op_valid != 0) continue;
    if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
    __syncwarp();
    const int a = d.row0 + lane;
    const bool rowok = lane < d.nrows;
    float4 fa = make_float4(0.f, 0.f, 0.f, 0.f);
    int len = 0;
    if (rowok) {
      fa = k.phi4[a];
      len = k.row[a + 1] - k.row[a];
    }
    const bool scan = rowok && fa.z != 0.0f && fa.w == 0.0f;
    const int* hb = s_hb[warp];
    const QuadPtr op(sell_w(k, d), lane);
    const float4* wls = reinterpret_cast<const float4*>(sell_lo_col(k, d)) + lane;
    // sum_j w phi_j over the liquid columns as an FP32 pair in bond order (k_prep_slices
    // adds the solid columns' exact zeros, so both give the same bits).  The mask
    // sums also write the row into the CG operator's slices: its bonds to possible unknowns
    // (liquid, no potential Dirichlet value), codes relative to that slice's windows, zero
    // padding, and the slice's longest row.
    const int cpos = scan ? k.cg_pos[a] : -1;
    const SliceDesc* cd = nullptr;
    CgRowWriter<float> out;
    int cby = 0, cbz = 0;
    if (cpos >= 0) {
      cd = v.cslices + v.cslice_first[d.inst] + (cpos >> 5);
      const size_t col0 = (size_t)(cd->off >> 5);
      out.sell = k.sell_cg + col0 * kSellW;
      out.lo = k.sell_cg_lo + col0 * 32;
      out.lane = cpos & 31;
      out.n = 0;
      out.clear();
      cby = cd->tile & 0xffff;
      cbz = cd->tile >> 16;
    }
    float dh = 0.f, dl = 0.f, ch = 0.f, cl = 0.f;
    float ph_[K], pl_[K];  // sum w phi in the K parts of k_prep_slices
    for (int h = 0; h < K; ++h) ph_[h] = pl_[h] = 0.0f;
    int anyll = 0;
    if (__any_sync(0xffffffffu, scan)) {
      const int width = d.width;
      for (int c0 = 0; c0 < width; c0 += kResB) {
        const int h = c0 / kResB % K;
        float sh = ph_[h], sl = pl_[h];
        const int nc = min(kResB, width - c0);  // a multiple of 4
        float w[kResB], wl[kResB];
        unsigned int code[kResB];
        load_residual_quads(op, wls, c0, nc, w, wl, code);
        float4 f[kResB];
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) f[u] = __ldg(k.phi4 + code_node(hb, code[u]));
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc && c0 + u < len && f[u].z != 0.0f) {
            float ph, pl;
            pair_mul(w[u], wl[u], f[u].x, f[u].y, ph, pl);
            pair_add(sh, sl, ph, pl);
            pair_add(dh, dl, w[u], wl[u]);
            anyll = 1;
            if (f[u].w != 0.0f) {
              pair_add(ch, cl, ph, pl);
            } else if (cpos >= 0) {
              const int m = code_node(hb, code[u]);
              const int xr = k.xrow[m];
              const int r = ((xr & 0xffff) - cby + 1) + 3 * ((xr >> 16) - cbz + 1);
              out.add(w[u], wl[u], (unsigned int)((r << 12) | (m - cd->gbase[r])));
            }
          }
        ph_[h] = sh;
        pl_[h] = sl;
      }
    }
    if (cpos >= 0) {
      // zero padding up to the slice's capacity (its longest full row)
      out.finish(cd->width);
      atomicMax(&k.cg_width[cpos >> 5], out.n);
    }
    const bool fr = scan && anyll;
    const double dsum = (double)dh + (double)dl, cpl = (double)ch + (double)cl;
    if (rowok) {
      k.freem[a] = fr ? 1 : 0;
      k.dsum64[a] = fr ? dsum : 1.0;
      k.cpl64[a] = fr ? cpl : 0.0;
      k.dinv64[a] = fr ? 1.0 / dsum : 0.0;
      k.d32[a] = fr ? (float)dsum : 1.0f;
      k.dinv32[a] = fr ? (float)(1.0 / dsum) : 0.0f;
    }
    float sh = ph_[0], sl = pl_[0];
    for (int h = 1; h < K; ++h) pair_add(sh, sl, ph_[h], pl_[h]);
    prep_row(v, k, sg, lane, a, rowok, fr, dsum, cpl, (double)sh + (double)sl, (double)fa.x + (double)fa.y);
    __syncwarp();
  }
}

template <int K>
__global__ void __launch_bounds__(kBlock, 4) k_prep_slices(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[2 * kBlock / 32];
  __shared__ float2 s_part[K > 1 ? kBlock : 1];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % K;
  // K == 1: warps claim slices one at a time (slices of solid nodes, narrow and partial slices
  // cost less than full ones)
  constexpr int kAtOnce = SplitSlice<K>::kSlices;
  for (int base = K == 1 ? claim_slice(v, lane) : (int)blockIdx.x * kAtOnce; base < v.nslices;
       base = K == 1 ? claim_slice(v, lane) : base + (int)gridDim.x * kAtOnce) {
    const int sg = K == 1 ? base : min(base + warp / K, v.nslices - 1);
    const SliceDesc& d = v.slices[sg];
    const KParams& k = v.inst[d.inst];
    // the others are k_prep_masks's
    const bool mine = (K == 1 || base + warp / K < v.nslices) && k.ds->op_valid != 0;
    if (K == 1 && !mine) continue;
    if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
    __syncwarp();
    const int a = d.row0 + lane;
    const bool rowok = mine && lane < d.nrows;
    const bool fr = rowok && k.freem[a] != 0;
    const int* hb = s_hb[warp];
    float sh = 0.f, sl = 0.f;
    if (__any_sync(0xffffffffu, fr)) {
      const QuadPtr op(sell_w(k, d), lane);
      const float4* wls = reinterpret_cast<const float4*>(sell_lo_col(k, d)) + lane;
      const int width = d.width;
      for (int c0 = kResB * part; c0 < width; c0 += kResB * K) {
        const int nc = min(kResB, width - c0);  // a multiple of 4
        float w[kResB], wl[kResB];
        unsigned int code[kResB];
        load_residual_quads(op, wls, c0, nc, w, wl, code);
        float2 f[kResB];
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) f[u] = __ldg(reinterpret_cast<const float2*>(k.phi4 + code_node(hb, code[u])));
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) {
            float ph, pl;
            pair_mul(w[u], wl[u], f[u].x, f[u].y, ph, pl);
            pair_add(sh, sl, ph, pl);
          }
      }
    }
    if (K > 1) {
      s_part[threadIdx.x] = make_float2(sh, sl);
      __syncthreads();
      if (part == 0)
#pragma unroll
        for (int h = 1; h < K; ++h) pair_add(sh, sl, s_part[threadIdx.x + 32 * h].x, s_part[threadIdx.x + 32 * h].y);
    }
    double dsum = 1.0, cpl = 0.0, pha = 0.0;
    if (fr && part == 0) {
      const float2 fa = __ldg(reinterpret_cast<const float2*>(k.phi4 + a));
      dsum = k.dsum64[a];
      cpl = k.cpl64[a];
      pha = (double)fa.x + (double)fa.y;
    }
    if (mine && part == 0) prep_row(v, k, sg, lane, a, rowok, fr, dsum, cpl, (double)sh + (double)sl, pha);
    if (K > 1)
      __syncthreads();
    else
      __syncwarp();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[2];
      reduce_pair_items<2>(v.partials, v.stride, v.slice_first[i], v.slice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        prep_decide(v.inst[i].ds, tot[0], tot[1]);
        instance_finished(v, i, 0, hc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      v.ticket[v.M + 1] = 0;
      v.ticket[v.M + 2] = 0;
    }
  }
}

// The FP64 path's prep on the transport's slices (k_prep_slices with FP64 weights and sums): b,
// r = b - A phi and their norms, K warps a slice; phi of the liquid nodes (zero on solid ones)
// is gathered from z64 (written by k_phi4, free until the CG starts).  While the mask sums
// hold (op_valid) only sum_j w phi_j is formed; otherwise part 0 forms the row's sums alone and
// writes its bonds to possible unknowns into the CG slices.
template <int K>
__global__ void __launch_bounds__(kBlock) k_prep64(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ double s_acc[K > 1 ? kBlock : 1];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[2 * kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.nslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.slices[have ? ss.sg : 0];
    const KParams& k = v.inst[d.inst];
    const bool cached = k.ds->op_valid != 0;
    if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
    __syncwarp();
    const int* hb = s_hb[warp];
    const int a = d.row0 + lane;
    const bool rowok = have && lane < d.nrows;
    float4 fa = make_float4(0.f, 0.f, 0.f, 0.f);
    int len = 0;
    if (rowok) {
      fa = k.phi4[a];
      len = k.row[a + 1] - k.row[a];
    }
    const bool scan = rowok && fa.z != 0.0f && fa.w == 0.0f;
    const QuadPtr op(sell_w(k, d), lane);
    const double* w64 = k.sell64 + (size_t)(d.off >> 5) * 32 + 4 * lane;
    const double* phil = k.z64;
    double dsum = 0.0, cpl = 0.0;
    int anyll = 0;
    // sum_j w phi_j over the liquid columns (zero elsewhere), the same order whether the rows are
    // cached or not: a step that is repeated from a restored state gives the same bits
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    if (scan && (cached ? k.freem[a] != 0 : K > 1)) {
      const int nq = (len + 3) >> 2;
#pragma unroll 2
      for (int q = ss.part; q < nq; q += K) {
        double w[4];
        const uint2 code = op.codes(q);
        ld_stream_d4(w64 + 128 * (size_t)q, w);
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[t] = fma(w[t], __ldg(phil + code_node(hb, quad_code(code, t))), acc[t]);
      }
    }
    if (!cached && ss.part == 0) {
      const int cpos = scan ? k.cg_pos[a] : -1;
      const SliceDesc* cd = nullptr;
      CgRowWriter<double> out;
      int cby = 0, cbz = 0;
      if (cpos >= 0) {
        cd = v.cslices + v.cslice_first[d.inst] + (cpos >> 5);
        const size_t col0 = (size_t)(cd->off >> 5);
        out.w64 = k.sell_cg64 + col0 * 32;
        out.sell = k.sell_cg + col0 * kSellW;
        out.lane = cpos & 31;
        out.n = 0;
        out.clear();
        cby = cd->tile & 0xffff;
        cbz = cd->tile >> 16;
      }
      if (scan)
        for (int q = 0; 4 * q < len; ++q) {
          double w[4];
          const uint2 code = op.codes(q);
          ld_stream_d4(w64 + 128 * (size_t)q, w);
          float4 f[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) f[t] = __ldg(k.phi4 + code_node(hb, quad_code(code, t)));
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (4 * q + t >= len || f[t].z == 0.0f) continue;
            const int m = code_node(hb, quad_code(code, t));
            const double ph = phil[m];
            dsum += w[t];
            if (K == 1) acc[t] = fma(w[t], ph, acc[t]);
            anyll = 1;
            if (f[t].w != 0.0f) {
              cpl += w[t] * ph;
            } else if (cpos >= 0) {
              const int xr = k.xrow[m];
              const int r = ((xr & 0xffff) - cby + 1) + 3 * ((xr >> 16) - cbz + 1);
              out.add(w[t], 0.0f, (unsigned int)((r << 12) | (m - cd->gbase[r])));
            }
          }
        }
      if (cpos >= 0) {
        out.finish(cd->width);
        atomicMax(&k.cg_width[cpos >> 5], out.n);
      }
    }
    double swphi[1] = {(acc[0] + acc[1]) + (acc[2] + acc[3])};
    if (K > 1) split_sum<K, 1>(swphi, s_acc);
    if (have && ss.part == 0) {
      double part[2] = {0.0, 0.0};
      if (rowok) {
        double b;
        if (k.b_override) {
          b = k.b_override[a];
        } else {
          double R11 = 0.0;
          for (int s = 0; s < S; ++s) R11 += k.z[s] * conc_of<double>(k, a, s);
          b = k.lam * R11;
        }
        bool fr;
        if (cached) {
          fr = k.freem[a] != 0;
          dsum = k.dsum64[a];
          cpl = k.cpl64[a];
        } else {
          fr = scan && anyll;
          k.freem[a] = fr ? 1 : 0;
          k.dsum64[a] = fr ? dsum : 1.0;
          k.cpl64[a] = fr ? cpl : 0.0;
          k.dinv64[a] = fr ? 1.0 / dsum : 0.0;
          k.d32[a] = fr ? (float)dsum : 1.0f;
          k.dinv32[a] = fr ? (float)(1.0 / dsum) : 0.0f;
        }
        const double bb = fr ? b : 0.0;
        const double r = fr ? bb - (dsum * k.phi64[a] - swphi[0]) : 0.0;
        k.b64[a] = bb;
        k.r64[a] = r;
        const double be = bb + (fr ? cpl : 0.0);
        part[0] = be * be;
        part[1] = r * r;
      }
      part[0] = warp_sum_d(part[0]);
      part[1] = warp_sum_d(part[1]);
      slice_partials64<2>(v, d.inst, v.slice_first[d.inst], v.slice_count[d.inst], ss.sg, part);
    }
    if (K > 1) __syncthreads();
    else __syncwarp();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[2];
      reduce_slices64<2>(v, i, v.slice_first[i], v.slice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        prep_decide(v.inst[i].ds, tot[0], tot[1]);
        instance_finished(v, i, 0, hc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// an instance's outer decision from ||r||^2 after a refinement (one thread)
__device__ __forceinline__ void refine_decide(DevState* ds, double rr) {
  if (!ds->outer_active) return;
  ds->rnorm2 = rr;
  ds->outer_it += 1;
  ds->outer_total += 1;
  const bool conv = rr <= ds->tol * ds->tol * ds->bnorm2;
  const bool go = !conv && ds->outer_it < ds->max_outer && ds->solve_iters < ds->max_iter && isfinite(rr) &&
                  !ds->wait_timeout;
  if (!go) {
    ds->cg_solves += 1;
    ds->last_relres = sqrt(rr / ds->bnorm2);
    if (!conv) ds->cg_nc += 1;
  }
  ds->outer_active = go ? 1 : 0;
}

// the refinement with K warps a slice (small cases): k_ir_slices below, the pairs of the parts'
// sums added in part order
template <int K>
__global__ void __launch_bounds__(kBlock) k_ir_split(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ float2 s_sum[kBlock];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.ncslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.cslices[have ? ss.sg : 0];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    float sh = 0.f, sl = 0.f;
    int a = -1;
    bool live = false;
    if (have && *((volatile int*)&k.ds->outer_active) != 0) {
      if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
      __syncwarp();
      a = k.cg_rows[__ldg(&d.row0) + lane];
      live = a >= 0 && k.freem[a];
      const int len = __any_sync(0xffffffffu, live) ? (k.cg_width[ss.sg - __ldg(&v.cslice_first[inst])] + 3) & ~3 : 0;
      const QuadPtr op(sell_cg_w(k, d), lane);
      const float4* wls = reinterpret_cast<const float4*>(k.sell_cg_lo + (size_t)(__ldg(&d.off) >> 5) * 32) + lane;
      for (int c0 = kResB * ss.part; c0 < len; c0 += kResB * K) {
        const int nc = min(kResB, len - c0);
        float w[kResB], wl[kResB], ev[kResB];
        unsigned int code[kResB];
        load_residual_quads(op, wls, c0, nc, w, wl, code);
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) ev[u] = __ldg(k.e32 + code_node(s_hb[warp], code[u]));
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) {
            float ph, pl;
            pair_mul(w[u], wl[u], ev[u], 0.0f, ph, pl);
            pair_add(sh, sl, ph, pl);
          }
      }
    }
    if (ss.part) s_sum[threadIdx.x] = make_float2(sh, sl);
    __syncthreads();
    if (have && ss.part == 0) {
#pragma unroll
      for (int h = 1; h < K; ++h) pair_add(sh, sl, s_sum[threadIdx.x + 32 * h].x, s_sum[threadIdx.x + 32 * h].y);
      float rh = 0.0f, rl = 0.0f;
      if (live) {
        const double ea = (double)k.e32[a];
        const double r = k.r64[a] - (k.dsum64[a] * ea - ((double)sh + (double)sl));
        k.r64[a] = r;
        const double ph = k.phi64[a] + ea;
        k.phi64[a] = ph;
        set_phi_rec(k, a, ph, true);
        pair_square(r, rh, rl);
      }
      pair_warp_sum(rh, rl);
      if (lane == 0) store_pair(v.partials, ss.sg, rh, rl);
    }
    __syncthreads();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        refine_decide(v.inst[i].ds, tot[0]);
        instance_finished(v, i, 0, hc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// FP64 path: phi += e on the unknowns, r -= A e, outer stop test
template <int K>
__global__ void __launch_bounds__(kBlock, 4) k_ir64(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ double s_acc[K > 1 ? kBlock : 1];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.ncslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.cslices[have ? ss.sg : 0];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    const int first = __ldg(&v.cslice_first[inst]);
    double sum[1] = {0.0};
    int a = -1;
    bool live = false;
    if (have && *((volatile int*)&k.ds->outer_active) != 0) {
      a = k.cg_rows[__ldg(&d.row0) + lane];
      live = a >= 0 && k.freem[a];
      if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
      __syncwarp();
      if (live) sum[0] = cg_row64<K>(k, d.off, (k.cg_width[ss.sg - first] + 3) >> 2, lane, ss.part, s_hb[warp], k.e64);
    }
    if (K > 1) split_sum<K, 1>(sum, s_acc);
    if (have && ss.part == 0) {
      double part[1] = {0.0};
      if (live) {
        const double ea = k.e64[a];
        const double r = k.r64[a] - (k.dsum64[a] * ea - sum[0]);
        k.r64[a] = r;
        const double ph = k.phi64[a] + ea;
        k.phi64[a] = ph;
        set_phi_rec(k, a, ph, false);
        part[0] = r * r;
      }
      part[0] = warp_sum_d(part[0]);
      slice_partials64<1>(v, inst, first, __ldg(&v.cslice_count[inst]), ss.sg, part);
    }
    if (K > 1) __syncthreads();
    else __syncwarp();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_slices64<1>(v, i, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        refine_decide(v.inst[i].ds, tot[0]);
        instance_finished(v, i, 0, hc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// refinement: phi += e on the unknowns, r -= A e (FP32 pairs of the FP64 weights times the
// FP32 correction), outer stop test
__global__ void __launch_bounds__(kBlock) k_ir_slices(EngineView v, cudaGraphConditionalHandle hc) {
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warps claim slices one at a time (slices of solid nodes, narrow and partial slices
  // cost less than full ones)
  for (int sg = claim_slice(v, lane); sg < v.ncslices; sg = claim_slice(v, lane)) {
    const SliceDesc& d = v.cslices[sg];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    float rh = 0.0f, rl = 0.0f;  // r.r of the slice as an FP32 pair
    if (*((volatile int*)&k.ds->outer_active) != 0) {
      if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
      __syncwarp();
      // the CG operator's slices: the correction e is zero off the unknowns
      const int a = k.cg_rows[__ldg(&d.row0) + lane];
      const bool live = a >= 0 && k.freem[a];
      const int len = __any_sync(0xffffffffu, live) ? (k.cg_width[sg - __ldg(&v.cslice_first[inst])] + 3) & ~3 : 0;
      const int* hb = s_hb[warp];
      const QuadPtr op(sell_cg_w(k, d), lane);
      const float4* wls = reinterpret_cast<const float4*>(k.sell_cg_lo + (size_t)(__ldg(&d.off) >> 5) * 32) + lane;
      const float* e = k.e32;
      float sh = 0.f, sl = 0.f;
      for (int c0 = 0; c0 < len; c0 += kResB) {
        const int nc = min(kResB, len - c0);
        float w[kResB], wl[kResB], ev[kResB];
        unsigned int code[kResB];
        load_residual_quads(op, wls, c0, nc, w, wl, code);
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) ev[u] = __ldg(e + code_node(hb, code[u]));
#pragma unroll
        for (int u = 0; u < kResB; ++u)
          if (u < nc) {
            float ph, pl;
            pair_mul(w[u], wl[u], ev[u], 0.0f, ph, pl);
            pair_add(sh, sl, ph, pl);
          }
      }
      if (live) {
        const double ea = (double)e[a];
        const double r = k.r64[a] - (k.dsum64[a] * ea - ((double)sh + (double)sl));
        k.r64[a] = r;
        const double ph = k.phi64[a] + ea;
        k.phi64[a] = ph;
        set_phi_rec(k, a, ph, true);
        pair_square(r, rh, rl);
      }
      __syncwarp();
    }
    pair_warp_sum(rh, rl);
    if (lane == 0) store_pair(v.partials, sg, rh, rl);
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[1];
      reduce_pair_items<1>(v.partials, v.stride, v.cslice_first[i], v.cslice_count[i], tot, sm);
      if (threadIdx.x == 0) {
        refine_decide(v.inst[i].ds, tot[0]);
        instance_finished(v, i, 0, hc);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      v.ticket[v.M + 1] = 0;
      v.ticket[v.M + 2] = 0;
    }
  }
}

// ------------------------------------------------------------------- transport -----------
__device__ __forceinline__ double dissolve_switch(double c0, double csat, double sw) {
  if (sw > 0.0) return 1.0 / (1.0 + exp(-(c0 - csat) / sw));
  return c0 > csat ? 1.0 : 0.0;
}

constexpr int kDiagSlots = 8;  // mass[4], solid, vol, dissolved, nonfinite

// Per-step diagnostics of one instance from its reduced transport partials (thread 0).
__device__ __forceinline__ void finish_instance(const KParams& k, const double (&tot)[kDiagSlots]) {
  DevState* ds = k.ds;
  for (int s = 0; s < S; ++s) ds->mass[s] = tot[s];
  ds->solid_count = (long long)tot[4];
  ds->steps += 1;
  if (k.dissolve_count) ds->dissolved += tot[6];
  if (tot[7] != 0.0) ds->nonfinite = 1;
  ds->mg_mass_now = tot[0];
  if (k.hist_m >= 3) {
    ds->hist_head = (ds->hist_head + 1) % k.hist_m;
    ds->hist_n = ds->hist_n < k.hist_m ? ds->hist_n + 1 : k.hist_m;
  }
  if (k.sub_step_no > 0 && ds->steps % k.sub_step_no == 0) {
    ds->voln1rel = ds->vol0rel != 0.0 ? tot[5] / ds->vol0rel : 0.0;
    ds->BV = pow(10., -k.vol_red * (1. - ds->voln1rel));  // utils.h:100-116
  }
}

// The solution of this step's solve and its image A x = b - r into the warm-start ring.
__device__ __forceinline__ void record_history(const KParams& k, int a, int hslot) {
  if (k.hist_m < 3) return;
  const size_t o = (size_t)hslot * k.N + a;
  k.xh[o] = k.phi64[a];
  k.bh[o] = k.freem[a] ? k.b64[a] - k.r64[a] : 0.0;
}

// Warm start of the next solve: phi = 2 phi^n - phi^{n-1} on the unknowns (phi_prev keeps
// phi^n); the returned value also goes into the next record so that both agree.  A node the
// previous transport turned liquid (its phi^{n-1} is the solid's) is not extrapolated.
__device__ __forceinline__ double next_phi_guess(const KParams& k, int a) {
  const double ph = k.phi64[a];
  if (k.phi_keep) k.phi_keep[a] = ph;  // the step's solved potential (forward_ckpt)
  if (!k.extrapolate || !k.freem[a] || k.flip_step[a] == (int)k.ds->steps) {
    k.phi_prev[a] = ph;
    return ph;
  }
  const double g = 2.0 * ph - k.phi_prev[a];
  k.phi_prev[a] = ph;
  k.phi64[a] = g;
  return g;
}

// A neighbour's whole 32-byte record (c[4] | phi_hi, phi_lo, phase, pad) in one 256-bit
// read-only load (records are 32-byte aligned): half the gather instructions and L1 requests
// of two 16-byte loads of the same sector.
__device__ __forceinline__ void ld_rec32(const float4* p, float4& c, float4& t) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w), "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
      : "l"(p));
}

// an FP64 record's concentrations and {phi, phase} in a 256-bit and a 128-bit read-only load
__device__ __forceinline__ void ld_rec64(const Rec64* p, double (&c)[S], double (&t)[2]) {
  const double* q = reinterpret_cast<const double*>(p);
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(c[0]), "=d"(c[1]), "=d"(c[2]), "=d"(c[3]) : "l"(q));
  asm("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(t[0]), "=d"(t[1]) : "l"(q + 4));
}

// Mixed transport of one 32-row slice sg.  RESID: write F_k = sum_KRk1 + sum_KRk2 - R_k
// (utils.h:177) to F_out (single instance) and change nothing; otherwise advance the state
// into rec32_nxt / clo and store the slice's diagnostics partials.  One lane per node streams
// the row's bond columns (codes and weights, column-major: one coalesced load per column) and
// gathers each neighbour's 32-byte record through rec(i), where i = hb[code >> 12] +
// (code & 4095) and hb[r] = gbase[r] - radj[r] (radj == nullptr: i is the node).  hb is the
// warp's 9-int table in shared memory.
// bond columns per batch of the FP32 transport, two quads: 128 registers, 2 CTAs an SM.  Weights
// and codes by the quad (16 and 8 bytes a lane) take 0.318 ms at 512k; by the column (4 and 2
// bytes, batches of 7) 0.358
constexpr int kTrB = 8;
template <bool RESID, int B, bool EARLY, bool PIPE, typename Rec>
__device__ __forceinline__ void transport_slice(const EngineView& v, int sg, int lane, int* hbw,
                                                const int* radj, Rec rec, double* F_out) {
  const SliceDesc& d = v.slices[sg];
  const KParams& k = v.inst[__ldg(&d.inst)];
  if (lane < 9) hbw[lane] = __ldg(&d.gbase[lane]) - (radj ? radj[lane] : 0);
  __syncwarp();
  float ph_hi[6], ph_lo[6];  // masses[4], solid volume sum, dissolved (FP32 pairs)
#pragma unroll
  for (int q = 0; q < 6; ++q) ph_hi[q] = ph_lo[q] = 0.0f;
  int n_solid = 0, n_bad = 0;
  const int a = __ldg(&d.row0) + lane;
  const bool rowok = lane < __ldg(&d.nrows);
  float a1[S], a2[S];
#pragma unroll
  for (int s = 0; s < S; ++s) a1[s] = a2[s] = 0.0f;
  int iface = 0;
  float4 ca = make_float4(0.0f, 0.0f, 0.0f, 0.0f), cb = ca;  // the node's record: c | phi_hi, phi_lo, phase, pad
  float pa = 0.0f;
  if (rowok) {
    const float4* rc = reinterpret_cast<const float4*>(k.rec32_cur);
    const double BV = *k.bv_ptr;
    float cLL[S], cX[S], cSS[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      cLL[s] = k.DLf[s];
      cX[s] = s == 0 ? (float)(k.DSo[0] * BV) : k.DSof[s];
      cSS[s] = s == 0 ? k.DSof[0] : 0.0f;
    }
    ca = rc[2 * a];
    cb = rc[2 * a + 1];
    pa = cb.z;
    // bond coefficient by the neighbour's phase (utils.h:100-153): liquid-liquid D_liquid,
    // mixed D_solid (BV for Mg), solid-solid D_solid for Mg only
    float cfL[S], cfS[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      cfL[s] = pa == 0.0f ? cLL[s] : cX[s];
      cfS[s] = pa == 0.0f ? cX[s] : cSS[s];
    }
    const QuadPtr op(sell_w(k, d), lane);
    const int len = k.row[a + 1] - k.row[a];
    // bonds in batches of B columns: the batch's streamed codes and weights, then its
    // neighbour records, all in flight before the arithmetic (column order is kept, so the
    // sums do not depend on the batch size)
    // PIPE: the next batch's codes and weights are loaded before the current batch's terms
    constexpr int QB = B / 4;
    float4 wn[PIPE ? QB : 1];
    uint2 coden[PIPE ? QB : 1];
    if (PIPE)
#pragma unroll
      for (int u = 0; u < QB; ++u)
        if (4 * u < len) {
          wn[PIPE ? u : 0] = op.weights(u);
          coden[PIPE ? u : 0] = op.codes(u);
        }
    for (int c0 = 0; c0 < len; c0 += B) {
      float4 wq[QB];
      uint2 cq[QB];
#pragma unroll
      for (int u = 0; u < QB; ++u)
        if (PIPE) {
          wq[u] = wn[PIPE ? u : 0];
          cq[u] = coden[PIPE ? u : 0];
        } else if (c0 + 4 * u < len) {
          wq[u] = op.weights((c0 >> 2) + u);
          cq[u] = op.codes((c0 >> 2) + u);
        }
      if (PIPE)
#pragma unroll
        for (int u = 0; u < QB; ++u)
          if (c0 + B + 4 * u < len) {
            wn[PIPE ? u : 0] = op.weights(((c0 + B) >> 2) + u);
            coden[PIPE ? u : 0] = op.codes(((c0 + B) >> 2) + u);
          }
      float w[B];
      unsigned int code[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        w[u] = quad_weight(wq[u >> 2], u & 3);
        code[u] = quad_code(cq[u >> 2], u & 3);
      }
      // EARLY: the batch's records all in flight before the arithmetic (L1/L2 latency);
      // otherwise each one just before its bond's terms (shared memory)
      float4 cn[EARLY ? B : 1], nb[EARLY ? B : 1];
      if (EARLY)
#pragma unroll
        for (int u = 0; u < B; ++u)
          if (c0 + u < len) rec(code_node(hbw, code[u]), cn[EARLY ? u : 0], nb[EARLY ? u : 0]);
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (c0 + u < len) {
          const int ur = EARLY ? u : 0;
          if (!EARLY) rec(code_node(hbw, code[u]), cn[0], nb[0]);
          const bool nsol = nb[ur].z != 0.0f;
          const float dphi = (nb[ur].x - cb.x) + (nb[ur].y - cb.y);
          iface |= (pa != 0.0f && !nsol) ? 1 : 0;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const float cw = (nsol ? cfS[s] : cfL[s]) * w[u];
            const float cns = sel4(cn[ur], s);
            a1[s] = fmaf(cw, cns - sel4(ca, s), a1[s]);
            a2[s] = fmaf(cw * cns, dphi, a2[s]);
          }
        }
    }
    const unsigned char dm = k.dirmask[a];
    const float4 lo4 = k.clo[a];
    const bool src_on = iface && !(dm & 1);
    const double swv = src_on ? dissolve_switch((double)ca.x + (double)lo4.x, k.csat, k.sw) : 0.0;
    const float Rmg = src_on ? (float)(-k.k_diss * swv) : 0.0f;
    const float* K1f = k.K1f;
    const float* K2f = k.K2zFf;
    if (RESID) {
#pragma unroll
      for (int s = 0; s < S; ++s)
        F_out[(size_t)s * k.N + a] =
            -(double)K1f[s] * a1[s] - (double)K2f[s] * a2[s] - (s == 0 ? (double)Rmg : 0.0);
    } else {
      // c + dt (K1 a1 + K2 a2 + R) on the compensated pair (hi, lo), renormalised: hi is
      // the FP32 rounding of the exact pair sum and lo its exact remainder
      const float dtf = k.dtf;
      float hi[S], lo[S];
      bool bad = false;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const float inc = dtf * (K1f[s] * a1[s] + K2f[s] * a2[s] + (s == 0 ? Rmg : 0.0f));
        float tt, e1, sh, e2;
        two_sum(sel4(lo4, s), inc, tt, e1);
        two_sum(sel4(ca, s), tt, sh, e2);
        two_sum(sh, e1 + e2, hi[s], lo[s]);
        if ((dm >> s) & 1) {
          const double x = k.bcval[(size_t)s * k.N + a];
          hi[s] = (float)x;
          lo[s] = (float)(x - (double)hi[s]);
        }
        // clamp c >= c_floor (main.cpp:805-837), compared on the normalised pairs
        if (hi[s] < k.cfl_hi || (hi[s] == k.cfl_hi && lo[s] < k.cfl_lo)) {
          hi[s] = k.cfl_hi;
          lo[s] = k.cfl_lo;
        }
        bad = bad || !isfinite(hi[s]);
      }
      float pnew = pa;
      // saturation test in FP64 (main.cpp:914-922)
      if (pa != 0.0f && (double)hi[0] + (double)lo[0] <= k.csat) {
        pnew = 0.0f;
        k.flip_step[a] = (int)(k.ds->steps + 1);
        k.flip_list[atomicAdd(&k.ds->nflip, 1)] = a;
        k.ds->op_valid = 0;
        k.ds->defl = 0;
      }
      record_history(k, a, k.hist_m >= 3 ? (k.ds->hist_head + 1) % k.hist_m : 0);
      const double g = next_phi_guess(k, a);
      Rec32 out;
#pragma unroll
      for (int s = 0; s < S; ++s) out.c[s] = hi[s];
      out.phi_hi = (float)g;
      out.phi_lo = (float)(g - (double)out.phi_hi);
      out.phase = pnew;
      out.pad = 0.0f;
      k.rec32_nxt[a] = out;
      k.clo[a] = make_float4(lo[0], lo[1], lo[2], lo[3]);
      // diagnostics as FP32 pairs: masses, solid volume sum (c_0 - CSat/CSolid), dissolved
#pragma unroll
      for (int s = 0; s < S; ++s) {
        ph_hi[s] = hi[s];
        ph_lo[s] = lo[s];
      }
      if (pnew != 0.0f) {
        n_solid = 1;
        float vs, ve;
        two_sum(hi[0], -k.csat_hi, vs, ve);
        ph_hi[4] = vs;
        ph_lo[4] = ve + (lo[0] - k.csat_lo);
      }
      if (src_on) {
        const double dv = k.k_diss * swv;
        ph_hi[5] = (float)dv;
        ph_lo[5] = (float)(dv - (double)ph_hi[5]);
      }
      n_bad = bad ? 1 : 0;
    }
  }
  __syncwarp();
  if (!RESID) {
#pragma unroll
    for (int q = 0; q < 6; ++q) pair_warp_sum(ph_hi[q], ph_lo[q]);
    n_solid = __reduce_add_sync(0xffffffffu, n_solid);
    n_bad = __reduce_add_sync(0xffffffffu, n_bad);
    if (lane == 0) {
      const size_t st = v.stride;
#pragma unroll
      for (int s = 0; s < S; ++s) store_pair(v.partials, s * st + sg, ph_hi[s], ph_lo[s]);
      store_pair(v.partials, 4 * st + sg, (float)n_solid, 0.0f);  // counts <= 32: exact
      store_pair(v.partials, 5 * st + sg, ph_hi[4], ph_lo[4]);
      store_pair(v.partials, 6 * st + sg, ph_hi[5], ph_lo[5]);
      store_pair(v.partials, 7 * st + sg, (float)n_bad, 0.0f);
    }
  }
}

// the transport's last CTA: every instance's diagnostics from its slices' partials, then
// the counters' reset
template <int BLK>
__device__ __forceinline__ void transport_last_cta(const EngineView& v, double* sm, int* s_last) {
  if (!take_last_ticket(&v.ticket[v.M + 1], s_last)) return;
  for (int i = 0; i < v.M; ++i) {
    double tot[kDiagSlots];
    reduce_pair_items<kDiagSlots, BLK>(v.partials, v.stride, v.slice_first[i], v.slice_count[i], tot, sm);
    if (threadIdx.x == 0) finish_instance(v.inst[i], tot);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    v.ticket[v.M + 1] = 0;
    v.ticket[v.M + 2] = 0;
  }
}

// Mixed transport, neighbour records gathered from L1/L2.  Warps claim slices one at a time
// (slices of solid nodes, narrow and partial slices cost less than full ones); the residual
// form, which has no last CTA to reset the counter, keeps the static split.
template <bool RESID>
__global__ void __launch_bounds__(kBlock, 2) k_transport32(EngineView v, double* F_out) {
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[kDiagSlots * kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr bool kClaim = !RESID;
  int s0, s1;
  if (kClaim) {
    s0 = claim_slice(v, lane);
    s1 = v.nslices;
  } else {
    warp_slices(v, &s0, &s1);
  }
  for (int sg = s0; sg < s1; sg = kClaim ? claim_slice(v, lane) : sg + 1) {
    const float4* rc = reinterpret_cast<const float4*>(v.inst[__ldg(&v.slices[sg].inst)].rec32_cur);
    transport_slice<RESID, kTrB, true, false>(v, sg, lane, s_hb[warp], nullptr,
                                 [rc](int n, float4& c, float4& t) { ld_rec32(rc + 2 * n, c, t); }, F_out);
  }
  if (RESID) return;
  transport_last_cta<kBlock>(v, sm, &s_last);
}

// Halo-staged mixed transport.  A CTA claims tiles one at a time; thread 0 copies the tile's
// halo records (its 9 halo rows: contiguous node ranges, 32-byte records) into shared memory
// by bulk copies on one mbarrier (a bounded wait: a timeout is recorded in the instance's state
// and reported as NNPP_ERR_CUDA), then the CTA's warps take the tile's slices and gather
// every neighbour's record from shared memory (its slot in the halo: the slice's window code
// rebased from the slice's window rows onto the tile's halo rows).  HBM and L2 see the
// streamed codes and weights and one copy of each halo; the per-bond gathers stay on chip.
constexpr int kTrHBlock = 128;
__host__ __device__ constexpr size_t smem_tr_halo(int halo_max) { return (size_t)halo_max * 32; }
// largest halo staged: two CTAs of 4 warps an SM at least
constexpr size_t kTrHaloSmemMax = 110 * 1024;

template <int B, bool PIPE, int MINB>
__global__ void __launch_bounds__(kTrHBlock, MINB) k_transport32h(EngineView v) {
  extern __shared__ __align__(16) float4 hrec[];  // 2 float4 a halo node
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_tile, s_stop, s_last;
  __shared__ int s_adj[9];  // halo row r: first node - its first slot
  __shared__ int s_hb[kTrHBlock / 32][12];
  __shared__ double sm[kDiagSlots * kTrHBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    s_stop = 0;
  }
  __syncthreads();
  unsigned phase = 0;
  for (;;) {
    if (threadIdx.x == 0) s_tile = s_stop ? v.ntiles : (int)atomicAdd(&v.ticket[v.M + 2], 1u);
    __syncthreads();
    const int t = s_tile;
    if (t >= v.ntiles) break;
    const TileDesc& td = v.tiles[t];
    const KParams& k = v.inst[td.inst];
    if (threadIdx.x == 0) {
      const float4* rc = reinterpret_cast<const float4*>(k.rec32_cur);
      unsigned bytes = 0;
      int acc = 0;
      for (int r = 0; r < 9; ++r) {
        s_adj[r] = td.hb[r] - acc;
        acc += td.hl[r];
        bytes += (unsigned)td.hl[r] * 32u;
      }
      // the previous tile's reads of the buffer come before the copies
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&bar, bytes);
      acc = 0;
      for (int r = 0; r < 9; ++r) {
        if (td.hl[r] > 0) bulk_g2s(hrec + 2 * acc, rc + 2 * (size_t)td.hb[r], (unsigned)td.hl[r] * 32u, &bar);
        acc += td.hl[r];
      }
    }
    __syncthreads();
    if (!mbar_wait_bounded(&bar, phase, kHaloWaitPolls)) {
      k.ds->wait_timeout = 1;
      s_stop = 1;
    }
    phase ^= 1u;
    const int nsl = (td.own_end - td.own_begin + 31) >> 5;
    for (int q = warp; q < nsl; q += kTrHBlock / 32)
      transport_slice<false, B, false, PIPE>(v, td.slice0 + q, lane, s_hb[warp], s_adj,
                                    [](int i, float4& c, float4& tt) {
                                      c = hrec[2 * i];
                                      tt = hrec[2 * i + 1];
                                    },
                                    nullptr);
    __syncthreads();
  }
  transport_last_cta<kTrHBlock>(v, sm, &s_last);
}

// Next-solve guess of the nodes a transport turned liquid.  As solids they carried no
// potential (zero); a potential solve started from that zero spends its first refinement
// sweeps on those few nodes.  Each listed node instead takes the w-weighted mean of the
// potentials that its liquid neighbours carry into the next solve, counting only neighbours
// that were liquid before this step (so every value read is one this pass does not write, and
// the result does not depend on the list's order), and the same value in every slot of the
// warm-start history, where the backward differences then vanish.  phi_prev keeps the step's
// potential (the adjoint's snapshots read it), and the next transport does not extrapolate
// these nodes.  Potential-Dirichlet nodes keep their boundary value.  The last CTA resets the
// count for the next transport.
template <typename P>
__global__ void __launch_bounds__(kBlock) k_flip_guess(EngineView v) {
  __shared__ int s_last;
  for (int i = 0; i < v.M; ++i) {
    const KParams& k = v.inst[i];
    const int n = k.ds->nflip;
    const int step_no = (int)k.ds->steps;  // the transport's last CTA has counted its step
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
      const int a = k.flip_list[q];
      if ((k.dirmask[a] >> S) & 1) continue;
      double sw = 0.0, swp = 0.0;
      for (int j = k.row[a]; j < k.row[a + 1]; ++j) {
        const int m = k.col[j];
        if (m == a || k.flip_step[m] == step_no) continue;
        const bool liq = sizeof(P) == 4 ? k.rec32_nxt[m].phase == 0.0f : k.rec64_nxt[m].phase == 0.0;
        if (!liq) continue;
        const double w = (double)k.w32[j];
        sw += w;
        swp += w * k.phi64[m];
      }
      if (!(sw > 0.0)) continue;
      const double g = swp / sw;
      k.phi64[a] = g;
      if constexpr (sizeof(P) == 4) {
        const float hi = (float)g;
        k.rec32_nxt[a].phi_hi = hi;
        k.rec32_nxt[a].phi_lo = (float)(g - (double)hi);
      } else {
        k.rec64_nxt[a].phi = g;
      }
      if (k.hist_m >= 3)
        for (int sl = 0; sl < k.hist_m; ++sl) k.xh[(size_t)sl * k.N + a] = g;
    }
  }
  if (take_last_ticket(&v.ticket[v.M + 3], &s_last) && threadIdx.x == 0) {
    for (int i = 0; i < v.M; ++i) v.inst[i].ds->nflip = 0;
    v.ticket[v.M + 3] = 0;
  }
}

// FP64 bond sums of the residual entry point (F_k = sum_KRk1 + sum_KRk2 - R_k, utils.h:177): CTA per
// tile, its halo staged in shared memory, W lanes a node
template <int W>
__global__ void __launch_bounds__(kBlock) k_residual64(EngineView v, double* F_out) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ TileSmem ts;
  const int sub = threadIdx.x % W, seg = threadIdx.x / W, nseg = kBlock / W;
  for (int item = blockIdx.x; item < v.ntiles; item += gridDim.x) {
    const TileDesc t = v.tiles[item];
    const KParams& k = v.inst[t.inst];
    load_tile(t, ts);
    double* hrec = reinterpret_cast<double*>(dsm);  // 6 doubles per halo node (SoA)
    const unsigned short* sslot = stage_slots(k.slot16, t, dsm + (size_t)6 * t.halo * sizeof(double));
    const Rec64* rc = k.rec64_cur;
    const int H = t.halo;
    for (int s = threadIdx.x; s < H; s += kBlock) {
      const Rec64 r = rc[halo_node(ts, s)];
#pragma unroll
      for (int q = 0; q < S; ++q) hrec[(size_t)q * H + s] = r.c[q];
      hrec[(size_t)S * H + s] = r.phi;
      hrec[(size_t)(S + 1) * H + s] = r.phase;
    }
    __syncthreads();
    const double BV = *k.bv_ptr;
    double cLL[S], cX[S], cSS[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      cLL[s] = k.DL[s];
      cX[s] = s == 0 ? k.DSo[0] * BV : k.DSo[s];
      cSS[s] = s == 0 ? k.DSo[0] : 0.0;
    }
    const int* row = k.row;
    const double* w64 = k.w64;
    const int own0 = ts.off[4] + (t.own_begin - t.hb[4]);
    for (int a0 = t.own_begin; a0 < t.own_end; a0 += nseg) {
      const int a = a0 + seg;
      const bool act = a < t.own_end;
      const int so = own0 + (a - t.own_begin);
      double ca[S], pha = 0.0, pa = 0.0;
#pragma unroll
      for (int s = 0; s < S; ++s) ca[s] = act ? hrec[(size_t)s * H + so] : 0.0;
      if (act) {
        pha = hrec[(size_t)S * H + so];
        pa = hrec[(size_t)(S + 1) * H + so];
      }
      double a1[S], a2[S];
#pragma unroll
      for (int s = 0; s < S; ++s) a1[s] = a2[s] = 0.0;
      int iface = 0;
      if (act) {
        for (int j = row[a] + sub; j < row[a + 1]; j += W) {
          const int sl = sslot[j - t.bond0];
          const double w = w64[j];
          const double pn = hrec[(size_t)(S + 1) * H + sl];
          const double dphi = hrec[(size_t)S * H + sl] - pha;
          const bool ll = (pa == 0.0) && (pn == 0.0);
          const bool ss = (pa != 0.0) && (pn != 0.0);
          iface |= (pa != 0.0 && pn == 0.0) ? 1 : 0;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const double coef = ll ? cLL[s] : (ss ? cSS[s] : cX[s]);
            const double cw = coef * w;
            const double cns = hrec[(size_t)s * H + sl];
            a1[s] += cw * (cns - ca[s]);
            a2[s] += cw * cns * dphi;
          }
        }
      }
#pragma unroll
      for (int s = 0; s < S; ++s) {
        a1[s] = seg_reduce_d<W>(a1[s]);
        a2[s] = seg_reduce_d<W>(a2[s]);
      }
      iface = seg_or<W>(iface);
      if (!act || sub != 0) continue;
      const unsigned char dm = k.dirmask[a];
      const bool src_on = iface && !(dm & 1);
      const double swv = src_on ? dissolve_switch(ca[0], k.csat, k.sw) : 0.0;
      const double Rmg = src_on ? -k.k_diss * swv : 0.0;
#pragma unroll
      for (int s = 0; s < S; ++s)
        F_out[(size_t)s * k.N + a] = -k.K1[s] * a1[s] - k.K2zF[s] * a2[s] - (s == 0 ? Rmg : 0.0);
    }
    __syncthreads();
  }
}

// FP64 transport (the plain FP64 path), one lane a row of the transport's slices, K warps a slice.
// A bond adds w (c_n - c_a) and w dphi c_n to the sums of its neighbour's phase (the bond
// coefficients follow from the two phases, utils.h:100-153, and multiply the sums at the end): 14
// FP64 instructions for the four species.  Bound by the FP64 pipe, which a warp-wide instruction
// holds for 64 cycles.  512k nodes 2.14 ms, against 3.78 with the
// coefficients multiplied into every bond (26 FP64 instructions).
template <int K>
__global__ void __launch_bounds__(kBlock, 1) k_transport64(EngineView v) {
  constexpr int NV = 4 * S;  // liquid: w d, w dphi c; solid: the same
  extern __shared__ __align__(16) unsigned char dsm[];
  double* s_sum = reinterpret_cast<double*>(dsm);  // kBlock * NV (K > 1)
  __shared__ int s_iface[kBlock];
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[kDiagSlots * kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = v.nslices;
  for (int base = blockIdx.x * SplitSlice<K>::kSlices; base < ns; base += gridDim.x * SplitSlice<K>::kSlices) {
    const SplitSlice<K> ss(base);
    const bool have = ss.sg < ns;
    const SliceDesc& d = v.slices[have ? ss.sg : 0];
    const int inst = __ldg(&d.inst);
    const KParams& k = v.inst[inst];
    if (lane < 9) s_hb[warp][lane] = d.gbase[lane];
    __syncwarp();
    const int* hb = s_hb[warp];
    const int a = d.row0 + lane;
    const bool rowok = have && lane < d.nrows;
    double sum[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) sum[q] = 0.0;
    double ca[S], pha = 0.0;
    int solid = 0, liquids = 0;
    if (rowok) {
      const Rec64* rc = k.rec64_cur;
      double pp[2];
      ld_rec64(rc + a, ca, pp);
      pha = pp[0];
      solid = __double2hiint(pp[1]) != 0;
      const int len = k.row[a + 1] - k.row[a];
      const QuadPtr op(sell_w(k, d), lane);
      const double* w64 = k.sell64 + (size_t)(d.off >> 5) * 32 + 4 * lane;
      for (int q = ss.part; 4 * q < len; q += K) {
        double w[4];
        const uint2 code = op.codes(q);
        ld_stream_d4(w64 + 128 * (size_t)q, w);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double cn[2][S], pn[2][2];
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (4 * q + 2 * h + t < len) ld_rec64(rc + code_node(hb, quad_code(code, 2 * h + t)), cn[t], pn[t]);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (4 * q + 2 * h + t >= len) continue;
            const double wt = w[2 * h + t];
            const double wd = wt * (pn[t][0] - pha);
            if (__double2hiint(pn[t][1]) == 0) {
              ++liquids;
#pragma unroll
              for (int s = 0; s < S; ++s) {
                sum[s] = fma(wt, cn[t][s] - ca[s], sum[s]);
                sum[S + s] = fma(wd, cn[t][s], sum[S + s]);
              }
            } else {
#pragma unroll
              for (int s = 0; s < S; ++s) {
                sum[2 * S + s] = fma(wt, cn[t][s] - ca[s], sum[2 * S + s]);
                sum[3 * S + s] = fma(wd, cn[t][s], sum[3 * S + s]);
              }
            }
          }
        }
      }
    }
    if (K > 1) {
      s_iface[threadIdx.x] = liquids;
      split_sum<K, NV>(sum, s_sum);
    }
    if (have && ss.part == 0) {
      if (K > 1)
        for (int h = 1; h < K; ++h) liquids += s_iface[threadIdx.x + 32 * h];
      double part[kDiagSlots];
#pragma unroll
      for (int q = 0; q < kDiagSlots; ++q) part[q] = 0.0;
      if (rowok) {
        const unsigned char dm = k.dirmask[a];
        const bool src_on = solid && liquids > 0 && !(dm & 1);
        const double swv = src_on ? dissolve_switch(ca[0], k.csat, k.sw) : 0.0;
        const double Rmg = src_on ? -k.k_diss * swv : 0.0;
        double val[S];
        bool bad = false;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const double cX = s == 0 ? k.DSo[0] * *k.bv_ptr : k.DSo[s];
          const double cL = solid ? cX : k.DL[s], cS = solid ? (s == 0 ? k.DSo[0] : 0.0) : cX;
          const double a1 = cL * sum[s] + cS * sum[2 * S + s], a2 = cL * sum[S + s] + cS * sum[3 * S + s];
          const double F = -k.K1[s] * a1 - k.K2zF[s] * a2 - (s == 0 ? Rmg : 0.0);
          double x = ca[s] - k.dt * F;
          if ((dm >> s) & 1) x = k.bcval[(size_t)s * k.N + a];
          if (x < k.c_floor) x = k.c_floor;
          if (!isfinite(x)) bad = true;
          val[s] = x;
        }
        double pnew = solid ? 1.0 : 0.0;
        if (solid && val[0] <= k.csat) {
          pnew = 0.0;
          k.flip_step[a] = (int)(k.ds->steps + 1);
          k.flip_list[atomicAdd(&k.ds->nflip, 1)] = a;
          k.ds->op_valid = 0;
          k.ds->defl = 0;
        }
        record_history(k, a, k.hist_m >= 3 ? (k.ds->hist_head + 1) % k.hist_m : 0);
        const double g = next_phi_guess(k, a);
        Rec64 out;
#pragma unroll
        for (int s = 0; s < S; ++s) out.c[s] = val[s];
        out.phi = g;
        out.phase = pnew;
        out.pad[0] = out.pad[1] = 0.0;
        k.rec64_nxt[a] = out;
#pragma unroll
        for (int s = 0; s < S; ++s) part[s] = val[s];
        if (pnew != 0.0) {
          part[4] = 1.0;
          part[5] = val[0] - k.csat;
        }
        part[6] = k.k_diss * swv;
        part[7] = bad ? 1.0 : 0.0;
      }
      static_assert(kDiagSlots == 8, "warp_sums8");
      warp_sums8(part);
      slice_partials64<kDiagSlots>(v, inst, __ldg(&v.slice_first[inst]), __ldg(&v.slice_count[inst]), ss.sg, part);
    }
    if (K > 1) __syncthreads();
    else __syncwarp();
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[kDiagSlots];
      reduce_slices64<kDiagSlots>(v, i, v.slice_first[i], v.slice_count[i], tot, sm);
      if (threadIdx.x == 0) finish_instance(v.inst[i], tot);
      __syncthreads();
    }
    if (threadIdx.x == 0) v.ticket[v.M + 1] = 0;
  }
}

// ------------------------------------------------------------------- state transfer -----
__global__ void k_load_state(KParams k, const int* perm, const double* c_user, const double* phi_user,
                             const int* phase_user, int mixed, int dirichlet_phi, int keep_history) {
  const int N = k.N;
  // the history pairs (x, A x) stay valid guesses for the same operator; a new state
  // starts without them unless the caller continues a run (nnpp_step_host)
  if (blockIdx.x == 0 && threadIdx.x == 0 && !keep_history) k.ds->hist_n = 0;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += gridDim.x * blockDim.x) {
    const int u = perm[a];
    double c[S];
    for (int s = 0; s < S; ++s) c[s] = c_user[(size_t)s * N + u];
    double phi = phi_user ? phi_user[u] : k.phi_prev[a];
    if (dirichlet_phi && ((k.dirmask[a] >> S) & 1)) phi = k.bcval[(size_t)S * N + a];
    const float ph_old = mixed ? k.rec32_cur[a].phase : (float)k.rec64_cur[a].phase;
    const float ph = phase_user ? (phase_user[u] != 0 ? 1.0f : 0.0f) : ph_old;
    if (ph != ph_old) {  // a new liquid mask: the prep recomputes the diagonal, no deflation
      k.ds->op_valid = 0;
      k.ds->defl = 0;
    }
    k.phi64[a] = phi;
    k.phi_prev[a] = phi;
    if (mixed) {
      Rec32 r;
      float lo[S];
      for (int s = 0; s < S; ++s) {
        r.c[s] = (float)c[s];
        lo[s] = (float)(c[s] - (double)r.c[s]);
      }
      r.phi_hi = (float)phi;
      r.phi_lo = (float)(phi - (double)r.phi_hi);
      r.phase = ph;
      r.pad = 0.0f;
      k.rec32_cur[a] = r;
      k.clo[a] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    } else {
      Rec64 r;
      for (int s = 0; s < S; ++s) r.c[s] = c[s];
      r.phi = phi;
      r.phase = ph;
      r.pad[0] = r.pad[1] = 0.0;
      k.rec64_cur[a] = r;
    }
  }
}

// The potential of the last solve is phi_prev (after a step phi64 holds the next warm
// start; before any step both agree).
__global__ void k_store_state(KParams k, const int* perm, double* c_user, double* phi_user,
                              int* phase_user, int mixed) {
  const int N = k.N;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += gridDim.x * blockDim.x) {
    const int u = perm[a];
    if (mixed) {
      const Rec32 r = k.rec32_cur[a];
      const float4 lo = k.clo[a];
      if (c_user)
        for (int s = 0; s < S; ++s) c_user[(size_t)s * N + u] = (double)r.c[s] + (double)sel4(lo, s);
      if (phase_user) phase_user[u] = r.phase != 0.0f ? 1 : 0;
    } else {
      const Rec64 r = k.rec64_cur[a];
      if (c_user)
        for (int s = 0; s < S; ++s) c_user[(size_t)s * N + u] = r.c[s];
      if (phase_user) phase_user[u] = r.phase != 0.0 ? 1 : 0;
    }
    if (phi_user) phi_user[u] = k.phi_prev[a];
  }
}

// convert the current state between the two representations
__global__ void k_convert(KParams k, int to_mixed) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    if (to_mixed) {
      const Rec64 s64 = k.rec64_cur[a];
      Rec32 r;
      float lo[S];
      for (int s = 0; s < S; ++s) {
        r.c[s] = (float)s64.c[s];
        lo[s] = (float)(s64.c[s] - (double)r.c[s]);
      }
      r.phi_hi = (float)s64.phi;
      r.phi_lo = (float)(s64.phi - (double)r.phi_hi);
      r.phase = (float)s64.phase;
      r.pad = 0.0f;
      k.rec32_cur[a] = r;
      k.clo[a] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    } else {
      const Rec32 s32 = k.rec32_cur[a];
      const float4 lo = k.clo[a];
      Rec64 r;
      for (int s = 0; s < S; ++s) r.c[s] = (double)s32.c[s] + (double)sel4(lo, s);
      r.phi = (double)s32.phi_hi + (double)s32.phi_lo;
      r.phase = (double)s32.phase;
      r.pad[0] = r.pad[1] = 0.0;
      k.rec64_cur[a] = r;
    }
  }
}

// initial diagnostics (main.cpp:472-480): solid count, vol0rel, masses; restart != 0 keeps
// vol0rel and the initial Mg mass and recomputes the relative volume of the current state
// instead (main.cpp:527-533, after a restart from file)
__global__ void k_init_diag(KParams k, int mixed, double* partials, int restart) {
  __shared__ double sm[7 * kBlock / 32];
  __shared__ int s_last;
  double part[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    double c[S];
    float ph;
    if (mixed) {
      const Rec32 r = k.rec32_cur[a];
      const float4 lo = k.clo[a];
      for (int s = 0; s < S; ++s) c[s] = (double)r.c[s] + (double)sel4(lo, s);
      ph = r.phase;
    } else {
      const Rec64 r = k.rec64_cur[a];
      for (int s = 0; s < S; ++s) c[s] = r.c[s];
      ph = (float)r.phase;
    }
    for (int s = 0; s < S; ++s) part[s] += c[s];
    if (ph != 0.0f) {
      part[4] += 1.0;
      part[5] += c[0] - k.csat;
    }
  }
  block_sum<7, kBlock>(part, sm);
  if (threadIdx.x == 0)
    for (int q = 0; q < 7; ++q) partials[q * gridDim.x + blockIdx.x] = part[q];
  if (!take_last_ticket(&k.ds->ticket[0], &s_last)) return;
  double tot[7];
  reduce_partials<7, kBlock>(partials, gridDim.x, tot, sm);
  if (threadIdx.x == 0) {
    DevState* ds = k.ds;
    ds->ticket[0] = 0;
    for (int s = 0; s < S; ++s) ds->mass[s] = tot[s];
    ds->mg_mass_now = tot[0];
    ds->solid_count = (long long)tot[4];
    if (restart) {
      ds->voln1rel = ds->vol0rel != 0.0 ? tot[5] / ds->vol0rel : 0.0;
    } else {
      ds->mg_mass_t0 = tot[0];
      ds->vol0rel = tot[5];
      ds->voln1rel = 0.0;
    }
    ds->BV = pow(10., -k.vol_red * (1. - ds->voln1rel));
  }
}

template <typename F>
nnpp_status dispatch_lanes(int lanes, F&& f) {
  switch (lanes) {
    case 4: return f(std::integral_constant<int, 4>());
    case 8: return f(std::integral_constant<int, 8>());
    case 16: return f(std::integral_constant<int, 16>());
    default: return set_error(NNPP_ERR_INVALID, "lanes per node must be 4, 8 or 16");
  }
}

// Persistent grid: as many CTAs as fit on the device at once (at most one per item).
template <typename K>
int occ_grid_b(K kern, int block, size_t smem, int sms, int items) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, block, smem) != cudaSuccess) {
    cudaGetLastError();
    nb = 1;
  }
  if (nb < 1) nb = 1;
  const int g = sms * nb;
  return items < g ? (items > 0 ? items : 1) : g;
}

template <typename K>
int occ_grid(K kern, size_t smem, int sms, int items) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kBlock, smem) != cudaSuccess) {
    cudaGetLastError();
    nb = 1;
  }
  if (nb < 1) nb = 1;
  const int g = sms * nb;
  return items < g ? (items > 0 ? items : 1) : g;
}

// Grid of a slice kernel with several CTAs per SM: as many 8-warp CTAs as give every warp
// the same number of slices (the fewest rounds the resident warps need), so that no warp
// idles a whole slice at the end while the others of its CTA finish a second one.
template <typename K>
int slice_grid(K kern, size_t smem, int sms, int nslices) {
  const int g = occ_grid(kern, smem, sms, (nslices + 7) / 8);
  const int rounds = (nslices + 8 * g - 1) / (8 * g);
  const int g2 = (nslices + 8 * rounds - 1) / (8 * rounds);
  return g2 < 1 ? 1 : g2;
}

// kernels whose warps claim slices: as many CTAs as the SMs hold at once (fewer when the
// slices are fewer than the warps)
template <typename K>
int claim_grid(K kern, size_t smem, int sms, int nslices) {
  return occ_grid(kern, smem, sms, (nslices + 7) / 8);
}

size_t smem_slots(int B) { return (size_t)(B + 16) * sizeof(unsigned short); }
size_t smem_prep(int H, int B) { return align16((size_t)H * (sizeof(double) + 1)) + smem_slots(B); }
size_t smem_transport64() { return (size_t)kBlock * 4 * S * sizeof(double); }
size_t smem_spmv_staged() { return kTmaRingBytes + kTmaWinBytes + kTmaBarBytes; }
// streamed operator: the deepest ring (2..4 stages) that fits beside windows of win_cap nodes
constexpr size_t kSmemCta = 225 * 1024;
// stages of kStreamCol columns (2 .. kStreamMaxStages)
constexpr int kStreamCol = 32;
constexpr int kStreamMaxStages = 4;
size_t smem_spmv_stream(int win_cap, int* stages) {
  const size_t win = (size_t)kWarpsCta * 2 * win_cap * sizeof(float) + (size_t)kWarpsCta * kDescRing * sizeof(SliceDesc);
  const size_t sb = (size_t)kStreamCol * kSellW * 4 + sizeof(uint64_t);
  int st = kStreamMaxStages;
  while (st > 2 && (size_t)kWarpsCta * st * sb + win > kSmemCta) --st;
  *stages = st;
  return (size_t)kWarpsCta * st * sb + win;
}
size_t smem_spmv_win() { return (size_t)(kBlock / 32) * kWinCap * sizeof(float); }
size_t smem_tr64(int H, int B) { return (size_t)H * 6 * sizeof(double) + smem_slots(B); }
size_t smem_adj(int H, int B) { return align16((size_t)H * (9 * sizeof(double) + 1)) + smem_slots(B) + 16; }

template <typename K>
nnpp_status allow_smem(K kern, size_t bytes) {
  if (bytes > 32 * 1024)  // the default limit counts static shared memory too
    NNPP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return NNPP_OK;
}

// ------------------------------------------------------------------- adjoint -------------
// Transpose of one explicit step (FP64).  For node m, with lh = lambda^{n+1} masked to zero
// on Dirichlet and clamped entries, a = dt K1 D w and b = dt K2 z F/(RT) D w:
//   mu_k,m = lh_k,m + sum_i a (lh_k,i - lh_k,m) + sum_i lh_k,i b (phi_m - phi_i)
//            [+ lh_0,m (-dt k S'(c_0,m)) on interface nodes]
//   nu_m   = sum_k dt K2zF_k (c_k,m sum_i D w lh_k,i - lh_k,m sum_i D w c_k,i)   (d/dphi)
// and the parameter sensitivities dL/dD_k = sum_m lh_k,m (transport increment)/D_k,
// dL/dk = sum_m lh_0,m (-dt S(c_0,m)) over interface nodes.  The bond terms are the
// off-diagonal weights of the reference's tangent (utils.h:955-963), applied transposed.
struct AdjArgs {
  const Rec64* snap;   // c^n, phi^n, phase^n
  const Rec64* snap1;  // c^{n+1} (clamp mask)
  const double* lam;   // lambda^{n+1}, S*N
  double* mu;          // S*N
  double* nu;          // N
  double* acc;         // 5 accumulators (dL/dD_k, dL/dk)
};

__device__ __forceinline__ double pair_D(const KParams& k, int s, bool pm, bool pi) {
  if (!pm && !pi) return k.DL[s];
  if (s == 0) return k.DSo[0];  // BV = 1: the adjoint requires vol_red = 0
  if (pm && pi) return 0.0;
  return k.DSo[s];
}

template <int W>
__global__ void __launch_bounds__(kBlock) k_adj_transport(EngineView v, AdjArgs ad) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ TileSmem ts;
  __shared__ double sm[5 * kBlock / 32];
  __shared__ int s_last;
  const int sub = threadIdx.x % W, seg = threadIdx.x / W, nseg = kBlock / W;
  for (int item = blockIdx.x; item < v.ntiles; item += gridDim.x) {
    const TileDesc t = v.tiles[item];
    const KParams& k = v.inst[t.inst];
    load_tile(t, ts);
    const int H = t.halo;
    const int N = k.N;
    double* hc = reinterpret_cast<double*>(dsm);  // c: S*H
    double* hl = hc + (size_t)S * H;              // masked lambda: S*H
    double* hphi = hl + (size_t)S * H;            // H
    unsigned char* hph = reinterpret_cast<unsigned char*>(hphi + H);
    const unsigned short* sslot = stage_slots(k.slot16, t, dsm + align16((size_t)9 * H * sizeof(double) + H));
    for (int s = threadIdx.x; s < H; s += kBlock) {
      const int n = halo_node(ts, s);
      const Rec64 r = ad.snap[n];
      const Rec64 r1 = ad.snap1[n];
      const unsigned char dm = k.dirmask[n];
#pragma unroll
      for (int q = 0; q < S; ++q) {
        hc[(size_t)q * H + s] = r.c[q];
        const bool zero = ((dm >> q) & 1) || r1.c[q] == k.c_floor;
        hl[(size_t)q * H + s] = zero ? 0.0 : ad.lam[(size_t)q * N + n];
      }
      hphi[s] = r.phi;
      hph[s] = r.phase != 0.0 ? 1 : 0;
    }
    __syncthreads();
    const int* row = k.row;
    const double* w64 = k.w64;
    const double dt = k.dt;
    const int own0 = ts.off[4] + (t.own_begin - t.hb[4]);
    double part[5] = {0, 0, 0, 0, 0};
    for (int a0 = t.own_begin; a0 < t.own_end; a0 += nseg) {
      const int a = a0 + seg;
      const bool act = a < t.own_end;
      const int so = own0 + (a - t.own_begin);
      double cm[S], lm[S];
      double phm = 0.0;
      bool pm = false;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        cm[q] = act ? hc[(size_t)q * H + so] : 0.0;
        lm[q] = act ? hl[(size_t)q * H + so] : 0.0;
      }
      if (act) {
        phm = hphi[so];
        pm = hph[so] != 0;
      }
      double acc[S], a1[S], a2[S], sl[S], sc[S];
#pragma unroll
      for (int q = 0; q < S; ++q) acc[q] = a1[q] = a2[q] = sl[q] = sc[q] = 0.0;
      int iface = 0;
      if (act) {
        for (int j = row[a] + sub; j < row[a + 1]; j += W) {
          const int si = sslot[j - t.bond0];
          const double w = w64[j];
          const bool pi = hph[si] != 0;
          const double phi_i = hphi[si];
          iface |= (pm && !pi) ? 1 : 0;
#pragma unroll
          for (int q = 0; q < S; ++q) {
            const double Dw = pair_D(k, q, pm, pi) * w;
            const double li = hl[(size_t)q * H + si];
            const double ci = hc[(size_t)q * H + si];
            acc[q] += dt * k.K1[q] * Dw * (li - lm[q]) + li * dt * k.K2zF[q] * Dw * (phm - phi_i);
            a1[q] += Dw * (ci - cm[q]);
            a2[q] += Dw * ci * (phi_i - phm);
            sl[q] += Dw * li;
            sc[q] += Dw * ci;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < S; ++q) {
        acc[q] = seg_reduce_d<W>(acc[q]);
        a1[q] = seg_reduce_d<W>(a1[q]);
        a2[q] = seg_reduce_d<W>(a2[q]);
        sl[q] = seg_reduce_d<W>(sl[q]);
        sc[q] = seg_reduce_d<W>(sc[q]);
      }
      iface = seg_or<W>(iface);
      if (!act || sub != 0) continue;
      const bool src = iface && !(k.dirmask[a] & 1);
      double nu = 0.0;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        double m = lm[q] + acc[q];
        if (q == 0 && src) {
          const double sw = dissolve_switch(cm[0], k.csat, k.sw);
          const double dsw = k.sw > 0.0 ? sw * (1.0 - sw) / k.sw : 0.0;
          m += lm[0] * (-dt * k.k_diss * dsw);
          part[4] += lm[0] * (-dt * sw);
        }
        ad.mu[(size_t)q * N + a] = m;
        nu += dt * k.K2zF[q] * (cm[q] * sl[q] - lm[q] * sc[q]);
        part[q] += lm[q] * dt * (k.K1[q] * a1[q] + k.K2zF[q] * a2[q]) / k.DL[q];
      }
      ad.nu[a] = nu;
    }
    write_partials<5>(v, item, part, sm);
    if (item_done(&v.ticket[t.inst], v.tile_count[t.inst], &s_last)) {
      double tot[5];
      reduce_items<5>(v.partials, v.stride, v.tile_first[t.inst], v.tile_count[t.inst], tot, sm);
      if (threadIdx.x == 0) {
        for (int q = 0; q < 5; ++q) ad.acc[q] += tot[q];
        v.ticket[t.inst] = 0;
      }
    }
    __syncthreads();
  }
}

// Mixed adjoint transport: the same transpose in FP32 on the sliced operator.  k_adj_pack
// writes per node the 48-byte record {c[4], masked lambda[4], phi_hi, phi_lo, phase, 0};
// k_adj_transport32 streams the slices (one lane per node), gathers the neighbours' records
// from L1/L2, forms the differences directly (no cancellation of large sums) and
// accumulates the parameter sensitivities as FP32 pairs.
__global__ void k_adj_pack(KParams k, const Rec64* snap, const Rec64* snap1, const double* lam,
                           float4* rec) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    const Rec64 r = snap[a];
    const Rec64 r1 = snap1[a];
    const unsigned char dm = k.dirmask[a];
    float lh[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      const bool zero = ((dm >> q) & 1) || r1.c[q] == k.c_floor;
      lh[q] = zero ? 0.0f : (float)lam[(size_t)q * k.N + a];
    }
    const float ph = (float)r.phi;
    rec[3 * a] = make_float4((float)r.c[0], (float)r.c[1], (float)r.c[2], (float)r.c[3]);
    rec[3 * a + 1] = make_float4(lh[0], lh[1], lh[2], lh[3]);
    rec[3 * a + 2] = make_float4(ph, (float)(r.phi - (double)ph), r.phase != 0.0 ? 1.0f : 0.0f, 0.0f);
  }
}

// bond columns per batch of the FP32 adjoint transport: 4 at 127 registers (2 CTAs an SM);
// the 400-step backward of the 262k calibration workload took 1014 ms against 1059 with 2
constexpr int kAdjB = 4;
template <int W>
__global__ void __launch_bounds__(kBlock, 2) k_adj_transport32(EngineView v, const float4* rec,
                                                               double* mu, double* nu, double* acc) {
  __shared__ int s_hb[kBlock / 32][12];
  __shared__ double sm[5 * kBlock / 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warps claim slices one at a time (slices of solid nodes, narrow and partial slices
  // cost less than full ones)
  for (int sg = claim_slice(v, lane); sg < v.nslices; sg = claim_slice(v, lane)) {
    const SliceDesc d = v.slices[sg];
    const KParams& k = v.inst[d.inst];
    if (lane < 9) s_hb[warp][lane] = v.slices[sg].gbase[lane];
    __syncwarp();
    float gh[5], gl[5];  // dL/dD_k (4), dL/dk as FP32 pairs
#pragma unroll
    for (int q = 0; q < 5; ++q) gh[q] = gl[q] = 0.0f;
    const int a = d.row0 + lane;
    if (lane < d.nrows) {
      const int* hb = s_hb[warp];
      const float4 cm4 = rec[3 * a], lm4 = rec[3 * a + 1], pm4 = rec[3 * a + 2];
      const bool pm = pm4.z != 0.0f;
      float cfL[S], cfS[S];  // pair coefficient for a liquid / solid neighbour (BV = 1)
#pragma unroll
      for (int q = 0; q < S; ++q) {
        const float dl = k.DLf[q], ds = k.DSof[q];
        cfL[q] = pm ? ds : dl;
        cfS[q] = pm ? (q == 0 ? ds : 0.0f) : ds;
      }
      float A1[S], A2[S], a1[S], a2[S], sl[S], sc[S];
#pragma unroll
      for (int q = 0; q < S; ++q) A1[q] = A2[q] = a1[q] = a2[q] = sl[q] = sc[q] = 0.0f;
      int iface = 0;
      const QuadPtr op(sell_w(k, d), lane);
      const int len = k.row[a + 1] - k.row[a];
      // bonds in batches of kAdjB columns (codes, weights and records in flight together;
      // the column order of the sums is kept)
      for (int c0 = 0; c0 < len; c0 += kAdjB) {
        static_assert(kAdjB == 4, "the adjoint's batch is a quad");
        const float4 wq = op.weights(c0 >> 2);
        const uint2 cq = op.codes(c0 >> 2);
        float wv[kAdjB];
        unsigned int code[kAdjB];
#pragma unroll
        for (int u = 0; u < kAdjB; ++u) {
          wv[u] = quad_weight(wq, u);
          code[u] = quad_code(cq, u);
        }
        float4 cnv[kAdjB], lnv[kAdjB], pnv[kAdjB];
#pragma unroll
        for (int u = 0; u < kAdjB; ++u)
          if (c0 + u < len) {
            const int n = code_node(hb, code[u]);
            cnv[u] = __ldg(rec + 3 * n);
            lnv[u] = __ldg(rec + 3 * n + 1);
            pnv[u] = __ldg(rec + 3 * n + 2);
          }
#pragma unroll
        for (int u = 0; u < kAdjB; ++u)
          if (c0 + u < len) {
            const float w = wv[u];
            const float4 cn = cnv[u], ln = lnv[u], pn = pnv[u];
            const bool nsol = pn.z != 0.0f;
            iface |= (pm && !nsol) ? 1 : 0;
            const float dphi = (pm4.x - pn.x) + (pm4.y - pn.y);  // phi_m - phi_i
#pragma unroll
            for (int q = 0; q < S; ++q) {
              const float Dw = (nsol ? cfS[q] : cfL[q]) * w;
              const float li = sel4(ln, q), ci = sel4(cn, q);
              A1[q] = fmaf(Dw, li - sel4(lm4, q), A1[q]);
              a1[q] = fmaf(Dw, ci - sel4(cm4, q), a1[q]);
              const float tl = Dw * li, tc = Dw * ci;
              A2[q] = fmaf(tl, dphi, A2[q]);
              a2[q] = fmaf(-tc, dphi, a2[q]);
              sl[q] += tl;
              sc[q] += tc;
            }
          }
      }
      const unsigned char dm = k.dirmask[a];
      const bool src = iface && !(dm & 1);
      const float dt = k.dtf;
      float nu_a = 0.0f;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        const float K1 = k.K1f[q], K2 = k.K2zFf[q];
        const float lmq = sel4(lm4, q), cmq = sel4(cm4, q);
        float m = lmq + dt * (K1 * A1[q] + K2 * A2[q]);
        if (q == 0 && src) {
          const double swd = dissolve_switch((double)cm4.x, k.csat, k.sw);
          const double dsw = k.sw > 0.0 ? swd * (1.0 - swd) / k.sw : 0.0;
          m += lmq * (float)(-k.dt * k.k_diss * dsw);
          const float gk = lmq * (float)(-k.dt * swd);
          float ek;
          two_sum(gh[4], gk, gh[4], ek);
          gl[4] += ek;
        }
        mu[(size_t)q * k.N + a] = (double)m;
        nu_a = fmaf(dt * K2, cmq * sl[q] - lmq * sc[q], nu_a);
        const float gq = lmq * dt * (K1 * a1[q] + K2 * a2[q]) / k.DLf[q];
        float e;
        two_sum(gh[q], gq, gh[q], e);
        gl[q] += e;
      }
      nu[a] = (double)nu_a;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 5; ++q) pair_warp_sum(gh[q], gl[q]);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < 5; ++q) store_pair(v.partials, (size_t)q * v.stride + sg, gh[q], gl[q]);
  }
  if (take_last_ticket(&v.ticket[v.M + 1], &s_last)) {
    for (int i = 0; i < v.M; ++i) {
      double tot[5];
      reduce_pair_items<5>(v.partials, v.stride, v.slice_first[i], v.slice_count[i], tot, sm);
      if (threadIdx.x == 0)
        for (int q = 0; q < 5; ++q) acc[q] += tot[q];
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      v.ticket[v.M + 1] = 0;
      v.ticket[v.M + 2] = 0;
    }
  }
}

// lambda^n = mu + (1/(K sigma)) F CSolid z_k psi on the unknowns, + the loss injection on
// species 0 (d(mass loss)/dc_0 = -dV times dL/d(sample))
__global__ void k_adj_combine(KParams k, const double* mu, double* lam, double inject) {
  const int N = k.N;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < N; a += gridDim.x * blockDim.x) {
    const double psi = k.freem[a] ? k.phi64[a] : 0.0;
    for (int s = 0; s < S; ++s)
      lam[(size_t)s * N + a] = mu[(size_t)s * N + a] + k.lam * k.z[s] * psi + (s == 0 ? inject : 0.0);
  }
}

// snapshot c and phase of the current state (either representation)
__global__ void k_snap_state(KParams k, Rec64* dst, int mixed) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    Rec64 r = dst[a];
    if (mixed) {
      const Rec32 s32 = k.rec32_cur[a];
      const float4 lo = k.clo[a];
      for (int s = 0; s < S; ++s) r.c[s] = (double)s32.c[s] + (double)sel4(lo, s);
      r.phase = (double)s32.phase;
    } else {
      const Rec64 s64 = k.rec64_cur[a];
      for (int s = 0; s < S; ++s) r.c[s] = s64.c[s];
      r.phase = s64.phase;
    }
    dst[a] = r;
  }
}

// Recomputation without the potential solve: a step's solved potential (stored by
// forward_ckpt) as the solve leaves it -- phi64 and the current records' potential (the
// FP32 pair as set_phi_rec writes it) -- and into the step's snapshot.  On the nodes the
// solve does not change the stored value is the one the records already hold.
__global__ void k_load_phi(KParams k, const double* phi, Rec64* snap, int mixed) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    const double ph = phi[a];
    k.phi64[a] = ph;
    set_phi_rec(k, a, ph, mixed != 0);
    snap[a].phi = ph;
  }
}

// phi^n (the last solve's potential) into a snapshot
__global__ void k_snap_phi(KParams k, Rec64* dst) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x)
    dst[a].phi = k.phi_prev[a];
}

// adjoint solve set-up: phase^n into the current records, warm start psi (0 on Dirichlet
// and solid nodes).  The operator arrays stay valid where the previous adjoint solve's phases were the
// same (most steps: forming them takes 0.21 ms of 262k nodes against 0.09 for a pass that uses them).
__global__ void k_adj_solve_setup(KParams k, const Rec64* snap, const double* psi_prev, int mixed) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
    const double ph = snap[a].phase;
    if ((mixed ? (double)k.rec32_cur[a].phase : k.rec64_cur[a].phase) != ph) k.ds->op_valid = 0;
    k.rec32_cur[a].phase = (float)ph;
    k.rec64_cur[a].phase = ph;
    const bool zero = ph != 0.0 || ((k.dirmask[a] >> S) & 1);
    const double x = zero ? 0.0 : psi_prev[a];
    k.phi64[a] = x;
    k.phi_prev[a] = x;
    k.rec32_cur[a].phi_hi = (float)x;
    k.rec32_cur[a].phi_lo = (float)(x - (double)(float)x);
    k.rec64_cur[a].phi = x;
  }
}

// out[block]: the block's share of sum c_0, in a fixed order; with parts, the sum of those
__global__ void k_sum_c0(KParams k, int mixed, const double* parts, int n, double* out) {
  __shared__ double sm[kBlock / 32];
  double part[1] = {0.0};
  if (parts) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) part[0] += parts[i];
  } else {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < k.N; a += gridDim.x * blockDim.x) {
      if (mixed)
        part[0] += (double)k.rec32_cur[a].c[0] + (double)k.clo[a].x;
      else
        part[0] += k.rec64_cur[a].c[0];
    }
  }
  block_sum<1, kBlock>(part, sm);
  if (threadIdx.x == 0) out[blockIdx.x] = part[0];
}

}  // namespace

nnpp_status launch_adj_transport(const Engine& e, const EngineView& v, const Rec64* snap,
                                 const Rec64* snap1, const double* lam, double* mu, double* nu,
                                 double* acc, cudaStream_t st) {
  AdjArgs ad{snap, snap1, lam, mu, nu, acc};
  const size_t sh = smem_adj(v.halo_max, v.bond_max);
  if (sh > 227 * 1024) return set_error(NNPP_ERR_UNSUPPORTED, "adjoint: tile halo too large");
  return dispatch_lanes(e.W, [&](auto wc) -> nnpp_status {
    constexpr int W = decltype(wc)::value;
    NNPP_TRY(allow_smem(k_adj_transport<W>, sh));
    k_adj_transport<W><<<occ_grid(k_adj_transport<W>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(v, ad);
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  });
}

nnpp_status launch_adj_transport32(const Engine& e, const EngineView& v, Handle& h, const Rec64* snap,
                                   const Rec64* snap1, const double* lam, float4* rec, double* mu,
                                   double* nu, double* acc, cudaStream_t st) {
  KParams kp = make_kparams(h, h.cur);
  k_adj_pack<<<h.grid, kBlock, 0, st>>>(kp, snap, snap1, lam, rec);
  NNPP_CUDA(cudaGetLastError());
  k_adj_transport32<4><<<claim_grid(k_adj_transport32<4>, 0, e.sms, v.nslices), kBlock, 0, st>>>(
      v, rec, mu, nu, acc);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_adj_combine(Handle& h, const double* mu, double* lam, double inject) {
  KParams kp = make_kparams(h, h.cur);
  k_adj_combine<<<h.grid, kBlock, 0, h.st>>>(kp, mu, lam, inject);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_snap_state(Handle& h, Rec64* dst) {
  KParams kp = make_kparams(h, h.cur);
  k_snap_state<<<h.grid, kBlock, 0, h.st>>>(kp, dst, h.state_prec == NNPP_MIXED ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_snap_phi(Handle& h, Rec64* dst) {
  KParams kp = make_kparams(h, h.cur);
  k_snap_phi<<<h.grid, kBlock, 0, h.st>>>(kp, dst);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_load_phi(Handle& h, const double* phi, Rec64* snap) {
  KParams kp = make_kparams(h, h.cur);
  k_load_phi<<<h.grid, kBlock, 0, h.st>>>(kp, phi, snap, h.state_prec == NNPP_MIXED ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_record_solve(Handle& h, int slot) {
  KParams kp = make_kparams(h, h.cur);
  k_record_solve<<<h.grid, kBlock, 0, h.st>>>(kp, slot);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_adj_solve_setup(Handle& h, const Rec64* snap, const double* psi_prev, bool first) {
  // the adjoint solve's unknowns are those of step n; after a forward solve the Dirichlet coupling is
  // another one as well
  if (first) NNPP_TRY(invalidate_operator(h));
  KParams kp = make_kparams(h, h.cur);
  k_adj_solve_setup<<<h.grid, kBlock, 0, h.st>>>(kp, snap, psi_prev, h.state_prec == NNPP_MIXED ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  // deflated adjoint solve when the step's phases are those of the installed coarse operator
  return coarse_defl_check(h);
}

nnpp_status launch_sum_c0(Handle& h, double* out) {
  KParams kp = make_kparams(h, h.cur);
  // block parts and their sum, a fixed summation order: repeated runs give the same mass to the bit.
  // (One block alone took 0.65 ms at 262k nodes.)
  double* parts = h.engine->d_partials.get();
  const int mixed = h.state_prec == NNPP_MIXED ? 1 : 0;
  const int blocks = std::max(1, std::min((h.N + kBlock - 1) / kBlock, h.engine->sms));
  k_sum_c0<<<blocks, kBlock, 0, h.st>>>(kp, mixed, nullptr, 0, parts);
  k_sum_c0<<<1, kBlock, 0, h.st>>>(kp, mixed, parts, blocks, out);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// ---------------------------------------------------------------------------------------
nnpp_status prepare_kernels(int H, int B, int lanes) {
  // every tile kernel, the adjoint's included, must fit its staged halo
  if (smem_tr64(H, B) > 220 * 1024 || smem_adj(H, B) > 220 * 1024)
    return set_error(NNPP_ERR_UNSUPPORTED, "tile halo too large for shared memory");
  NNPP_TRY(allow_smem(k_cg_spmv32h<false>, 200 * 1024));  // spmv_halo_fits bounds the size used
  NNPP_TRY(allow_smem(k_cg_spmv32h<true>, 200 * 1024));
  // transport_halo_fits bounds the size used
  NNPP_TRY(allow_smem(k_transport32h<8, true, 4>, kTrHaloSmemMax));
  return dispatch_lanes(lanes, [&](auto wc) -> nnpp_status {
    constexpr int W = decltype(wc)::value;
    NNPP_TRY(allow_smem(k_f11<float, W>, smem_prep(H, B)));
    NNPP_TRY(allow_smem(k_f11<double, W>, smem_prep(H, B)));
    NNPP_TRY(allow_smem(k_cg_spmv32t<W>, smem_spmv_staged()));
    NNPP_TRY(allow_smem(k_cg_spmv32s<W, kStreamCol>, kSmemCta));
    NNPP_TRY(allow_smem(k_cg_spmv32<W, true, 8, true, 3>, smem_spmv_win()));
    NNPP_TRY(allow_smem(k_cg_spmv32<W, true, 16, false, 3>, smem_spmv_win()));
    NNPP_TRY(allow_smem(k_cg_spmv32<W, true, 16, false, 3, 3>, smem_spmv_win()));
    NNPP_TRY(allow_smem(k_cg_spmv32<W, true, 8, true, 3, 4>, smem_spmv_win()));
    NNPP_TRY(allow_smem(k_residual64<W>, smem_tr64(H, B)));
    NNPP_TRY(allow_smem(k_transport64<2>, smem_transport64()));
    NNPP_TRY(allow_smem(k_transport64<4>, smem_transport64()));
    return NNPP_OK;
  });
}

// FP32 CG operator variants without the staged ring (the autotuner's list): 0 L1/L2 gathers
// in batches of 16 bond columns, pipelined (the next batch's weights and codes in flight while the
// current one gathers), 79 registers (three CTAs an SM); 2 shared-memory windows, pipelined batches
// of 8; 3 L1/L2 gathers in pipelined batches of 8, 48 registers (five CTAs an SM); 4 shared-memory
// windows, batches of 16; 5, 6, 7: 4, gathers in batches of 16 and 2 with bulk L2 prefetches of the
// operator stream 3, 3, 4 batches ahead
template <int W>
void launch_spmv_gather(int variant, const EngineView& v, int sms, cudaStream_t st) {
  switch (variant) {
    case 2: {
      const size_t sh = smem_spmv_win();
      k_cg_spmv32<W, true, 8, true, 3><<<claim_grid(k_cg_spmv32<W, true, 8, true, 3>, sh, sms, v.ncslices), kBlock, sh, st>>>(v);
      break;
    }
    case 3:
      k_cg_spmv32<W, false, 8, true, 5><<<claim_grid(k_cg_spmv32<W, false, 8, true, 5>, 0, sms, v.ncslices), kBlock, 0, st>>>(v);
      break;
    case 4: {
      const size_t sh = smem_spmv_win();
      k_cg_spmv32<W, true, 16, false, 3><<<claim_grid(k_cg_spmv32<W, true, 16, false, 3>, sh, sms, v.ncslices), kBlock, sh, st>>>(v);
      break;
    }
    case 5: {
      const size_t sh = smem_spmv_win();
      k_cg_spmv32<W, true, 16, false, 3, 3><<<slice_grid(k_cg_spmv32<W, true, 16, false, 3, 3>, sh, sms, v.ncslices), kBlock, sh, st>>>(v);
      break;
    }
    case 6:
      k_cg_spmv32<W, false, 16, false, 4, 3><<<slice_grid(k_cg_spmv32<W, false, 16, false, 4, 3>, 0, sms, v.ncslices), kBlock, 0, st>>>(v);
      break;
    case 7: {
      const size_t sh = smem_spmv_win();
      k_cg_spmv32<W, true, 8, true, 3, 4><<<slice_grid(k_cg_spmv32<W, true, 8, true, 3, 4>, sh, sms, v.ncslices), kBlock, sh, st>>>(v);
      break;
    }
    default:
      // measured at 512k (ms): 0.0575; pipelined batches of 8 at five CTAs 0.0588 (variant 3), of 12
      // at four 0.0592, of 16 at four (64 registers, spilling) 0.0687; unpipelined 16 at five 0.0615
      k_cg_spmv32<W, false, 16, true, 3><<<claim_grid(k_cg_spmv32<W, false, 16, true, 3>, 0, sms, v.ncslices), kBlock, 0, st>>>(v);
  }
}

bool spmv_staged_fits(const Engine& e) { return e.windows_fit && smem_spmv_staged() <= 227 * 1024; }

// the halo-staged operator's dynamic shared memory: the halo (plus the padding slot) as
// float4 and the largest tile code block
size_t smem_spmv_halo(int halo_max, int code_max16, int quad_max) {
  return (size_t)(halo_max + 1) * sizeof(float4) + (size_t)halo_zcap(halo_max + 1) * sizeof(float) +
         (size_t)((quad_max + 1) & ~1) * sizeof(float2) + (size_t)code_max16 * 16;
}
// the halo-staged transport runs when the largest tile halo fits a CTA's share
bool transport_halo_fits(const Engine& e) {
  return e.halo_max > 0 && smem_tr_halo(e.halo_max) <= kTrHaloSmemMax;
}

// variant 8 runs when every member has its layout, the tiles are at most 8 bins long (the
// halo-frame coordinates keep ~1e-7 of a bin) and a CTA's halo and code block fit
bool spmv_halo_fits(const Engine& e) {
  return e.halo_op && e.T <= 8 && smem_spmv_halo(e.halo_max, e.hcode_max16, e.hquad_max) <= 200 * 1024;
}

// Warps that share a slice: the most of 1, 2, 4, 8 with which the slices' warps still fit about half
// of the SMs' 48-64 resident ones.  Measured, split against one warp a slice, us: 8k nodes FP32
// operator 9.0 against 12.3, its refinement 12.8 against 22.9, FP64 operator 12.4 against 19.6,
// refinement 16.4 against 22.0, transport 96 against 239; 64k nodes FP32 operator 16.5 against 18.3,
// refinement 25 against 37; from 262k nodes on one warp a slice fills the SMs.
constexpr int kSplitWarpsPerSm = 32;
int split_warps(int sms, int slices, int most) {
  int k = 1;
  while (k < most && (long long)slices * 2 * k <= (long long)sms * kSplitWarpsPerSm) k *= 2;
  return k;
}
// calls f with the split as a constant
template <typename F>
void dispatch_split(int k, F&& f) {
  if (k >= 8)
    f(std::integral_constant<int, 8>());
  else if (k == 4)
    f(std::integral_constant<int, 4>());
  else if (k == 2)
    f(std::integral_constant<int, 2>());
  else
    f(std::integral_constant<int, 1>());
}
// CTAs of a split slice kernel: every one that fits at once, at most one per group of slices
template <int K, typename Kern>
int split_grid(Kern kern, size_t smem, int sms, int slices) {
  return occ_grid(kern, smem, sms, (slices + SplitSlice<K>::kSlices - 1) / SplitSlice<K>::kSlices);
}

nnpp_status launch_warm_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st) {
  if (prec == NNPP_MIXED) {
    k_warm_dots<float><<<occ_grid(k_warm_dots<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
    k_warm_apply<float><<<occ_grid(k_warm_apply<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
  } else {
    k_warm_dots<double><<<occ_grid(k_warm_dots<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
    k_warm_apply<double><<<occ_grid(k_warm_apply<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
  }
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_prep_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st,
                          cudaGraphConditionalHandle hc, double* F11_out) {
  if (prec == NNPP_MIXED && !F11_out) {
    k_phi4<float><<<occ_grid(k_phi4<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
    dispatch_split(split_warps(e.sms, v.nslices, 8), [&](auto kc) {
      constexpr int K = decltype(kc)::value;
      k_prep_masks<K><<<occ_grid(k_prep_masks<K>, 0, e.sms, (v.nslices + 7) / 8), kBlock, 0, st>>>(v);
      if (K > 1)
        k_prep_slices<K><<<split_grid<K>(k_prep_slices<K>, 0, e.sms, v.nslices), kBlock, 0, st>>>(v, hc);
      else
        k_prep_slices<K><<<claim_grid(k_prep_slices<K>, 0, e.sms, v.nslices), kBlock, 0, st>>>(v, hc);
    });
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  }
  if (!F11_out) {
    k_phi4<double><<<occ_grid(k_phi4<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v);
    dispatch_split(split_warps(e.sms, v.nslices, 8), [&](auto kc) {
      constexpr int K = decltype(kc)::value;
      k_prep64<K><<<split_grid<K>(k_prep64<K>, 0, e.sms, v.nslices), kBlock, 0, st>>>(v, hc);
    });
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  }
  return dispatch_lanes(e.W, [&](auto wc) -> nnpp_status {
    constexpr int W = decltype(wc)::value;
    const size_t sh = smem_prep(v.halo_max, v.bond_max);
    if (prec == NNPP_MIXED)
      k_f11<float, W><<<occ_grid(k_f11<float, W>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(v, F11_out);
    else
      k_f11<double, W><<<occ_grid(k_f11<double, W>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(v, F11_out);
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  });
}

// largest row stride of the members' coarse inverses (shared memory of k_coarse_gemv)
int cld_max(const Engine& e) {
  int m = 4;
  for (const Handle* h : e.members) m = std::max(m, h->coarse.valid ? h->coarse.ld : 0);
  return m;
}

// CTAs of the coarse kernels: one a tile of aggregates (agg_tile), at most eight an SM
int coarse_grid(const Engine& e) {
  long long tiles = 0;
  for (const Handle* h : e.members) tiles += h->coarse.valid ? (h->coarse.n + kAggTile - 1) / kAggTile : 0;
  return (int)std::max(1ll, std::min(tiles, (long long)e.sms * 8));
}

// z = M^-1 r with the two-level preconditioner: restriction, coarse solve, z and the dots
template <typename P>
nnpp_status launch_coarse_z(const Engine& e, const EngineView& v, cudaStream_t st, cudaGraphConditionalHandle hc,
                            int init) {
  const int which = init ? 0 : 1;
  const int rg = coarse_grid(e);
  k_coarse_restrict<P><<<rg, kBlock, 0, st>>>(v, which);
  k_coarse_gemv<<<rg, kBlock, (size_t)cld_max(e) * sizeof(float), st>>>(v, which, 0, 0, 0);
  k_cg_zdots<P><<<occ_grid(k_cg_zdots<P>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, hc, init,
                                                                               sizeof(P) == 8 ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

bool engine_coarse(const Engine& e) {
  for (const Handle* h : e.members)
    if (!h->coarse_enabled || !h->coarse.valid) return false;
  return !e.members.empty();
}

nnpp_status launch_cg_init_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st,
                             cudaGraphConditionalHandle hc) {
  const int split = engine_coarse(e) ? 1 : 0;
  if (prec == NNPP_MIXED)
    k_cg_init<float><<<occ_grid(k_cg_init<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, split ? 0 : hc, 0, split);
  else
    k_cg_init<double><<<occ_grid(k_cg_init<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, split ? 0 : hc, 1, split);
  NNPP_CUDA(cudaGetLastError());
  if (split) return prec == NNPP_MIXED ? launch_coarse_z<float>(e, v, st, hc, 1) : launch_coarse_z<double>(e, v, st, hc, 1);
  return NNPP_OK;
}

// The inner solve in one launch (k_cg_sweep): single instances with the two-level preconditioner,
// with the gathering operator (variant 0) or in FP64.
bool cg_sweep_applies(const Engine& e, int prec) {
  return e.members.size() == 1 && engine_coarse(e) && (prec == NNPP_FP64 || e.spmv_variant == 0);
}

template <typename P, int NW>
nnpp_status launch_sweep_w(const Engine& e, const EngineView& v, int grid, cudaStream_t st) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * NW);
  cfg.dynamicSmemBytes = (size_t)cld_max(e) * sizeof(float);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  NNPP_CUDA(cudaLaunchKernelEx(&cfg, k_cg_sweep<P, NW>, v));
  return NNPP_OK;
}
// Slices up to which a CTA has 16 warps: four or more share each of them, and with 128 registers the
// passes are inlined and a warp has four quads in flight; above, 32 warps of 64 registers.  Measured, 16
// against 32 (ms a step): 8k nodes 0.251 against 0.322, 64k (1,429 slices) 0.494 against 0.471, 262k
// 1.40 against 1.27, 2M 24.4 against 18.2.
constexpr long long kSweepSlices = 152 * 4;
// CTAs: every SM where the slices are more than the warps of three quarters of them; those three quarters
// below, and half of the SMs for few slices.  A solve alone gets little or nothing slower and the solves
// of other handles' threads run beside it.  Measured (ms a step of each handle, 1 / 8 threads): 8k nodes
// 76 CTAs 0.284 / 0.88, 152 0.294 / 1.63; 22k 76 0.275 / 0.97, 114 0.266 / 1.29; 64k 114 0.396 / 2.48,
// 152 0.394 / 3.10, 76 0.472 / 2.34.  (As launches that share the SMs: 0.64 / 1.03, 0.61 / 1.14 and
// 0.76 / 2.54; from 125k nodes on eight threads' solves one after another are 5 to 16% slower than
// launches were, 8.4 to 9.0 against 8.1 to 8.2 at 262k, one alone 1.09 against 1.64.)
int sweep_grid(int sms, int slices, bool few) {
  const int part = few ? sms / 2 : sms * 3 / 4;
  return slices > part * (few ? 16 : 32) ? sms : std::max(1, part);
}
nnpp_status launch_cg_sweep_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st) {
  const bool few = v.ncslices <= kSweepSlices;
  const int grid = sweep_grid(e.sms, v.ncslices, few);
  if (prec == NNPP_MIXED)
    return few ? launch_sweep_w<float, 16>(e, v, grid, st) : launch_sweep_w<float, 32>(e, v, grid, st);
  return few ? launch_sweep_w<double, 16>(e, v, grid, st) : launch_sweep_w<double, 32>(e, v, grid, st);
}

nnpp_status launch_cg_spmv_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st) {
  return dispatch_lanes(e.W, [&](auto wc) -> nnpp_status {
    constexpr int W = decltype(wc)::value;
    if (prec == NNPP_MIXED)
      if (e.spmv_variant == kSpmvHalo) {
        const size_t sh = smem_spmv_halo(e.halo_max, e.hcode_max16, e.hquad_max);
        const int qcap = (e.hquad_max + 1) & ~1;  // keeps the code block 16-byte aligned
        if (e.checks)
          k_cg_spmv32h<true><<<occ_grid(k_cg_spmv32h<true>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(
              v, e.halo_max + 1, qcap);
        else
          k_cg_spmv32h<false><<<occ_grid(k_cg_spmv32h<false>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(
              v, e.halo_max + 1, qcap);
      } else if (e.spmv_variant == 1 && e.members.size() == 1) {
        int stages = 2;
        const size_t sh = smem_spmv_stream(e.win_cap, &stages);
        k_cg_spmv32s<W, kStreamCol><<<occ_grid(k_cg_spmv32s<W, kStreamCol>, sh, e.sms, (v.nslices + 7) / 8), kBlock, sh, st>>>(
            v, stages, e.win_cap);
      } else if (e.spmv_variant == 1) {
        const size_t sh = smem_spmv_staged();
        k_cg_spmv32t<W><<<occ_grid(k_cg_spmv32t<W>, sh, e.sms, (v.nslices + 7) / 8), kBlock, sh, st>>>(v);
      } else if (const int split = split_warps(e.sms, v.ncslices, 8); split > 1 && e.spmv_variant == 0) {
        dispatch_split(split, [&](auto kc) {
          constexpr int K = decltype(kc)::value;
          k_cg_spmv32k<K><<<split_grid<K>(k_cg_spmv32k<K>, 0, e.sms, v.ncslices), kBlock, 0, st>>>(v);
        });
      } else {
        launch_spmv_gather<W>(e.spmv_variant, v, e.sms, st);
      }
    else
      dispatch_split(split_warps(e.sms, v.ncslices, 8), [&](auto kc) {
        constexpr int K = decltype(kc)::value;
        k_cg_spmv64<K><<<split_grid<K>(k_cg_spmv64<K>, 0, e.sms, v.ncslices), kBlock, 0, st>>>(v);
      });
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  });
}

// after the inner loop of a mixed solve: the deflated CG's final correction e = e^ + Q (r0 - t)
// (every kernel passes over instances that are not deflating)
nnpp_status launch_cg_final_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st) {
  if (prec != NNPP_MIXED || !engine_coarse(e) || e.members.size() != 1) return NNPP_OK;
  const int rg = coarse_grid(e);
  const int cg = occ_grid(k_def_final, 0, e.sms, v.nchunks);
  k_def_final<<<cg, kBlock, 0, st>>>(v, 1);
  k_coarse_restrict<float><<<rg, kBlock, 0, st>>>(v, 2);
  k_coarse_gemv<<<rg, kBlock, (size_t)cld_max(e) * sizeof(float), st>>>(v, 2, 0, 0, 1);
  k_def_final<<<cg, kBlock, 0, st>>>(v, 2);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// update fused with the restriction, coarse product, z and the dots
template <typename P>
nnpp_status launch_coarse_update(const Engine& e, const EngineView& v, cudaStream_t st, cudaGraphConditionalHandle hc) {
  const int rg = coarse_grid(e);
  k_cg_update_restrict<P><<<rg, kBlock, 0, st>>>(v);
  if (e.members.size() == 1) {
    // one instance: the dots come from the aggregates, the decisions from the coarse product's
    // last CTA, and z is a plain elementwise pass
    k_coarse_gemv<<<rg, kBlock, (size_t)cld_max(e) * sizeof(float), st>>>(v, 1, hc, 1, sizeof(P) == 4 ? 1 : 0);
    k_z_form<P><<<occ_grid(k_z_form<P>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, hc);
  } else {
    // ensembles: per-instance reductions in parallel (the last chunk of each instance)
    k_coarse_gemv<<<rg, kBlock, (size_t)cld_max(e) * sizeof(float), st>>>(v, 1, 0, 0, 0);
    k_cg_zdots<P><<<occ_grid(k_cg_zdots<P>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, hc, 0, sizeof(P) == 8 ? 1 : 0);
  }
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// one kernel of a single instance's split-iteration update (0 restriction and CG update,
// 1 coarse product, 2 z and the dots), for timing them one by one
nnpp_status launch_coarse_part_b(const Engine& e, const EngineView& v, int prec, int part, cudaStream_t st) {
  if (!engine_coarse(e) || e.members.size() != 1 || part < 0 || part > 2)
    return set_error(NNPP_ERR_INVALID, "time_kernel: the coarse update parts need one instance with a coarse space");
  const int n = std::max(1, e.members[0]->coarse.valid ? e.members[0]->coarse.n : 0);
  const int rg = std::max(1, std::min((n * 32 + kBlock - 1) / kBlock, e.sms * 8));
  const bool mixed = prec == NNPP_MIXED;
  if (part == 0) {
    if (mixed) k_cg_update_restrict<float><<<rg, kBlock, 0, st>>>(v);
    else k_cg_update_restrict<double><<<rg, kBlock, 0, st>>>(v);
  } else if (part == 1) {
    k_coarse_gemv<<<rg, kBlock, (size_t)cld_max(e) * sizeof(float), st>>>(v, 1, 0, 1, mixed ? 1 : 0);
  } else {
    if (mixed) k_z_form<float><<<occ_grid(k_z_form<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, 0);
    else k_z_form<double><<<occ_grid(k_z_form<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, 0);
  }
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_cg_update_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st,
                               cudaGraphConditionalHandle hc) {
  if (engine_coarse(e))
    return prec == NNPP_MIXED ? launch_coarse_update<float>(e, v, st, hc) : launch_coarse_update<double>(e, v, st, hc);
  if (prec == NNPP_MIXED)
    k_cg_update<float><<<occ_grid(k_cg_update<float>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, hc);
  else
    k_cg_update<double><<<occ_grid(k_cg_update<double>, 0, e.sms, v.nchunks), kBlock, 0, st>>>(v, hc);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status launch_ir_update_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st,
                               cudaGraphConditionalHandle hc) {
  const int split = split_warps(e.sms, v.ncslices, 8);
  if (prec == NNPP_MIXED) {
    if (split > 1)
      dispatch_split(split, [&](auto kc) {
        constexpr int K = decltype(kc)::value;
        k_ir_split<K><<<split_grid<K>(k_ir_split<K>, 0, e.sms, v.ncslices), kBlock, 0, st>>>(v, hc);
      });
    else
      k_ir_slices<<<claim_grid(k_ir_slices, 0, e.sms, v.ncslices), kBlock, 0, st>>>(v, hc);
  } else {
    dispatch_split(split, [&](auto kc) {
      constexpr int K = decltype(kc)::value;
      k_ir64<K><<<split_grid<K>(k_ir64<K>, 0, e.sms, v.ncslices), kBlock, 0, st>>>(v, hc);
    });
  }
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

// The halo-staged FP32 transport (form 1): batches of 8 bond columns, the next batch's codes
// and weights in flight.  Measured at 512k (bins per tile 4, ms a launch): 0.409, against
// 0.451 / 0.441 without the next batch in flight (batches of 8 / 16), 0.459 / 0.418 with it
// (16 / 4), 0.51-0.68 with tiles of 2 bins; the L1/L2 gathers of form 0 take 0.358.
void launch_transport_staged(const EngineView& v, int sms, cudaStream_t st) {
  const size_t sh = smem_tr_halo(v.halo_max);
  k_transport32h<8, true, 4><<<occ_grid_b(k_transport32h<8, true, 4>, kTrHBlock, sh, sms, v.ntiles), kTrHBlock, sh,
                               st>>>(v);
}

// CTAs of the next-guess pass (a step turns at most a few thousand nodes liquid)
constexpr int kFlipGuessCtas = 32;

nnpp_status launch_transport_b(const Engine& e, const EngineView& v, int prec, cudaStream_t st,
                               double* F_out) {
  return dispatch_lanes(e.W, [&](auto wc) -> nnpp_status {
    constexpr int W = decltype(wc)::value;
    if (prec == NNPP_MIXED) {
      if (F_out)
        k_transport32<true><<<slice_grid(k_transport32<true>, 0, e.sms, v.nslices), kBlock, 0, st>>>(v, F_out);
      else {
        if (e.tr_variant > 0 && transport_halo_fits(e)) {
          launch_transport_staged(v, e.sms, st);
        } else {
          k_transport32<false><<<claim_grid(k_transport32<false>, 0, e.sms, v.nslices), kBlock, 0, st>>>(v, nullptr);
        }
        k_flip_guess<float><<<kFlipGuessCtas, kBlock, 0, st>>>(v);
      }
    } else {
      const size_t sh = smem_tr64(v.halo_max, v.bond_max);
      if (F_out)
        k_residual64<W><<<occ_grid(k_residual64<W>, sh, e.sms, v.ntiles), kBlock, sh, st>>>(v, F_out);
      else {
        dispatch_split(split_warps(e.sms, v.nslices, 4), [&](auto kc) {
          constexpr int K = decltype(kc)::value < 4 ? decltype(kc)::value : 4;
          const size_t sh = K > 1 ? smem_transport64() : 0;
          k_transport64<K><<<split_grid<K>(k_transport64<K>, sh, e.sms, v.nslices), kBlock, sh, st>>>(v);
        });
        k_flip_guess<double><<<kFlipGuessCtas, kBlock, 0, st>>>(v);
      }
    }
    NNPP_CUDA(cudaGetLastError());
    return NNPP_OK;
  });
}

// ---------------------------------------------------------------------------------------
nnpp_status step_alloc(Handle& h) {
  const size_t N = (size_t)h.N;
  bool ok = h.dirmask.alloc(N) && h.bcval.alloc((S + 1) * N) && h.rec32[0].alloc(N) &&
            h.rec32[1].alloc(N) && h.clo.alloc(N) && h.rec64[0].alloc(N) && h.rec64[1].alloc(N) &&
            h.phi64.alloc(N) && h.phi_prev.alloc(N) && h.flip_step.alloc(N) && h.flip_list.alloc(N) &&
            h.b64.alloc(N) &&
            h.r64.alloc(N) && h.dsum64.alloc(N) && h.cpl64.alloc(N) && h.dinv64.alloc(N) && h.rin64.alloc(N) &&
            h.z64.alloc(N) && h.p64.alloc(N) && h.q64.alloc(N) && h.e64.alloc(N) && h.d32.alloc(N) &&
            h.dinv32.alloc(N) && h.rin32.alloc(N) && h.z32.alloc(N + 16) && h.p32.alloc(N) &&
            h.q32.alloc(N) && h.e32.alloc(N) && h.r0_32.alloc(N) && h.t32.alloc(N) && h.freem.alloc(N) &&
            h.phi4.alloc(N) && h.dstate.alloc(1) &&
            h.scratch_d.alloc(16 + 7 * 4096) && h.user_stage.alloc((S + 1) * N) &&
            h.user_stage_i.alloc(N);
  if (ok && h.warm_hist >= 3) ok = h.xh.alloc((size_t)h.warm_hist * N) && h.bh.alloc((size_t)h.warm_hist * N);
  if (!ok) return set_error(NNPP_ERR_NOMEM, "device state allocation");
  NNPP_CUDA(cudaMemsetAsync(h.freem.get(), 0, N, h.st));
  NNPP_CUDA(cudaMemsetAsync(h.rec32[1].get(), 0, N * sizeof(Rec32), h.st));
  NNPP_CUDA(cudaMemsetAsync(h.rec64[1].get(), 0, N * sizeof(Rec64), h.st));
  NNPP_CUDA(cudaMemsetAsync(h.e32.get(), 0, N * sizeof(float), h.st));
  NNPP_CUDA(cudaMemsetAsync(h.e64.get(), 0, N * sizeof(double), h.st));
  // z32 is padded by 16 (read, never used) elements: window copies round their rows up to 4
  NNPP_CUDA(cudaMemsetAsync(h.z32.get(), 0, (N + 16) * sizeof(float), h.st));
  NNPP_CUDA(cudaMemsetAsync(h.z64.get(), 0, N * sizeof(double), h.st));
  NNPP_CUDA(cudaMemsetAsync(h.flip_step.get(), 0xff, N * sizeof(int), h.st));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h.device);
  if (sms <= 0) sms = 152;
  long long g = std::min<long long>(((long long)h.N + 255) / 256, (long long)sms * 8);
  if (g > 4096) g = 4096;
  if (g < 1) g = 1;
  h.grid = (int)g;
  return NNPP_OK;
}

KParams make_kparams(Handle& h, int cur) {
  KParams k;
  std::memset(&k, 0, sizeof(k));
  const nnpp_params& p = h.p;
  k.N = h.N;
  k.row = h.lay.row.get();
  k.col = h.lay.col.get();
  k.slot16 = h.slot16.get();
  k.sell = h.sell.get();
  k.sell_lo = h.sell_lo.get();
  k.sell_cg = h.sell_cg.get();
  k.sell_cg_lo = h.sell_cg_lo.get();
  k.sell64 = h.sell64.get();
  k.sell_cg64 = h.sell_cg64.get();
  k.cg_width = h.cg_width.get();
  k.cg_rows = h.cg_rows.get();
  k.cg_pos = h.cg_pos.get();
  k.xrow = h.xrow.get();
  k.phi4 = h.phi4.get();
  k.w64 = h.lay.w64.get();
  k.w32 = h.lay.w32.get();
  k.wlo32 = h.lay.wlo32.get();
  k.dirmask = h.dirmask.get();
  k.bcval = h.bcval.get();
  k.rec32_cur = h.rec32[cur].get();
  k.rec32_nxt = h.rec32[cur ^ 1].get();
  k.clo = h.clo.get();
  k.rec64_cur = h.rec64[cur].get();
  k.rec64_nxt = h.rec64[cur ^ 1].get();
  k.phi64 = h.phi64.get();
  k.phi_prev = h.phi_prev.get();
  k.phi_keep = h.phi_keep[cur & 1];
  k.flip_step = h.flip_step.get();
  k.flip_list = h.flip_list.get();
  k.b64 = h.b64.get();
  k.r64 = h.r64.get();
  k.dsum64 = h.dsum64.get();
  k.cpl64 = h.cpl64.get();
  k.freem = h.freem.get();
  k.d32 = h.d32.get();
  k.dinv32 = h.dinv32.get();
  k.dinv64 = h.dinv64.get();
  k.rin32 = h.rin32.get();
  k.z32 = h.z32.get();
  k.p32 = h.p32.get();
  k.q32 = h.q32.get();
  k.e32 = h.e32.get();
  k.rin64 = h.rin64.get();
  k.z64 = h.z64.get();
  k.p64 = h.p64.get();
  k.q64 = h.q64.get();
  k.e64 = h.e64.get();
  k.ds = h.dstate.get();
  k.bv_ptr = &h.dstate.get()->BV;
  k.b_override = h.b_override;
  // halo-staged CG operator: weights in units of the bin side hb (FP32 of the bins' side)
  k.hquad = h.hquad.get();
  k.hquad_n = (int)h.hquad.size();
  k.checks = h.checks;
  k.hcode = h.hcode.get();
  k.posrec = h.posrec.get();
  {
    const double hb = (double)h.h32;
    k.hinv = (float)(1.0 / hb);
    k.hc0 = (float)((p.delta + 0.5 * p.dx) / p.dx);
    k.hc1 = (float)(hb / p.dx);
    k.hsw = (float)(p.dx * p.dy * p.dz / (hb * hb * hb));
  }
  k.dt = p.dt;
  k.csat = p.CSat / p.CSolid;
  k.c_floor = p.c_floor;
  k.csat_hi = (float)k.csat;
  k.csat_lo = (float)(k.csat - (double)k.csat_hi);
  k.cfl_hi = (float)k.c_floor;
  k.cfl_lo = (float)(k.c_floor - (double)k.cfl_hi);
  k.k_diss = p.k_diss;
  k.sw = p.switch_width;
  k.vol_red = p.vol_red;
  k.lam = (1. / (p.K_phi * p.sigma)) * p.F * p.CSolid;
  for (int s = 0; s < S; ++s) {
    k.K1[s] = p.K1[s];
    k.K2zF[s] = p.K2[s] * p.z[s] * p.F / (p.R * p.T);
    k.DL[s] = p.D_liquid[s];
    k.DSo[s] = p.D_solid[s];
    k.z[s] = p.z[s];
    k.K1f[s] = (float)k.K1[s];
    k.K2zFf[s] = (float)k.K2zF[s];
    k.DLf[s] = (float)k.DL[s];
    k.DSof[s] = (float)k.DSo[s];
  }
  k.dtf = (float)k.dt;
  k.sub_step_no = p.sub_step_no;
  k.dissolve_count = 1;
  k.extrapolate = h.extrapolate;
  k.hist_m = (h.extrapolate && h.warm_hist >= 3 && h.xh.get()) ? h.warm_hist : 0;
  k.xh = h.warm_x_alt ? h.warm_x_alt : h.xh.get();
  k.bh = h.warm_b_alt ? h.warm_b_alt : h.bh.get();
  const Coarse& co = h.coarse;
  k.coarse = (h.coarse_enabled && co.valid) ? 1 : 0;
  k.defl_ok = 0;  // set by the engine for single-instance runs
  k.agg = co.agg.get();
  k.cinv = co.inv.get();
  k.rc = const_cast<float*>(co.rc.get());
  k.xc = const_cast<float*>(co.xc.get());
  k.bin_start = h.lay.bin_start.get();
  k.cn = co.n;
  k.cld = co.ld;
  k.cdots = co.dots.get();
  k.ap_k = co.ap_k;
  k.ap_col = co.ap_col.get();
  k.ap_val = co.ap_val.get();
  k.r0_32 = h.r0_32.get();
  k.t32 = h.t32.get();
  k.cf = co.f;
  k.cna0 = co.na[0];
  k.cna1 = co.na[1];
  k.cna2 = co.na[2];
  k.nb0 = h.lay.nb[0];
  k.nb1 = h.lay.nb[1];
  k.nb2 = h.lay.nb[2];
  return k;
}

nnpp_status load_state(Handle& h, const double* d_c_user, const double* d_phi_user,
                       const int* d_phase_user, int prec, bool dirichlet_phi,
                       bool keep_history) {
  // the cached operator arrays stay valid for the same phases, precision and Dirichlet
  // potentials (a changed phase is detected by the kernel)
  if (prec != h.state_prec || !dirichlet_phi) NNPP_TRY(invalidate_operator(h));
  KParams kp = make_kparams(h, h.cur);
  k_load_state<<<h.grid, kBlock, 0, h.st>>>(kp, h.lay.perm.get(), d_c_user, d_phi_user, d_phase_user,
                                            prec == NNPP_MIXED ? 1 : 0, dirichlet_phi ? 1 : 0,
                                            keep_history ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  h.state_prec = prec;
  return NNPP_OK;
}

nnpp_status invalidate_operator(Handle& h) {
  NNPP_CUDA(cudaMemsetAsync(&h.dstate.get()->op_valid, 0, sizeof(int), h.st));
  return NNPP_OK;
}

nnpp_status store_state(Handle& h, double* d_c_user, double* d_phi_user, int* d_phase_user) {
  KParams kp = make_kparams(h, h.cur);
  k_store_state<<<h.grid, kBlock, 0, h.st>>>(kp, h.lay.perm.get(), d_c_user, d_phi_user, d_phase_user,
                                             h.state_prec == NNPP_MIXED ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

nnpp_status convert_state(Handle& h, int to_prec) {
  if (h.state_prec == to_prec) return NNPP_OK;
  KParams kp = make_kparams(h, h.cur);
  k_convert<<<h.grid, kBlock, 0, h.st>>>(kp, to_prec == NNPP_MIXED ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  h.state_prec = to_prec;
  // the two precisions form the diagonal with different arithmetic
  return invalidate_operator(h);
}

nnpp_status init_diag(Handle& h, bool restart) {
  KParams kp = make_kparams(h, h.cur);
  k_init_diag<<<h.grid, kBlock, 0, h.st>>>(kp, h.state_prec == NNPP_MIXED ? 1 : 0,
                                           h.scratch_d.get() + 16, restart ? 1 : 0);
  NNPP_CUDA(cudaGetLastError());
  return NNPP_OK;
}

}  // namespace nnpp
