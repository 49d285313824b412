// The e/o CG of K(+mu)K(-mu) in one cooperative launch, for lattices whose
// blocks of 32 sites (of each parity) are all resident at once: up to `iters`
// iterations with a grid barrier between the steps of each, instead of five
// launches an iteration.
//
// Bound by latency: at 8^3x16 an iteration of five launches took 23.5 us for
// work that moves 25 MB, most of it launch and drain.  The hops are those of
// tms_hop_dp.cuh (a site's directions in the eight warps of its block); the
// links of a block stay in L1 from one iteration to the next.  The vectors
// change under the kernel, so every read of them goes past L1.
// The scalars are computed by every block from the same partial sums in the
// same order, so no block waits for another's result beyond the barrier.
#pragma once

#include "tms_hop_dp.cuh"

namespace tms
{
  // ------------------------------------------------- accessors past L1
  template <> struct SpinorT<PREC_C64>
  {
    using R = double;
    double2* d;
    float* n; // unused
    int stride;
    __device__ __forceinline__ void load(int site, C<double> v[12]) const
    {
#pragma unroll
      for (int c = 0; c < 12; c++)
        {
          const double2 w = __ldcg(d + (size_t)c * stride + site);
          v[c] = {w.x, w.y};
        }
    }
    __device__ __forceinline__ void load_raw(int site, C<double> v[12], double& scale) const
    {
      load(site, v);
      scale = 1.0;
    }
    __device__ __forceinline__ void store(int site, const C<double> v[12]) const
    {
#pragma unroll
      for (int c = 0; c < 12; c++) d[(size_t)c * stride + site] = make_double2(v[c].re, v[c].im);
    }
  };
  template <> struct SpinorT<PREC_C32>
  {
    using R = float;
    float4* d;
    float* n; // unused
    int stride;
    __device__ __forceinline__ void load(int site, C<float> v[12]) const
    {
#pragma unroll
      for (int k = 0; k < 6; k++)
        {
          const float4 w = __ldcg(d + (size_t)k * stride + site);
          v[2 * k] = {w.x, w.y};
          v[2 * k + 1] = {w.z, w.w};
        }
    }
    __device__ __forceinline__ void load_raw(int site, C<float> v[12], float& scale) const
    {
      load(site, v);
      scale = 1.0f;
    }
    __device__ __forceinline__ void store(int site, const C<float> v[12]) const
    {
#pragma unroll
      for (int k = 0; k < 6; k++)
        d[(size_t)k * stride + site] = make_float4(v[2 * k].re, v[2 * k].im, v[2 * k + 1].re, v[2 * k + 1].im);
    }
  };
  template <> struct SpinorT<PREC_C16>
  {
    using R = float;
    uint4* d;
    float* n;
    int stride;
    __device__ __forceinline__ void load_raw(int site, C<float> v[12], float& scale) const
    {
      scale = __ldcg(n + site);
#pragma unroll
      for (int k = 0; k < 3; k++)
        {
          const uint4 w = __ldcg(d + (size_t)k * stride + site);
          const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int j = 0; j < 4; j++)
            {
              const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[j]));
              v[4 * k + j] = {f.x, f.y};
            }
        }
    }
    __device__ __forceinline__ void load(int site, C<float> v[12]) const
    {
      float s;
      load_raw(site, v, s);
#pragma unroll
      for (int c = 0; c < 12; c++) v[c] = cscale(v[c], s);
    }
    __device__ __forceinline__ void store(int site, const C<float> v[12]) const
    {
      SpinorT<PREC_F16>{d, n, stride}.store(site, v);
    }
  };

  // ------------------------------------------------------- grid barrier
  // All blocks of a cooperative launch arrive before any leaves.  The wait is
  // bounded: false if it gave up.
  constexpr int GRID_BAR_POLLS = 1 << 20; // about a second
  struct GridBarrier
  {
    unsigned* count; // 0 at launch
    unsigned target;
    int limit; // polls
    __device__ __forceinline__ bool sync()
    {
      __syncthreads();
      int ok = 1;
      target += gridDim.x;
      if (threadIdx.x == 0)
        {
          asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(count), "r"(1u) : "memory");
          unsigned v;
          int polls = 0;
          do asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
          while (v < target && ++polls < limit);
          ok = v >= target;
        }
      return __syncthreads_and(ok);
    }
  };

  static __global__ void grid_bar_reset_kernel(unsigned* count) { *count = 0u; }

  // the hop of the block's sites of parity p from `in`, then the epilogue; the
  // epilogue's sum of the block's sites in warp 0
  template <int P, int LF, class Epi>
  __device__ __forceinline__ double small_hop(DpShare<typename SpinorT<P>::R>& sh, const Lattice& g, int p, const Site& s,
                                              int ieo, int n, bool active, const SpinorT<P>& in, const LinkT<LF>& U,
                                              typename SpinorT<P>::R anis, const Epi& epi)
  {
    using R = typename SpinorT<P>::R;
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    C<R> L[9];
    R ls;
    U.template load_scaled<false>((d & 1) ? 1 - p : p, d >> 1, (d & 1) ? n : ieo, L, ls);
    dp_direction<P, LF>(sh, d, lane, n, in, L, ls);
    __syncthreads();
    double part = 0.0;
    if (d == 0 && active)
      {
        C<R> acc[12];
        dp_sum(sh, g, s, lane, anis, acc);
        part = epi(p, ieo, acc);
      }
    return part;
  }

  // the sum of the blocks' parts (in warp 0 of each), the same in every thread
  __device__ __forceinline__ bool small_sum(double part, double* partial, GridBarrier& bar, double* red, double& sum)
  {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w == 0)
      {
        part = warp_sum(part);
        if (lane == 0) partial[blockIdx.x] = part;
      }
    if (!bar.sync()) return false;
    double v = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += HOP_DP_THREADS) v += __ldcg(partial + i);
    v = warp_sum(v);
    if (lane == 0) red[w] = v;
    __syncthreads();
    sum = 0.0;
#pragma unroll
    for (int k = 0; k < HOP_DP_THREADS / 32; k++) sum += red[k];
    return true;
  }

  template <int P, int PX, int LF>
  __global__ void __launch_bounds__(HOP_DP_THREADS, 2)
    cg_small_kernel(Lattice g, SpinorT<P> r, SpinorT<P> p, SpinorT<P> t1, SpinorT<P> te, SpinorT<PX> x, LinkT<LF> U,
                    const OpParams* __restrict__ prm_g, CgState* st_g, double* partial, unsigned* bar_count, int polls,
                    int iters)
  {
    using R = typename SpinorT<P>::R;
    __shared__ DpShare<R> sh;
    __shared__ double red[2][HOP_DP_THREADS / 32];
    __shared__ CgState st; // the block's copy
    __shared__ OpParams prm;
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    if (threadIdx.x == 0)
      {
        st = *st_g;
        prm = *prm_g;
      }
    const bool active = blockIdx.x * HOP_DP_SITES + lane < g.Vh;
    const int ieo = active ? blockIdx.x * HOP_DP_SITES + lane : (int)g.Vh - 1;
    const Site s0 = eo_site(g, 0, ieo), s1 = eo_site(g, 1, ieo);
    const int n0 = dp_neighbour(g, s0, d) >> 1, n1 = dp_neighbour(g, s1, d) >> 1;
    GridBarrier bar{bar_count, 0u, polls};
    __syncthreads();
    const R anis = R(prm.anis);
    bool alive = true;
    for (int it = 0; it < iters && st.stop == STOP_RUN; it++)
      {
        double pAp, rr;
        small_hop<P, LF>(sh, g, 0, s0, ieo, n0, active, p, U, anis, EpiInvDiag<P>{{te, te}, &prm, -1.0});
        if (!(alive = bar.sync())) break;
        double part = small_hop<P, LF>(sh, g, 1, s1, ieo, n1, active, te, U, anis,
                                       EpiKern<P, true>{{t1, t1}, {p, p}, &prm, -1.0});
        if (!(alive = small_sum(part, partial, bar, red[0], pAp))) break;
        if (threadIdx.x == 0) FinAlpha{&st}(pAp);
        __syncthreads();
        if (st.stop != STOP_RUN) break;
        small_hop<P, LF>(sh, g, 0, s0, ieo, n0, active, t1, U, anis, EpiInvDiag<P>{{te, te}, &prm, +1.0});
        if (!(alive = bar.sync())) break;
        part = small_hop<P, LF>(sh, g, 1, s1, ieo, n1, active, te, U, anis,
                                EpiKernCgUpdate<P, PX, 1>{t1, r, p, x, &prm, &st, +1.0});
        if (!(alive = small_sum(part, partial + gridDim.x, bar, red[1], rr))) break;
        if (threadIdx.x == 0) FinBeta{&st}(rr);
        __syncthreads();
        if (st.stop != STOP_RUN) break;
        if (d == 0 && active)
          {
            C<R> a[12], b[12];
            r.load(ieo, a);
            p.load(ieo, b);
            const R beta = R(st.beta);
#pragma unroll
            for (int c = 0; c < 12; c++) b[c] = cadd(a[c], cscale(b[c], beta));
            p.store(ieo, b);
          }
        if (!(alive = bar.sync())) break;
      }
    // (a block that gave up stays away from the next barrier, so all give up there, or there is none: then
    // the others have finished the launch's work, and so had it, and either outcome is right)
    if (threadIdx.x == 0)
      {
        if (!alive) st_g->stop = STOP_TIMEOUT;
        else if (blockIdx.x == 0) *st_g = st;
      }
  }
}
