// The operator policy of the e/o twisted-mass CG: K(+mu)K(-mu) on odd sites
// (inv_tmDkern_eoprec_square_eos_cg).
#pragma once
#include "tms_solver.cuh"

namespace tms_int
{
  struct EoOp
  {
    static constexpr int slot0 = kSlotEo;
    static constexpr bool kHalfArith = true; // has the FP16-arithmetic hop
    static constexpr bool kOneLaunch = true; // has the one-launch CG (tms_cg_small.cuh)
    static constexpr int nlo = 6;
    static int stride(tms_ctx* c) { return c->g.stride; }
    static int nsites(tms_ctx* c) { return (int)c->g.Vh; }
    static Field* hi(tms_ctx* c) { return c->f64; }
    static Field* lo(tms_ctx* c) { return c->lo; }
    static int& lo_prec(tms_ctx* c) { return c->lo_prec; }
    static Field& xlo(tms_ctx* c) { return c->xlo32; }

    // r = b - K(+mu)K(-mu) x in FP64; returns |r|^2 (uses hi 4, 5, 6).  For the
    // mixed solvers (`mixed`) the links may be read as 12 reals.
    static tms_status true_residual(tms_ctx* ctx, const Field& b, const Field& x, const Field& r, double* rr,
                                    bool mixed = false)
    {
      Field &t1 = ctx->f64[4], &te = ctx->f64[5], &s = ctx->f64[6];
      if (mixed)
        {
          // the mixed solvers' recomputation: K(+mu) fused with r = b - s and |r|^2
          auto res = [&](const auto& U) {
            kern_op<PREC_F64>(ctx, U, x, te, t1, -1.0, ctx->prm);
            EpiInvDiag<PREC_F64> a{{view<PREC_F64>(te), view<PREC_F64>(te)}, ctx->prm, +1.0};
            launch_hop<PREC_F64>(ctx, ctx->stream, 0, 1, t1, t1, U, ctx->prm, a);
            EpiKernResidual<PREC_F64> e{view<PREC_F64>(r), view<PREC_F64>(t1), view<PREC_F64>(b), ctx->prm, +1.0};
            launch_hop<PREC_F64>(ctx, ctx->stream, 1, 1, te, te, U, ctx->prm, e);
          };
          if (reliable_links12(ctx)) res(links64r(ctx));
          else res(links64(ctx));
          CU(cudaGetLastError());
          *rr = read_result(ctx);
          return TMS_OK;
        }
      auto U = links64(ctx);
      kern_op<PREC_F64>(ctx, U, x, te, t1, -1.0, ctx->prm);
      kern_op<PREC_F64>(ctx, U, t1, te, s, +1.0, ctx->prm);
      const int n = nsites(ctx);
      ++ctx->launches;
      residual_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
        n, view<PREC_F64>(b), view<PREC_F64>(s), view<PREC_F64>(r), reducer(ctx));
      CU(cudaGetLastError());
      *rr = read_result(ctx);
      return TMS_OK;
    }

    // The one-launch CG: where every 32-site block is resident at once (two per SM: up to 9472 sites of a parity).  Whole solves, launches /
    // one launch, at 864, 4096, 6400 and 9216 sites: FP64 2.13 / 2.10, 3.13 / 2.95,
    // 4.05 / 3.24, 4.08 / 3.67 ms; FP32 2.22 / 1.84, 2.98 / 2.53, 3.03 / 2.69,
    // 3.41 / 2.91; FP16 2.34 / 1.83, 3.23 / 2.45, 3.43 / 2.60, 3.47 / 2.79.
    static constexpr int coherent(int P) { return P == PREC_F64 ? PREC_C64 : P == PREC_F32 ? PREC_C32 : PREC_C16; }
    template <int P, int LF>
    static auto one_kernel()
    {
      return cg_small_kernel<coherent(P), (P == PREC_F64) ? PREC_C64 : PREC_C32, LF>;
    }
    static constexpr int kOneIters = 64; // iterations of a launch: a bound on its length
    template <int P, int LF>
    static bool one_launch(tms_ctx* c)
    {
      const int blocks = div_up(c->g.Vh, HOP_DP_SITES);
      if (!c->small_lattice) return false;
      int coop = 0, sms = 0, per = 0;
      if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) != cudaSuccess || !coop ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, one_kernel<P, LF>(), HOP_DP_THREADS, 0) != cudaSuccess)
        {
          cudaGetLastError(); // the launches do without
          return false;
        }
      return blocks <= per * sms;
    }
    template <int P>
    static SpinorT<P> past_l1(const Field& f)
    {
      SpinorT<P> s;
      s.d = reinterpret_cast<decltype(s.d)>(f.d);
      s.n = f.n;
      s.stride = f.stride;
      return s;
    }
    template <int P, int LF>
    // false if the device refuses the launch (fewer SMs for this process than the device has)
    static bool launch_one(tms_ctx* ctx, const LinkT<LF>& U, const Field* v, const Field& x)
    {
      constexpr int PC = coherent(P), PXC = (P == PREC_F64) ? PREC_C64 : PREC_C32;
      Lattice g = ctx->g;
      SpinorT<PC> r = past_l1<PC>(v[1]), p = past_l1<PC>(v[2]), t1 = past_l1<PC>(v[3]), te = past_l1<PC>(v[4]);
      SpinorT<PXC> xx = past_l1<PXC>(x);
      LinkT<LF> u = U;
      const OpParams* prm = ctx->prm;
      CgState* st = ctx->st;
      double* partial = ctx->red_partial;
      unsigned* bar = ctx->grid_bar;
      int polls = ctx->grid_polls, iters = kOneIters;
      void* args[] = {&g, &r, &p, &t1, &te, &xx, &u, &prm, &st, &partial, &bar, &polls, &iters};
      ctx->launches += 2;
      grid_bar_reset_kernel<<<1, 1, 0, ctx->stream>>>(bar);
      if (cudaLaunchCooperativeKernel((const void*)one_kernel<P, LF>(), dim3(div_up(g.Vh, HOP_DP_SITES)),
                                      dim3(HOP_DP_THREADS), args, 0, ctx->stream) == cudaSuccess)
        return true;
      cudaGetLastError();
      return false;
    }

    // the paired x update (record with paired = true) keeps the second direction here
    static constexpr bool kPaired = true;
    static Field& p2(tms_ctx* c) { return c->lo[5]; }

    // `iters` CG iterations in precision P (x in PX): v 1 r, 2 p, 3 t1, 4 te.
    // paired (iters even): iteration 2k reads its direction from p and writes
    // the next into p2, iteration 2k+1 reads p2, writes p and adds both
    // iterations' steps to x; a replay starts and ends with the direction in p.
    template <int P, int PX, int LF>
    static void record(tms_ctx* c, cudaStream_t s, const LinkT<LF>& U, Field* v, const Field& x, int iters,
                       bool paired = false)
    {
      const Field &r = v[1], &t1 = v[3], &te = v[4];
      const int* stop = &c->st->stop;
      const OpParams* prm = c->prm;
      const int n = nsites(c);
      for (int it = 0; it < iters; it++)
        {
          const bool odd = paired && (it & 1);
          const Field& p = odd ? p2(c) : v[2];         // this iteration's direction
          const Field& pn = (paired && !odd) ? p2(c) : v[2]; // the next one
          EpiInvDiag<P> a1{{view<P>(te), view<P>(te)}, prm, -1.0};
          launch_hop<P, LF>(c, s, 0, 1, p, p, U, prm, a1, NoFin{}, stop);
          EpiKern<P, true> b1{{view<P>(t1), view<P>(t1)}, {view<P>(p), view<P>(p)}, prm, -1.0};
          launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b1, FinAlpha{c->st}, stop);
          EpiInvDiag<P> a2{{view<P>(te), view<P>(te)}, prm, +1.0};
          launch_hop<P, LF>(c, s, 0, 1, t1, t1, U, prm, a2, NoFin{}, stop);
          if (!paired)
            {
              EpiKernCgUpdate<P, PX, 1> b2{view<P>(t1), view<P>(r), view<P>(p), view<PX>(x), prm, c->st, +1.0};
              launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b2, FinBeta{c->st}, stop);
            }
          else if (!odd)
            {
              EpiKernCgUpdate<P, PX, 0> b2{view<P>(t1), view<P>(r), view<P>(p), view<PX>(x), prm, c->st, +1.0};
              launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b2, FinBeta{c->st}, stop);
            }
          else
            {
              EpiKernCgUpdate<P, PX, 2> b2{view<P>(t1), view<P>(r),   view<P>(p),       view<PX>(x),
                                           prm,          c->st,         +1.0,             view<P>(v[2])};
              launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b2, FinBeta{c->st}, stop);
            }
          ++c->launches;
          if (paired)
            launch_pdl(c, xpay_to_kernel<P>, div_up(n, BLAS_THREADS), BLAS_THREADS, 0, s, n, view<P>(r), view<P>(p),
                       view<P>(pn), (const CgState*)c->st, stop);
          else
            launch_pdl(c, xpay_kernel<P>, div_up(n, BLAS_THREADS), BLAS_THREADS, 0, s, n, view<P>(r), view<P>(p),
                       (const CgState*)c->st, stop);
        }
    }
  };
}

namespace tms_int
{
  // instantiated in tms_cg_half.cu
  extern template tms_status cg_half<EoOp>(tms_ctx*, int, double, bool, tms_stats*);
}
