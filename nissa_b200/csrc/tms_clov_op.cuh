// The operator policy of the e/o twisted-clover CG.
#pragma once
#include "tms_solver.cuh"

namespace tms_int
{
  // ClovOp: K_clov(dag=false) K_clov(dag=true) on odd sites
  // (inv_tmclovDkern_eoprec_square_eos_cg), on the e/o fields of EoOp
  struct ClovOp
  {
    static constexpr int slot0 = kSlotClov;
    static constexpr bool kHalfArith = false;
    static constexpr bool kOneLaunch = false;
    static constexpr bool kPaired = true;
    static Field& p2(tms_ctx* c) { return c->lo[5]; }
    static constexpr int nlo = 6;
    static int stride(tms_ctx* c) { return c->g.stride; }
    static int nsites(tms_ctx* c) { return (int)c->g.Vh; }
    static Field* hi(tms_ctx* c) { return c->f64; }
    static Field* lo(tms_ctx* c) { return c->lo; }
    static int& lo_prec(tms_ctx* c) { return c->lo_prec; }
    static Field& xlo(tms_ctx* c) { return c->xlo32; }

    // r = b - K(false)K(true) x in FP64; returns |r|^2 (uses hi 4, 5, 6).  For the
    // mixed solvers (`mixed`) the links may be read as 12 reals.
    static tms_status true_residual(tms_ctx* ctx, const Field& b, const Field& x, const Field& r, double* rr,
                                    bool mixed = false)
    {
      Field &t1 = ctx->f64[4], &te = ctx->f64[5], &s = ctx->f64[6];
      if (mixed && reliable_links12(ctx))
        {
          auto U = links64r(ctx);
          clov_kern_op<PREC_F64>(ctx, U, clov64(ctx), x, te, t1, 1, ctx->prm);
          clov_kern_op<PREC_F64>(ctx, U, clov64(ctx), t1, te, s, 0, ctx->prm);
        }
      else
        {
          auto U = links64(ctx);
          clov_kern_op<PREC_F64>(ctx, U, clov64(ctx), x, te, t1, 1, ctx->prm);
          clov_kern_op<PREC_F64>(ctx, U, clov64(ctx), t1, te, s, 0, ctx->prm);
        }
      const int n = nsites(ctx);
      ++ctx->launches;
      residual_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
        n, view<PREC_F64>(b), view<PREC_F64>(s), view<PREC_F64>(r), reducer(ctx));
      CU(cudaGetLastError());
      *rr = read_result(ctx);
      return TMS_OK;
    }

    // `iters` CG iterations in precision P (x in PX): v 1 r, 2 p, 3 t1, 4 te.
    // (p, K(false)K(true) p) = |K(true) p|^2 is reduced in the second launch.
    // paired: the two directions and every-other-iteration x update of EoOp.
    template <int P, int PX, int LF>
    static void record(tms_ctx* c, cudaStream_t s, const LinkT<LF>& U, Field* v, const Field& x, int iters,
                       bool paired = false)
    {
      const Field &r = v[1], &t1 = v[3], &te = v[4];
      const int* stop = &c->st->stop;
      const OpParams* prm = c->prm;
      const ClovT<P> cl = clov<P>(c);
      const int n = nsites(c);
      for (int it = 0; it < iters; it++)
        {
          const bool odd = paired && (it & 1);
          const Field& p = odd ? p2(c) : v[2];
          const Field& pn = (paired && !odd) ? p2(c) : v[2];
          EpiInvClov<P> a1{{view<P>(te), view<P>(te)}, cl, 1};
          launch_hop<P, LF>(c, s, 0, 1, p, p, U, prm, a1, NoFin{}, stop);
          EpiClovKern<P, true> b1{{view<P>(t1), view<P>(t1)}, {view<P>(p), view<P>(p)}, cl, prm, 1};
          launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b1, FinAlpha{c->st}, stop);
          EpiInvClov<P> a2{{view<P>(te), view<P>(te)}, cl, 0};
          launch_hop<P, LF>(c, s, 0, 1, t1, t1, U, prm, a2, NoFin{}, stop);
          if (!paired)
            {
              EpiClovKernCgUpdate<P, PX, 1> b2{view<P>(t1), view<P>(r), view<P>(p), view<PX>(x), cl, prm, c->st};
              launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b2, FinBeta{c->st}, stop);
            }
          else if (!odd)
            {
              EpiClovKernCgUpdate<P, PX, 0> b2{view<P>(t1), view<P>(r), view<P>(p), view<PX>(x), cl, prm, c->st};
              launch_hop<P, LF>(c, s, 1, 1, te, te, U, prm, b2, FinBeta{c->st}, stop);
            }
          else
            {
              EpiClovKernCgUpdate<P, PX, 2> b2{view<P>(t1), view<P>(r), view<P>(p),  view<PX>(x),
                                               cl,           prm,         c->st,        view<P>(v[2])};
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
  // instantiated in tms_cg_clover_half.cu
  extern template tms_status cg_half<ClovOp>(tms_ctx*, int, double, bool, tms_stats*);
}
