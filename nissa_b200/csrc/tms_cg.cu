// C ABI of the e/o solvers: the CG of K(+mu)K(-mu) (FP64, and FP32 / FP16
// inner with FP64 reliable updates) and the full solve of Eq. (8)-(11).
#include "tms_solver.cuh"
#include "tms_cg_small.cuh"

using namespace tms_int;

namespace
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

    // The one-launch CG: the default hop shape, and every 32-site block resident
    // at once (two per SM: up to 9472 sites of a parity).  Whole solves, launches /
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
      if (c->hop_cfg[P] != HOP_CFG_DEFAULT[P]) return false;
      int coop = 0, sms = 0, per = 0;
      if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) != cudaSuccess || !coop ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, one_kernel<P, LF>(), HOP_DP_THREADS, 0) != cudaSuccess)
        return false;
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
    static tms_status launch_one(tms_ctx* ctx, const LinkT<LF>& U, const Field* v, const Field& x)
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
      int iters = kOneIters;
      void* args[] = {&g, &r, &p, &t1, &te, &xx, &u, &prm, &st, &partial, &bar, &iters};
      ctx->launches += 2;
      grid_bar_reset_kernel<<<1, 1, 0, ctx->stream>>>(bar);
      CU(cudaLaunchCooperativeKernel((const void*)one_kernel<P, LF>(), dim3(div_up(g.Vh, HOP_DP_SITES)), dim3(HOP_DP_THREADS),
                                     args, 0, ctx->stream));
      return TMS_OK;
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

extern "C" {

tms_status tms_cg_eoprec_square(tms_ctx* ctx, double* sol, const double* guess, const double* src, double kappa,
                                int has_anis, double anis, double mu, int niter, double residue, int precision,
                                tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (!sol || !src || niter <= 0 || !(residue > 0)) return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  TRY(set_params(ctx, kappa, mu, has_anis, anis));
  Field* f = ctx->f64;
  TRY(spinor_in(ctx, src, f[0]));
  if (guess) TRY(spinor_in(ctx, guess, f[1]));
  const tms_status st = cg_dispatch<EoOp>(ctx, precision, niter, residue, guess != nullptr, stats);
  if (st == TMS_OK || st == TMS_ERR_NOT_CONVERGED) TRY(spinor_out(ctx, f[1], sol));
  TRY(finish(ctx));
  return st;
}

} // extern "C"

namespace
{
  // Eq. (8)-(11) of inv_tmD_cg_eoprec_native (cg_invert_tmD_eoprec.cpp:102-150) on
  // device fields: the source's parities in ex[0] (even) and ex[1] (odd), the
  // solution's in ex[2], ex[3].  The operator parameters must be set.
  // (the FP64 steps around a mixed-precision solve read the links as 12 reals
  // when the conf is SU(3) to rounding; the FP64 solve reads all 18)
  template <int LF>
  tms_status eo_full_solve_t(tms_ctx* ctx, const LinkT<LF>& U, int niter, double residue, int precision,
                             tms_stats* stats, const double* guess_Koo)
  {
    Field* f = ctx->f64;
    for (int i = 0; i <= 7; i++) TRY(alloc_field(ctx, f[i], PREC_F64));
    Field *eta = ctx->ex, *psi = ctx->ex + 2; // [0] even, [1] odd
    const int n = (int)ctx->g.Vh;
    auto V = [&](const Field& x) { return view<PREC_F64>(x); };
    // Eq. (8a): te = D_ee^-1 eta_e ; Eq. (8b): varphi = g5 (eta_o + hop(te)/2) -> f0
    ++ctx->launches;
    diag_kernel<PREC_F64><<<div_up(n, 256), 256, 0, ctx->stream>>>(n, V(eta[0]), V(f[5]), ctx->prm, 1.0, 1);
    EpiSrcPrep<PREC_F64> sp{{V(f[0]), V(f[0])}, {V(eta[1]), V(eta[1])}};
    launch_hop<PREC_F64, LF>(ctx, ctx->stream, 1, 1, f[5], f[5], U, ctx->prm, sp);
    CU(cudaGetLastError());
    // Eq. (9), from the caller's odd-site guess when given
    if (guess_Koo) TRY(spinor_in(ctx, guess_Koo, f[1]));
    const tms_status st = cg_dispatch<EoOp>(ctx, precision, niter, residue, guess_Koo != nullptr, stats);
    if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
    // Eq. (10): psi_o = K(-mu) x ; Eq. (11): psi_e = D_ee^-1 (eta_e + hop(psi_o)/2)
    kern_op<PREC_F64>(ctx, U, f[1], f[5], psi[1], -1.0, ctx->prm);
    EpiReco<PREC_F64> rc{{V(psi[0]), V(psi[0])}, {V(eta[0]), V(eta[0])}, ctx->prm, 1.0};
    launch_hop<PREC_F64, LF>(ctx, ctx->stream, 0, 1, psi[1], psi[1], U, ctx->prm, rc);
    CU(cudaGetLastError());
    return st;
  }
}

namespace tms_int
{
  tms_status eo_full_solve(tms_ctx* ctx, int niter, double residue, int precision, tms_stats* stats,
                           const double* guess_Koo)
  {
    if (precision != TMS_PREC_DOUBLE && reliable_links12(ctx))
      return eo_full_solve_t(ctx, links64r(ctx), niter, residue, precision, stats, guess_Koo);
    return eo_full_solve_t(ctx, links64(ctx), niter, residue, precision, stats, guess_Koo);
  }
}

namespace
{
  // inv_tmD_cg_eoprec between AoS lx spinors in device memory (the operator
  // parameters set): split the source into its parities, Eq. (8)-(11), paste
  // the solution's parities, then the reference's lx residual check.  When
  // given, `src_read` is recorded on the stream once the source has been read
  // and `dst_ready` once the solution is written.
  tms_status cg_eoprec_lx(tms_ctx* ctx, double* dst, const double* src, int niter, double residue, int precision,
                          tms_stats* stats, cudaEvent_t src_read, cudaEvent_t dst_ready,
                          const double* guess_Koo = nullptr)
  {
    Field* f = ctx->f64;
    for (int i = 0; i <= 7; i++) TRY(alloc_field(ctx, f[i], PREC_F64));
    Field *eta = ctx->ex, *psi = ctx->ex + 2; // [0] even, [1] odd
    for (auto& e : ctx->ex) TRY(alloc_field(ctx, e, PREC_F64));
    const int n = (int)ctx->g.Vh;
    const int lxblocks = div_up(ctx->g.V, LXCOPY_THREADS);
    auto V = [&](const Field& x) { return view<PREC_F64>(x); };
    // split_lx_vector_into_eo_parts(source)
    ++ctx->launches;
    lx_split_kernel<PREC_F64><<<lxblocks, LXCOPY_THREADS, 0, ctx->stream>>>(ctx->g, src, V(eta[0]), V(eta[1]));
    CU(cudaGetLastError());
    if (src_read) CU(cudaEventRecord(src_read, ctx->stream));
    const tms_status st = eo_full_solve(ctx, niter, residue, precision, stats, guess_Koo);
    if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
    // paste_eo_parts_into_lx_vector
    ++ctx->launches;
    lx_paste_kernel<PREC_F64><<<lxblocks, LXCOPY_THREADS, 0, ctx->stream>>>(ctx->g, V(psi[0]), V(psi[1]), dst);
    CU(cudaGetLastError());
    if (dst_ready) CU(cudaEventRecord(dst_ready, ctx->stream));
    // lx residual check (cg_invert_tmD_eoprec.cpp:192-212): |g5 Q sol - src|^2 / |src|^2
    if (stats)
      {
        EpiTmQ<PREC_F64, false> e{{V(f[2]), V(f[3])}, {V(psi[0]), V(psi[1])}, ctx->prm, +1.0};
        launch_hop<PREC_F64, LINK_F64_18>(ctx, ctx->stream, 0, 2, psi[0], psi[1], links64(ctx), ctx->prm, e);
        double num = 0, den = 0;
        for (int par = 0; par < 2; par++)
          {
            ++ctx->launches;
            g5_residual_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(n, V(f[2 + par]),
                                                                                         V(eta[par]), reducer(ctx));
            CU(cudaGetLastError());
            num += read_result(ctx);
            double e2;
            TRY(norm2<PREC_F64>(ctx, eta[par], &e2));
            den += e2;
          }
        stats->lx_rel_res2 = num / den;
      }
    return st;
  }

  // the copy stream, the staging buffers and the events of pipelined column solves
  tms_status ensure_columns(tms_ctx* ctx, size_t bytes)
  {
    if (!ctx->cstream) CU(cudaStreamCreateWithFlags(&ctx->cstream, cudaStreamNonBlocking));
    for (cudaEvent_t& e : ctx->colev)
      if (!e) CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if (ctx->colbuf_bytes >= bytes) return TMS_OK;
    for (double*& b : ctx->colbuf)
      {
        if (b) cudaFree(b);
        b = nullptr;
      }
    ctx->colbuf_bytes = 0;
    for (double*& b : ctx->colbuf) CU(cudaMalloc(&b, bytes));
    ctx->colbuf_bytes = bytes;
    return TMS_OK;
  }

  // Column k's source is copied in while column k-1 is solved, and its solution
  // copied out while column k+1 is solved: two staging buffers each way on a
  // copy stream, ordered against the solver's stream by events.
  tms_status columns_host(tms_ctx* ctx, int ncols, double* const* sols, const double* const* srcs, int niter,
                          double residue, int precision, tms_stats* stats, size_t bytes)
  {
    cudaEvent_t* in_ready = ctx->colev;
    cudaEvent_t* in_free = ctx->colev + 2;
    cudaEvent_t* out_ready = ctx->colev + 4;
    cudaEvent_t* out_free = ctx->colev + 6;
    double** in = ctx->colbuf;
    double** out = ctx->colbuf + 2;
    cudaStream_t cs = ctx->cstream;
    CU(cudaMemcpyAsync(in[0], srcs[0], bytes, cudaMemcpyHostToDevice, cs));
    CU(cudaEventRecord(in_ready[0], cs));
    tms_status worst = TMS_OK;
    for (int k = 0; k < ncols; k++)
      {
        const int b = k & 1;
        if (k + 1 < ncols)
          {
            const int nb = (k + 1) & 1;
            if (k >= 1) CU(cudaStreamWaitEvent(cs, in_free[nb], 0)); // column k-1 has read it
            CU(cudaMemcpyAsync(in[nb], srcs[k + 1], bytes, cudaMemcpyHostToDevice, cs));
            CU(cudaEventRecord(in_ready[nb], cs));
          }
        CU(cudaStreamWaitEvent(ctx->stream, in_ready[b], 0));
        if (k >= 2) CU(cudaStreamWaitEvent(ctx->stream, out_free[b], 0)); // column k-2 has been copied out
        const tms_status st = cg_eoprec_lx(ctx, out[b], in[b], niter, residue, precision, stats ? stats + k : nullptr,
                                           in_free[b], out_ready[b]);
        if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
        if (st != TMS_OK) worst = st;
        CU(cudaStreamWaitEvent(cs, out_ready[b], 0));
        CU(cudaMemcpyAsync(sols[k], out[b], bytes, cudaMemcpyDeviceToHost, cs));
        CU(cudaEventRecord(out_free[b], cs));
      }
    return worst;
  }
}

extern "C" {

tms_status tms_cg_eoprec(tms_ctx* ctx, double* sol_lx, const double* src_lx, double kappa, int has_anis, double anis,
                         double mu, int niter, double residue, int precision, tms_stats* stats)
{
  return tms_cg_eoprec_guess(ctx, sol_lx, nullptr, src_lx, kappa, has_anis, anis, mu, niter, residue, precision,
                             stats);
}

tms_status tms_cg_eoprec_guess(tms_ctx* ctx, double* sol_lx, const double* guess_Koo, const double* src_lx,
                               double kappa, int has_anis, double anis, double mu, int niter, double residue,
                               int precision, tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (!sol_lx || !src_lx || niter <= 0 || !(residue > 0)) return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  TRY(set_params(ctx, kappa, mu, has_anis, anis));
  const size_t bytes = (size_t)ctx->g.V * 24 * sizeof(double);
  const double* src = src_lx;
  double* dst = sol_lx;
  if (ctx->ptr_mode == TMS_PTR_HOST)
    {
      TRY(ensure_stage(ctx, bytes));
      CU(cudaMemcpyAsync(ctx->stage, src_lx, bytes, cudaMemcpyHostToDevice, ctx->stream));
      src = dst = ctx->stage; // the source is split before the solution is pasted
    }
  const tms_status st = cg_eoprec_lx(ctx, dst, src, niter, residue, precision, stats, nullptr, nullptr, guess_Koo);
  if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
  if (ctx->ptr_mode == TMS_PTR_HOST) CU(cudaMemcpyAsync(sol_lx, ctx->stage, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  TRY(finish(ctx));
  return st;
}

tms_status tms_cg_eoprec_columns(tms_ctx* ctx, int ncols, double* const* sols_lx, const double* const* srcs_lx,
                                 double kappa, int has_anis, double anis, double mu, int niter, double residue,
                                 int precision, tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (ncols <= 0 || !sols_lx || !srcs_lx || niter <= 0 || !(residue > 0))
    return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  for (int k = 0; k < ncols; k++)
    if (!sols_lx[k] || !srcs_lx[k]) return fail(ctx, TMS_ERR_BAD_ARG, "column %d: null pointer", k);
  TRY(set_params(ctx, kappa, mu, has_anis, anis));
  tms_status st = TMS_OK;
  if (ctx->ptr_mode == TMS_PTR_DEVICE)
    {
      for (int k = 0; k < ncols; k++)
        {
          const tms_status s = cg_eoprec_lx(ctx, sols_lx[k], srcs_lx[k], niter, residue, precision,
                                            stats ? stats + k : nullptr, nullptr, nullptr);
          if (s != TMS_OK && s != TMS_ERR_NOT_CONVERGED) return s;
          if (s != TMS_OK) st = s;
        }
      TRY(finish(ctx));
      return st;
    }
  const size_t bytes = (size_t)ctx->g.V * 24 * sizeof(double);
  TRY(ensure_columns(ctx, bytes));
  st = columns_host(ctx, ncols, sols_lx, srcs_lx, niter, residue, precision, stats, bytes);
  // no copy into or out of the caller's buffers outlives the call, whatever the outcome
  const cudaError_t e = cudaStreamSynchronize(ctx->cstream);
  if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
  if (e != cudaSuccess) return fail(ctx, TMS_ERR_CUDA, "column copies: %s", cudaGetErrorString(e));
  TRY(finish(ctx));
  return st;
}

} // extern "C"
