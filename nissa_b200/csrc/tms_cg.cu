// C ABI of the e/o solvers: the CG of K(+mu)K(-mu) (FP64, and FP32 / FP16
// inner with FP64 reliable updates) and the full solve of Eq. (8)-(11).
#include "tms_eo_op.cuh"

using namespace tms_int;

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
    for (double*& b : ctx->colbuf) CU(dev_alloc(ctx, &b, bytes));
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
