// C ABI of the twisted-clover solvers: the e/o CG of K(false)K(true) and the
// full solve, with the CG drivers of tms_solver.cuh.
#include "tms_clov_op.cuh"

using namespace tms_int;

extern "C" {

tms_status tms_cg_tmclov_eoprec_square(tms_ctx* ctx, double* sol, const double* guess, const double* src, double kappa,
                                       int has_anis, double anis, double mu, int niter, double residue, int precision,
                                       tms_stats* stats)
{
  TRY(check_clover(ctx));
  if (!sol || !src || niter <= 0 || !(residue > 0)) return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  TRY(set_params(ctx, kappa, mu, has_anis, anis));
  TRY(ensure_clover_inverse(ctx, kappa, mu));
  Field* f = ctx->f64;
  TRY(spinor_in(ctx, src, f[0]));
  if (guess) TRY(spinor_in(ctx, guess, f[1]));
  const tms_status st = cg_dispatch<ClovOp>(ctx, precision, niter, residue, guess != nullptr, stats);
  if (st == TMS_OK || st == TMS_ERR_NOT_CONVERGED) TRY(spinor_out(ctx, f[1], sol));
  TRY(finish(ctx));
  return st;
}

tms_status tms_cg_tmclov_eoprec(tms_ctx* ctx, double* sol_lx, const double* src_lx, double kappa, int has_anis,
                                double anis, double cSW, double mu, int niter, double residue, int precision,
                                tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (!sol_lx || !src_lx || niter <= 0 || !(residue > 0)) return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  // clover_term(Cl, cSW, conf) and invert_twisted_clover_term(invCl, mu, kappa, Cl) of the call
  // (cg_invert_tmclovD_eoprec.cpp:72-76), kept across calls with the same conf and parameters
  if (!ctx->clov_ok || ctx->clov_csw != cSW) TRY(tms_clover_term(ctx, cSW));
  TRY(set_params(ctx, kappa, mu, has_anis, anis));
  TRY(ensure_clover_inverse(ctx, kappa, mu));
  Field* f = ctx->f64;
  for (int i = 0; i <= 7; i++) TRY(alloc_field(ctx, f[i], PREC_F64));
  Field *eta = ctx->ex, *psi = ctx->ex + 2; // [0] even, [1] odd
  for (auto& e : ctx->ex) TRY(alloc_field(ctx, e, PREC_F64));
  const int n = (int)ctx->g.Vh;
  const size_t bytes = (size_t)ctx->g.V * 24 * sizeof(double);
  auto V = [&](const Field& x) { return view<PREC_F64>(x); };
  auto U = links64(ctx);
  const double* src = src_lx;
  if (ctx->ptr_mode == TMS_PTR_HOST)
    {
      TRY(ensure_stage(ctx, bytes));
      CU(cudaMemcpyAsync(ctx->stage, src_lx, bytes, cudaMemcpyHostToDevice, ctx->stream));
      src = ctx->stage;
    }
  launch_lx_split(ctx, src, V(eta[0]), V(eta[1]));
  // Eq. (8a): te = T_ee^-1 eta_e ; Eq. (8b): varphi = g5 (eta_o + hop(te)/2) -> f0  (:84-90)
  inv_clov_apply(ctx, eta[0], f[5], 0);
  EpiSrcPrep<PREC_F64> sp{{V(f[0]), V(f[0])}, {V(eta[1]), V(eta[1])}};
  launch_hop<PREC_F64, LINK_F64_18>(ctx, ctx->stream, 1, 1, f[5], f[5], U, ctx->prm, sp);
  CU(cudaGetLastError());
  // Eq. (9)
  const tms_status st = cg_dispatch<ClovOp>(ctx, precision, niter, residue, false, stats);
  if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
  // Eq. (10): psi_o = K(dag) x ; Eq. (11): psi_e = T_ee^-1 (eta_e + hop(psi_o)/2)  (:97-107)
  clov_kern_op<PREC_F64>(ctx, U, clov64(ctx), f[1], f[5], psi[1], 1, ctx->prm);
  EpiClovReco<PREC_F64> rc{{V(psi[0]), V(psi[0])}, {V(eta[0]), V(eta[0])}, clov64(ctx)};
  launch_hop<PREC_F64, LINK_F64_18>(ctx, ctx->stream, 0, 1, psi[1], psi[1], U, ctx->prm, rc);
  CU(cudaGetLastError());
  double* d = (ctx->ptr_mode == TMS_PTR_HOST) ? ctx->stage : sol_lx;
  launch_lx_paste(ctx, V(psi[0]), V(psi[1]), d);
  CU(cudaGetLastError());
  if (ctx->ptr_mode == TMS_PTR_HOST) CU(cudaMemcpyAsync(sol_lx, ctx->stage, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  // the residual check of inv_tmclovD_cg_eoprec (:140-175): |g5 Q_clov sol - src|^2 / |src|^2
  if (stats)
    {
      tmclovQ_op(ctx, psi[0], psi[1], f[2], f[3], ctx->prm);
      double num = 0, den = 0;
      for (int par = 0; par < 2; par++)
        {
          ++ctx->launches;
          g5_residual_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(n, V(f[2 + par]), V(eta[par]),
                                                                                       reducer(ctx));
          CU(cudaGetLastError());
          num += read_result(ctx);
          double e2;
          TRY(norm2<PREC_F64>(ctx, eta[par], &e2));
          den += e2;
        }
      stats->lx_rel_res2 = num / den;
    }
  TRY(finish(ctx));
  return st;
}

} // extern "C"
