// The conjugate-gradient drivers shared by the solver units: FP64, and FP32 /
// FP16 inner with FP64 reliable updates, over an operator policy.  Each
// iteration block is replayed as a CUDA graph.
#pragma once
#include "tms_internal.cuh"
#include <type_traits>

#include <algorithm>

namespace tms_int
{
  // ================================================================ operators
  // A CG "operator policy" fixes the matrix, the fields it works on and the
  // number of sites of its vectors.
  //   EoOp: K(+mu)K(-mu) on odd sites (inv_tmDkern_eoprec_square_eos_cg)
  //   LxOp: Q(+mu)Q(-mu) on the full lattice (inv_tmQ2_cg, and the per-shift
  //         refinement of the multi-shift solver)
  // hi fields (FP64): 0 b, 1 x, 2 r, 3 p, 4-6 temporaries; lo fields (inner
  // precision): 1 r, 2 p, 3-4 temporaries.

  // the policies' first graph slots (FP64, FP32, FP16 follow)
  constexpr int kSlotEo = 0, kSlotLx = 3, kSlotClov = 8;

  // capture a block of iterations once per (slot, fields); replayed every launch
  template <class Rec>
  tms_status capture(tms_ctx* ctx, int slot, const Rec& rec)
  {
    if (ctx->graph[slot]) return TMS_OK;
    cudaStream_t cs;
    CU(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph;
    CU(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    const uint64_t before = ctx->launches;
    rec(cs);
    ctx->graph_nodes[slot] = ctx->launches - before;
    ctx->launches = before;
    const cudaError_t launched = cudaGetLastError(); // a refused launch leaves its node out of the graph
    cudaError_t e = cudaStreamEndCapture(cs, &graph);
    cudaStreamDestroy(cs);
    if (e == cudaSuccess && launched != cudaSuccess) cudaGraphDestroy(graph);
    if (launched != cudaSuccess) e = launched;
    if (e != cudaSuccess) return fail(ctx, TMS_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&ctx->graph[slot], graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail(ctx, TMS_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
    return TMS_OK;
  }

  inline tms_status drop_graph(tms_ctx* ctx, int slot)
  {
    if (ctx->graph[slot])
      {
        CU(cudaStreamSynchronize(ctx->stream));
        cudaGraphExecDestroy(ctx->graph[slot]);
        ctx->graph[slot] = nullptr;
      }
    return TMS_OK;
  }

  inline tms_status launch_graph(tms_ctx* ctx, int slot)
  {
    CU(cudaGraphLaunch(ctx->graph[slot], ctx->stream));
    ctx->launches += ctx->graph_nodes[slot];
    return TMS_OK;
  }

  // One block of iterations: the policy's one-launch kernel while it applies
  // (`one`: decided at a solve's start by one_launch, and given up if the launch
  // is refused or its barrier gives up), else the graph that prepare() captures
  template <class Op, int P, int LF>
  bool one_launch(tms_ctx* ctx)
  {
    if constexpr (Op::kOneLaunch && LF != LINK_H16_12) return Op::template one_launch<P, LF>(ctx);
    else return false;
  }
  template <class Op, int P, int LF, class Prepare>
  tms_status run_block(tms_ctx* ctx, int slot, bool& one, const Prepare& prepare, const LinkT<LF>& U, const Field* v,
                       const Field& x)
  {
    if constexpr (Op::kOneLaunch && LF != LINK_H16_12)
      if (one)
        {
          if (Op::template launch_one<P, LF>(ctx, U, v, x)) return TMS_OK;
          one = false;
        }
    TRY(prepare());
    return launch_graph(ctx, slot);
  }

  inline void fill_stats(tms_stats* stats, tms_status st, int iters, int reliable, double it_res, double true_res, float ms)
  {
    if (!stats) return;
    stats->status = st;
    stats->iterations = iters;
    stats->reliable_updates = reliable;
    stats->iterated_rel_res2 = it_res;
    stats->true_rel_res2 = true_res;
    stats->seconds = ms * 1e-3;
  }

  // ------------------------------------------------------------- CG, FP64
  // b = hi[0], x = hi[1] (initial guess / solution).  cg_invert
  // (cg_invert_template_threaded.hpp:17-150) with the operator of the policy.
  template <class Op>
  tms_status cg_double(tms_ctx* ctx, int niter, double residue, bool have_guess, tms_stats* stats)
  {
    Field* f = Op::hi(ctx);
    const int n = Op::nsites(ctx);
    for (int i = 1; i <= 6; i++) TRY(alloc_field(ctx, f[i], PREC_F64, Op::stride(ctx)));
    double b2;
    TRY(norm2<PREC_F64>(ctx, f[0], &b2, n));
    if (b2 == 0.0 || std::isnan(b2)) return fail(ctx, TMS_ERR_INVALID_SOURCE, "invalid norm: %g", b2);
    double rr;
    if (have_guess) TRY(Op::true_residual(ctx, f[0], f[1], f[2], &rr));
    else
      {
        CU(cudaMemsetAsync(f[1].d, 0, f[1].bytes, ctx->stream));
        CU(cudaMemcpyAsync(f[2].d, f[0].d, f[0].bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        rr = b2;
      }
    CU(cudaMemcpyAsync(f[3].d, f[2].d, f[2].bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    CgState& S = *ctx->st_h;
    memset(&S, 0, sizeof S);
    S.rr = rr;
    S.b2 = b2;
    S.target = residue * b2;
    S.rel_trigger = -1.0;
    S.niter_max = niter;
    S.stop = (rr < S.target) ? STOP_CONVERGED : STOP_RUN;
    TRY(push_state(ctx));
    auto U = links64(ctx);
    Field v[5] = {Field{}, f[2], f[3], f[4], f[5]};
    const int slot = Op::slot0;
    bool one = one_launch<Op, PREC_F64, LINK_F64_18>(ctx);
    auto prepare = [&]() -> tms_status {
      return capture(ctx, slot, [&](cudaStream_t cs) {
        Op::template record<PREC_F64, PREC_F64>(ctx, cs, U, v, f[1], ctx->graph_iters);
      });
    };
    if (!one) TRY(prepare());
    CU(cudaEventRecord(ctx->ev0, ctx->stream));
    while (S.stop == STOP_RUN)
      {
        TRY(run_block<Op, PREC_F64>(ctx, slot, one, prepare, U, v, f[1]));
        TRY(pull_state(ctx));
        if (S.stop != STOP_TIMEOUT) continue;
        // the blocks left at different steps: on with the launches, from x as it is
        one = false;
        TRY(Op::true_residual(ctx, f[0], f[1], f[2], &rr));
        CU(cudaMemcpyAsync(f[3].d, f[2].d, f[2].bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        S.rr = rr;
        S.stop = (rr < S.target) ? STOP_CONVERGED : (S.iter >= niter) ? STOP_MAXITER : STOP_RUN;
        TRY(push_state(ctx));
      }
    CU(cudaEventRecord(ctx->ev1, ctx->stream));
    double tr;
    TRY(Op::true_residual(ctx, f[0], f[1], f[6], &tr));
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    tms_status st = TMS_OK;
    if (S.stop == STOP_BREAKDOWN) st = fail(ctx, TMS_ERR_NAN, "nanned (iteration %d)", S.iter);
    else if (S.stop == STOP_MAXITER) st = fail(ctx, TMS_ERR_NOT_CONVERGED, "exit without converging");
    fill_stats(stats, st, S.iter, 0, S.rr / b2, tr / b2, ms);
    return st;
  }

  // ------------------------------------------------- CG, mixed precision
  // FP32 (or FP16-spinor) inner CG with FP64 reliable updates: the solution is
  // accumulated in FP64 and the residual recomputed with the FP64 operator
  // whenever the iterated residual has dropped by delta since the last update
  // (the outer defect-correction loop of cg_128_invert_template_threaded.cpp:36-109,
  // here with the Krylov direction kept across updates).
  template <class Op, int P, int LF>
  tms_status cg_mixed(tms_ctx* ctx, const LinkT<LF>& U, int niter, double residue, bool have_guess,
                      tms_stats* stats)
  {
    constexpr int PX = (P == PREC_F16) ? PREC_F32 : P; // x accumulates in FP32 at least
    const int slot = Op::slot0 + (P == PREC_F16 ? 2 : 1);
    const int n = Op::nsites(ctx);
    Field* f = Op::hi(ctx);
    for (int i = 1; i <= 6; i++) TRY(alloc_field(ctx, f[i], PREC_F64, Op::stride(ctx)));
    Field* lo = Op::lo(ctx);
    if (Op::lo_prec(ctx) != P)
      {
        // the inner-precision fields move: graphs captured on the old ones are void
        // (the FP32 multi-shift graph uses the full-lattice inner fields too)
        TRY(drop_graph(ctx, Op::slot0 + 1));
        TRY(drop_graph(ctx, Op::slot0 + 2));
        if (Op::slot0 == kSlotLx) TRY(drop_graph(ctx, 7));
        // the twisted-mass and twisted-clover e/o solvers share the inner fields
        if (Op::slot0 == kSlotEo || Op::slot0 == kSlotClov)
          for (int k : {kSlotEo + 1, kSlotEo + 2, kSlotClov + 1, kSlotClov + 2}) TRY(drop_graph(ctx, k));
        for (int i = 0; i < Op::nlo; i++) TRY(alloc_field(ctx, lo[i], P, Op::stride(ctx)));
        Op::lo_prec(ctx) = P;
      }
    Field& xlo = Op::xlo(ctx);
    TRY(alloc_field(ctx, xlo, PX, Op::stride(ctx)));
    const double delta = (P == PREC_F16) ? ctx->delta_half : ctx->delta_single; // reliable-update trigger
    double b2;
    TRY(norm2<PREC_F64>(ctx, f[0], &b2, n));
    if (b2 == 0.0 || std::isnan(b2)) return fail(ctx, TMS_ERR_INVALID_SOURCE, "invalid norm: %g", b2);
    double rr;
    if (have_guess) TRY(Op::true_residual(ctx, f[0], f[1], f[2], &rr, true));
    else
      {
        CU(cudaMemsetAsync(f[1].d, 0, f[1].bytes, ctx->stream));
        CU(cudaMemcpyAsync(f[2].d, f[0].d, f[0].bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        rr = b2;
      }
    const double target = residue * b2;
    CgState& S = *ctx->st_h;
    memset(&S, 0, sizeof S);
    int reliable = 0;
    float ms = 0;
    tms_status st = TMS_OK;
    double last_rt = have_guess ? rr : -1.0; // true residual of the current x, if known
    if (rr >= target)
      {
        convert<P, PREC_F64>(ctx, f[2], lo[1], 1.0, n); // r_lo = r
        convert<P, PREC_F64>(ctx, f[2], lo[2], 1.0, n); // p_lo = r
        CU(cudaMemsetAsync(xlo.d, 0, xlo.bytes, ctx->stream));
        S.rr = rr;
        S.b2 = b2;
        S.target = target;
        S.rel_trigger = delta * delta * rr;
        S.niter_max = niter;
        S.stop = STOP_RUN;
        TRY(push_state(ctx));
        Field v[5] = {Field{}, lo[1], lo[2], lo[3], lo[4]};
        bool one = one_launch<Op, P, LF>(ctx);
        // replays update x every other iteration (e/o operator, even replay length)
        const bool pair = Op::kPaired && ctx->graph_iters % 2 == 0;
        auto prepare = [&]() -> tms_status {
          return capture(ctx, slot, [&](cudaStream_t cs) {
            Op::template record<P, PX>(ctx, cs, U, v, xlo, ctx->graph_iters, pair);
          });
        };
        if (!one) TRY(prepare());
        CU(cudaEventRecord(ctx->ev0, ctx->stream));
        for (;;)
          {
            const int iter0 = S.iter;
            TRY(run_block<Op, P>(ctx, slot, one, prepare, U, v, xlo));
            const bool paired = pair && !one;
            TRY(pull_state(ctx));
            if (S.stop == STOP_RUN) continue;
            if (S.stop == STOP_TIMEOUT)
              {
                // the blocks left at different steps: on with the launches, from the
                // FP64 solution of the last reliable update
                one = false;
                CU(cudaMemsetAsync(xlo.d, 0, xlo.bytes, ctx->stream));
                TRY(Op::true_residual(ctx, f[0], f[1], f[2], &rr, true));
                last_rt = rr;
                if (rr < target) break;
                if (S.iter >= niter)
                  {
                    st = fail(ctx, TMS_ERR_NOT_CONVERGED, "exit without converging");
                    break;
                  }
                convert<P, PREC_F64>(ctx, f[2], lo[1], 1.0, n);
                convert<P, PREC_F64>(ctx, f[2], lo[2], 1.0, n);
                S.rr = rr;
                S.rel_trigger = delta * delta * rr;
                S.stop = STOP_RUN;
                TRY(push_state(ctx));
                continue;
              }
            if (S.stop == STOP_BREAKDOWN)
              {
                st = fail(ctx, TMS_ERR_NAN, "nanned (iteration %d)", S.iter);
                break;
              }
            // a replay cut after an odd number of paired iterations leaves the last
            // step (alpha p, direction in p) out of x; after an even number the
            // direction to keep is in p2
            bool dir_in_p2 = false;
            if constexpr (Op::kPaired)
              if (paired)
                {
                  if ((S.iter - iter0) & 1)
                    {
                      ++ctx->launches;
                      axpby_kernel<PX, PX, P><<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
                        n, 1.0, view<PX>(xlo), S.alpha, view<P>(lo[2]), view<PX>(xlo));
                      CU(cudaGetLastError());
                    }
                  else
                    dir_in_p2 = true;
                }
            // reliable update: x += x_lo (FP64), r = b - A x (FP64)
            ++ctx->launches;
            axpby_kernel<PREC_F64, PREC_F64, PX><<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
              n, 1.0, view<PREC_F64>(f[1]), 1.0, view<PX>(xlo), view<PREC_F64>(f[1]));
            CU(cudaMemsetAsync(xlo.d, 0, xlo.bytes, ctx->stream));
            if (xlo.n) CU(cudaMemsetAsync(xlo.n, 0, sizeof(float) * xlo.stride, ctx->stream));
            double rt;
            TRY(Op::true_residual(ctx, f[0], f[1], f[2], &rt, true));
            reliable++;
            last_rt = rt; // the true residual of the current x
            if (rt < target) break;
            if (S.stop == STOP_MAXITER || S.iter >= niter)
              {
                st = fail(ctx, TMS_ERR_NOT_CONVERGED, "exit without converging");
                break;
              }
            // restart the recurrence from the true residual, keeping the direction
            convert<P, PREC_F64>(ctx, f[2], lo[1], 1.0, n);
            S.beta = rt / S.rr_prev;
            S.rr = rt;
            S.rel_trigger = delta * delta * rt;
            S.stop = STOP_RUN;
            TRY(push_state(ctx));
            ++ctx->launches;
            if constexpr (Op::kPaired)
              if (dir_in_p2)
                {
                  xpay_to_kernel<P><<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
                    n, view<P>(lo[1]), view<P>(Op::p2(ctx)), view<P>(lo[2]), ctx->st, nullptr);
                  CU(cudaGetLastError());
                  continue;
                }
            xpay_kernel<P><<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(n, view<P>(lo[1]),
                                                                                       view<P>(lo[2]), ctx->st,
                                                                                       nullptr);
            CU(cudaGetLastError());
          }
        CU(cudaEventRecord(ctx->ev1, ctx->stream));
        CU(cudaEventSynchronize(ctx->ev1));
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
      }
    // the last reliable update left x with its FP64 true residual; otherwise recompute it
    double tr = last_rt;
    if (tr < 0.0) TRY(Op::true_residual(ctx, f[0], f[1], f[6], &tr, true));
    fill_stats(stats, st, S.iter, reliable, S.rr / b2, tr / b2, ms);
    return st;
  }

  template <class Op>
  tms_status cg_half(tms_ctx* ctx, int niter, double residue, bool have_guess, tms_stats* stats)
  {
    // the e/o twisted-mass solver may run its hops in FP16 arithmetic (tuning "half_arith")
    if constexpr (Op::kHalfArith)
      if (ctx->su3 && ctx->half_arith)
        return cg_mixed<Op, PREC_F16>(ctx, links16h(ctx), niter, residue, have_guess, stats);
    return ctx->su3 ? cg_mixed<Op, PREC_F16>(ctx, links16r(ctx), niter, residue, have_guess, stats)
                    : cg_mixed<Op, PREC_F16>(ctx, links32f(ctx), niter, residue, have_guess, stats);
  }

  template <class Op>
  tms_status cg_dispatch(tms_ctx* ctx, int precision, int niter, double residue, bool have_guess, tms_stats* stats)
  {
    if (precision == TMS_PREC_DOUBLE) return cg_double<Op>(ctx, niter, residue, have_guess, stats);
    if (precision == TMS_PREC_MIXED_SINGLE)
      {
        if (!ctx->su3) return cg_mixed<Op, PREC_F32>(ctx, links32f(ctx), niter, residue, have_guess, stats);
        return ctx->single_links16 ? cg_mixed<Op, PREC_F32>(ctx, links16r(ctx), niter, residue, have_guess, stats)
                                   : cg_mixed<Op, PREC_F32>(ctx, links32r(ctx), niter, residue, have_guess, stats);
      }
    if (precision == TMS_PREC_MIXED_HALF) return cg_half<Op>(ctx, niter, residue, have_guess, stats);
    return fail(ctx, TMS_ERR_BAD_ARG, "unknown precision %d", precision);
  }

  // Eq. (8)-(11) on device fields (tms_cg.cu): the source's parities in ex[0]
  // (even) and ex[1] (odd), the solution's in ex[2], ex[3]
  tms_status eo_full_solve(tms_ctx* ctx, int niter, double residue, int precision, tms_stats* stats,
                           const double* guess_Koo = nullptr);
}
