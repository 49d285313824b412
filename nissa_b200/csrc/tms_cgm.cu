// C ABI of the full-lattice solvers: the CG of Q(+m)Q(-m) and the multi-shift
// CGM of the tm Q^2 operator, with the CG drivers of tms_solver.cuh.
#include "tms_solver.cuh"

using namespace tms_int;

namespace
{
  struct LxOp
  {
    static constexpr int slot0 = kSlotLx;
    static constexpr bool kHalfArith = false;
    static constexpr bool kOneLaunch = false;
    static constexpr bool kPaired = false;
    static constexpr int nlo = 5;
    static int stride(tms_ctx* c) { return 2 * c->g.stride; }
    static int nsites(tms_ctx* c) { return 2 * c->g.stride; }
    static Field* hi(tms_ctx* c) { return c->lx64; }
    static Field* lo(tms_ctx* c) { return c->lxlo; }
    static int& lo_prec(tms_ctx* c) { return c->lxlo_prec; }
    static Field& xlo(tms_ctx* c) { return c->lxxlo; }

    template <int P>
    static void qop(tms_ctx* c, cudaStream_t s, const Field& in, const Field& out, double sgn, const OpParams* prm)
    {
      EpiTmQ<P, false> e{{view_par<P>(out, 0), view_par<P>(out, 1)}, {view_par<P>(in, 0), view_par<P>(in, 1)}, prm,
                         sgn};
      launch_hop_v<P, LINK_F64_18>(c, s, 0, 2, view_par<P>(in, 0), view_par<P>(in, 1), links64(c), prm, e);
    }

    // r = b - Q(+mu)Q(-mu) x in FP64; returns |r|^2 (uses hi 4, 5); 18-real links always
    static tms_status true_residual(tms_ctx* ctx, const Field& b, const Field& x, const Field& r, double* rr,
                                    bool = false)
    {
      Field &t = ctx->lx64[4], &s = ctx->lx64[5];
      qop<PREC_F64>(ctx, ctx->stream, x, t, -1.0, ctx->prm);
      qop<PREC_F64>(ctx, ctx->stream, t, s, +1.0, ctx->prm);
      const int n = nsites(ctx);
      ++ctx->launches;
      residual_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
        n, view<PREC_F64>(b), view<PREC_F64>(s), view<PREC_F64>(r), reducer(ctx));
      CU(cudaGetLastError());
      *rr = read_result(ctx);
      return TMS_OK;
    }

    // `iters` CG iterations: t = Q(-mu) p reducing |t|^2 ; s = Q(+mu) t fused
    // with the x and r updates ; p = r + beta p.   v 1 r, 2 p, 3 t
    template <int P, int PX, int LF>
    static void record(tms_ctx* c, cudaStream_t s, const LinkT<LF>& U, Field* v, const Field& x, int iters,
                       bool = false)
    {
      const Field &r = v[1], &p = v[2], &t = v[3];
      const int* stop = &c->st->stop;
      const OpParams* prm = c->prm;
      auto V = [](const Field& f, int par) { return view_par<P>(f, par); };
      for (int it = 0; it < iters; it++)
        {
          EpiTmQ<P, true> a{{V(t, 0), V(t, 1)}, {V(p, 0), V(p, 1)}, prm, -1.0};
          launch_hop_v<P, LF>(c, s, 0, 2, V(p, 0), V(p, 1), U, prm, a, FinAlpha{c->st}, stop);
          EpiTmQCgUpdate<P, PX> b{{V(t, 0), V(t, 1)},
                                  {V(r, 0), V(r, 1)},
                                  {V(p, 0), V(p, 1)},
                                  {view_par<PX>(x, 0), view_par<PX>(x, 1)},
                                  prm,
                                  c->st,
                                  +1.0};
          launch_hop_v<P, LF>(c, s, 0, 2, V(t, 0), V(t, 1), U, prm, b, FinBeta{c->st}, stop);
          const int n = nsites(c);
          ++c->launches;
          launch_pdl(c, xpay_kernel<P>, div_up(n, BLAS_THREADS), BLAS_THREADS, 0, s, n, view<P>(r), view<P>(p),
                     (const CgState*)c->st, stop);
        }
    }
  };

  // ------------------------------------------------------ multi-shift CGM
  // cgm_invert (cgm_invert_template_threaded.hpp:11-295) on Q_W^2 = Q(0)Q(0),
  // shifts sigma_i = m_i^2, for the source in lx64[0].  Vectors in precision P;
  // solutions left in ctx->cgm_x.  Returns the solver status, *iters the
  // iteration count (the reference's final_iter).
  size_t per_site_bytes(int prec) { return prec == PREC_F64 ? 192 : prec == PREC_F32 ? 96 : 52; }

  // iterations whose shift updates are applied together: the largest divisor of
  // the replay length up to CGM_MAX_WINDOW (a replay starts and ends a window)
  int cgm_window(int graph_iters)
  {
    int w = std::min(graph_iters, CGM_MAX_WINDOW);
    while (graph_iters % w) w--;
    return w;
  }

  // The residuals of a window besides the running one.  They lie in full-lattice
  // FP64 fields that are idle while the multi-shift iteration runs (what is in
  // them is written anew after it): FP32 finds room for eight, FP64 for three.
  // An FP64 window of more takes the rest from ctx->cgm_r, or is shortened to a
  // divisor of `want` where memory is short.
  struct CgmStore
  {
    std::vector<void*> r;
    int window = 1;
  };
  // ctx->cgm_r outlives the call while it is at most this part of what is then free
  // (allocated on each call it costs 2.5 of 161 ms, 8 masses at 24^3x48), and until
  // an allocation of the context fails
  constexpr size_t CGM_KEEP_PART = 64;

  tms_status find_window(tms_ctx* ctx, int prec, size_t fbytes, int want, CgmStore& st)
  {
    const bool hi = prec == PREC_F64;
    std::vector<Field*> idle;
    if (hi) idle = {&ctx->lx64[1], &ctx->lx64[5], &ctx->lx64[6]};
    else idle = {&ctx->lx64[1], &ctx->lx64[2], &ctx->lx64[3], &ctx->lx64[4]};
    // sites of the padding stay zero in every layout that a field is read in
    if (ctx->g.stride != ctx->g.Vh)
      for (Field* f : idle) CU(cudaMemsetAsync(f->d, 0, f->bytes, ctx->stream));
    for (Field* f : idle)
      for (size_t o = 0; o + fbytes <= f->bytes; o += fbytes) st.r.push_back((unsigned char*)f->d + o);
    const int have = (int)st.r.size();
    // what the rest of the call may still allocate stays free
    const size_t reserve = (size_t)32 * 192 * ctx->g.stride;
    int w = want;
    for (; w > 1; w--)
      {
        if (want % w) continue;
        const size_t more = w - 1 > have ? fbytes * (w - 1 - have) : 0;
        if (more <= ctx->cgm_r_bytes) break;
        drop_window(ctx);
        size_t avail = 0, total = 0;
        CU(cudaMemGetInfo(&avail, &total));
        if (avail < more + reserve) continue;
        if (cudaMalloc(&ctx->cgm_r, more) == cudaSuccess)
          {
            ctx->cgm_r_bytes = more;
            CU(cudaMemsetAsync(ctx->cgm_r, 0, more, ctx->stream));
            break;
          }
        ctx->cgm_r = nullptr;
        cudaGetLastError(); // out of memory: a shorter window
      }
    for (size_t o = 0; o + fbytes <= ctx->cgm_r_bytes; o += fbytes) st.r.push_back((unsigned char*)ctx->cgm_r + o);
    st.window = w;
    // a graph holds the addresses it was captured with
    if (hi && (ctx->cgm_graph_window != w || ctx->cgm_graph_r != ctx->cgm_r))
      {
        TRY(drop_graph(ctx, 6));
        ctx->cgm_graph_window = w;
        ctx->cgm_graph_r = ctx->cgm_r;
      }
    return TMS_OK;
  }

  template <int W, class V, class R, class Get>
  void cgm_flush_w(tms_ctx* ctx, cudaStream_t s, const Get& get, int64_t words)
  {
    CgmWindow<W, V> win;
    for (int w = 0; w < W; w++) win.r[w] = get(w);
    cgm_flush_kernel<W, V, R><<<div_up(words, CGM_FLUSH_THREADS), CGM_FLUSH_THREADS, 0, s>>>(
      words, win, (V*)ctx->cgm_x, (V*)ctx->cgm_ps, words, ctx->cgm);
  }

  // the shift updates of the W iterations since the last flush
  template <class V, class R, class Get>
  void cgm_flush(tms_ctx* ctx, cudaStream_t s, int W, const Get& get, int64_t words)
  {
    ctx->launches += 2;
    switch (W)
      {
      case 8: cgm_flush_w<8, V, R>(ctx, s, get, words); break;
      case 7: cgm_flush_w<7, V, R>(ctx, s, get, words); break;
      case 6: cgm_flush_w<6, V, R>(ctx, s, get, words); break;
      case 5: cgm_flush_w<5, V, R>(ctx, s, get, words); break;
      case 4: cgm_flush_w<4, V, R>(ctx, s, get, words); break;
      case 3: cgm_flush_w<3, V, R>(ctx, s, get, words); break;
      case 2: cgm_flush_w<2, V, R>(ctx, s, get, words); break;
      default: cgm_flush_w<1, V, R>(ctx, s, get, words);
      }
    cgm_flushed_kernel<<<1, 1, 0, s>>>(ctx->cgm);
  }

  template <int P, int LF>
  tms_status cgm_run(tms_ctx* ctx, const LinkT<LF>& U, int nshift, const double* sigma, const double* target,
                     int niter, double b2, int* iters, float* ms)
  {
    const int slot = (P == PREC_F64) ? 6 : 7;
    const int stride = 2 * ctx->g.stride, n = stride;
    const size_t fbytes = per_site_bytes(P) * (size_t)stride;
    if (ctx->cgm_prec != P || ctx->cgm_nshift < nshift)
      {
        TRY(drop_graph(ctx, 6));
        TRY(drop_graph(ctx, 7));
        if (ctx->cgm_x) cudaFree(ctx->cgm_x);
        if (ctx->cgm_ps) cudaFree(ctx->cgm_ps);
        ctx->cgm_x = ctx->cgm_ps = nullptr;
        ctx->cgm_prec = -1;
        CU(dev_alloc(ctx, &ctx->cgm_x, fbytes * nshift));
        CU(dev_alloc(ctx, &ctx->cgm_ps, fbytes * nshift));
        ctx->cgm_prec = P;
        ctx->cgm_nshift = nshift;
      }
    // inner vectors: r, p, t in precision P (FP64: hi 2-4, otherwise lo 1-3)
    if (P == PREC_F64)
      {
        for (int i = 2; i <= 4; i++) TRY(alloc_field(ctx, ctx->lx64[i], PREC_F64, stride));
      }
    else if (ctx->lxlo_prec != P)
      {
        TRY(drop_graph(ctx, LxOp::slot0 + 1));
        TRY(drop_graph(ctx, LxOp::slot0 + 2));
        for (int i = 0; i < LxOp::nlo; i++) TRY(alloc_field(ctx, ctx->lxlo[i], P, stride));
        ctx->lxlo_prec = P;
      }
    const bool hi = (P == PREC_F64);
    const Field& r = hi ? ctx->lx64[2] : ctx->lxlo[1];
    const Field& p = hi ? ctx->lx64[3] : ctx->lxlo[2];
    const Field& t = hi ? ctx->lx64[4] : ctx->lxlo[3];
    CgmStore store;
    TRY(find_window(ctx, P, fbytes, cgm_window(ctx->graph_iters), store));
    // the window's residuals: iteration j of a window writes R(j), reading its predecessor's
    const int W = store.window;
    auto R = [&](int j) {
      Field f = r;
      if (j < W - 1) f.d = store.r[j];
      return f;
    };
    // solution / direction views of shift k
    auto shift_field = [&](void* base, int k) {
      Field f;
      f.prec = P;
      f.d = (unsigned char*)base + fbytes * k;
      f.n = nullptr;
      f.stride = stride;
      f.bytes = fbytes;
      return f;
    };
    // r = p = b ; ps_i = b ; x_i = 0
    convert<P, PREC_F64>(ctx, ctx->lx64[0], r, 1.0, n);
    convert<P, PREC_F64>(ctx, ctx->lx64[0], p, 1.0, n);
    for (int k = 0; k < nshift; k++) convert<P, PREC_F64>(ctx, ctx->lx64[0], shift_field(ctx->cgm_ps, k), 1.0, n);
    CU(cudaMemsetAsync(ctx->cgm_x, 0, fbytes * nshift, ctx->stream));
    CgmState& S = *ctx->cgm_h;
    memset(&S, 0, sizeof S);
    S.rr = b2;
    S.b2 = b2;
    S.betaa = 1.0;
    S.alpha = 0.0;
    S.nshift = nshift;
    S.nrun = nshift;
    S.niter_max = niter;
    for (int k = 0; k < nshift; k++)
      {
        S.sigma[k] = sigma[k];
        S.target[k] = target[k];
        S.zps[k] = S.zas[k] = 1.0;
        S.alphas[k] = 0.0;
        S.run[k] = 1;
      }
    CU(cudaMemcpyAsync(ctx->cgm, &S, sizeof S, cudaMemcpyHostToDevice, ctx->stream));
    const OpParams* prm = ctx->prm + 1; // the CGM operator: mu = 0
    using Word = typename std::conditional<P == PREC_F64, double2, float4>::type;
    const int64_t words = (int64_t)(fbytes / sizeof(Word));
    TRY(capture(ctx, slot, [&](cudaStream_t cs) {
      auto V = [](const Field& f, int par) { return view_par<P>(f, par); };
      const int* stop = &ctx->cgm->stop;
      for (int it = 0; it < ctx->graph_iters; it++)
        {
          const int j = it % W;
          const Field rin = R((j + W - 1) % W), rout = R(j);
          EpiTmQ<P, true> a{{V(t, 0), V(t, 1)}, {V(p, 0), V(p, 1)}, prm, +1.0};
          launch_hop_v<P, LF>(ctx, cs, 0, 2, V(p, 0), V(p, 1), U, prm, a, FinCgm1{ctx->cgm}, stop);
          EpiCgm2<P> b{{V(t, 0), V(t, 1)}, {V(rin, 0), V(rin, 1)}, {V(rout, 0), V(rout, 1)}, prm, ctx->cgm};
          launch_hop_v<P, LF>(ctx, cs, 0, 2, V(t, 0), V(t, 1), U, prm, b, FinCgm2{ctx->cgm, j}, stop);
          ++ctx->launches;
          cgm_p_kernel<P><<<div_up(n, 256), 256, 0, cs>>>(n, view<P>(rout), view<P>(p), ctx->cgm);
          if (j == W - 1)
            cgm_flush<Word, typename SpinorT<P>::R>(ctx, cs, W, [&](int w) { return (const Word*)R(w).d; }, words);
        }
    }));
    CU(cudaEventRecord(ctx->ev0, ctx->stream));
    do
      {
        TRY(launch_graph(ctx, slot));
        CU(cudaMemcpyAsync(ctx->cgm_h, ctx->cgm, sizeof(CgmState), cudaMemcpyDeviceToHost, ctx->stream));
        CU(cudaStreamSynchronize(ctx->stream));
      }
    while (S.stop == STOP_RUN);
    CU(cudaEventRecord(ctx->ev1, ctx->stream));
    CU(cudaEventSynchronize(ctx->ev1));
    cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1);
    *iters = S.iter;
    size_t avail = 0, total = 0;
    CU(cudaMemGetInfo(&avail, &total));
    if (ctx->cgm_r_bytes > avail / CGM_KEEP_PART) drop_window(ctx);
    // the fields that held FP32 residuals are FP64 fields again
    if (!hi && stride != 2 * ctx->g.Vh)
      for (int i = 1; i <= 4; i++) CU(cudaMemsetAsync(ctx->lx64[i].d, 0, ctx->lx64[i].bytes, ctx->stream));
    if (S.stop == STOP_BREAKDOWN) return fail(ctx, TMS_ERR_NAN, "nanned (cgm iteration %d)", S.iter);
    if (S.stop == STOP_MAXITER) return fail(ctx, TMS_ERR_NOT_CONVERGED, "exit without converging");
    return TMS_OK;
  }

  // x (FP64 full field) = solution of shift k of the last CGM
  template <int P>
  void cgm_solution(tms_ctx* ctx, int k, const Field& x)
  {
    const int stride = 2 * ctx->g.stride;
    Field f;
    f.prec = P;
    f.d = (unsigned char*)ctx->cgm_x + per_site_bytes(P) * (size_t)stride * k;
    f.stride = stride;
    convert<PREC_F64, P>(ctx, f, x, 1.0, stride);
  }
}

namespace
{
  // the reference's chiral gamma5 on lx AoS spinors (spins 2, 3 negated), in place
  __global__ void aos_g5_kernel(int64_t nsites, double* __restrict__ a)
  {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nsites * 12) return;
    const int64_t site = i / 12, k = i % 12;
    a[site * 24 + 12 + k] = -a[site * 24 + 12 + k];
  }

  // y += x over n doubles
  __global__ void aos_axpy_kernel(int64_t n, const double* __restrict__ x, double* __restrict__ y)
  {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += x[i];
  }

  struct DevArrays
  {
    std::vector<double*> p;
    ~DevArrays()
    {
      for (double* q : p)
        if (q) cudaFree(q);
    }
  };

  // Mixed multi-shift: every shift's FP32 multi-shift solution brought to its
  // target by defect correction through the e/o solver, all shifts at once:
  // (Q_W^2 + m^2)^-1 = Q(-m)^-1 Q(+m)^-1 and Q(mu)^-1 = D(mu)^-1 g5, so one
  // round is e_k = D(-m_k)^-1 g5 D(+m_k)^-1 g5 r_k for all unconverged shifts
  // as two batched e/o solves (one right-hand side per shift, per-shift mu),
  // then x_k += e_k and the FP64 true residual r_k = b - (Q_W^2 + m_k^2) x_k.
  // Each e/o solve goes to a tenth of the shift's remaining squared factor.
  tms_status cgm_refine_batched(tms_ctx* ctx, double kappa, int has_anis, double anis, const double* masses, int nmass,
                                int niter, const double* residues, int precision, double b2, tms_status st0,
                                int iters, float ms, double* const* sols, tms_stats* stats)
  {
    Field* f = ctx->lx64;
    const int64_t V = ctx->g.V;
    const size_t bytes = (size_t)V * 24 * sizeof(double);
    DevArrays X, Rg, Y, E;
    for (DevArrays* a : {&X, &Rg, &Y, &E})
      {
        a->p.assign(nmass, nullptr);
        for (int k = 0; k < nmass; k++) CU(dev_alloc(ctx, &a->p[k], bytes));
      }
    const int saved_mode = ctx->ptr_mode;
    struct ModeGuard
    {
      tms_ctx* c;
      int m;
      ~ModeGuard() { c->ptr_mode = m; }
    } guard{ctx, saved_mode};
    ctx->ptr_mode = TMS_PTR_DEVICE;
    const int blk = 256;
    const unsigned g5grid = (unsigned)div_up(V * 12, (int64_t)blk), axgrid = (unsigned)div_up(V * 24, (int64_t)blk);
    std::vector<double> rt(nmass);
    std::vector<tms_stats> sk(nmass);
    // the multi-shift solutions, their true residues and g5 r
    for (int k = 0; k < nmass; k++)
      {
        cgm_solution<PREC_F32>(ctx, k, f[1]);
        TRY(set_params(ctx, kappa, masses[k], has_anis, anis));
        TRY(LxOp::true_residual(ctx, f[0], f[1], f[2], &rt[k]));
        fill_stats(&sk[k], st0, iters, 0, ctx->cgm_h->res[k], rt[k] / b2, ms);
        TRY(lx_out(ctx, f[1], X.p[k]));
        TRY(lx_out(ctx, f[2], Rg.p[k]));
        ++ctx->launches;
        aos_g5_kernel<<<g5grid, blk, 0, ctx->stream>>>(V, Rg.p[k]);
      }
    CU(cudaGetLastError());
    tms_status worst = TMS_OK;
    for (int round = 0; round < 4; round++)
      {
        std::vector<int> act;
        for (int k = 0; k < nmass; k++)
          if (rt[k] >= residues[k] * b2) act.push_back(k);
        if (act.empty()) break;
        const int na = (int)act.size();
        std::vector<double*> src(na), sol(na);
        std::vector<double> mu(na), rel(na);
        std::vector<tms_stats> es(na);
        for (int a = 0; a < na; a++)
          {
            const int k = act[a];
            rel[a] = std::min(1e-2, std::max(1e-22, 1e-1 * residues[k] * b2 / rt[k]));
          }
        for (int pass = 0; pass < 2; pass++)
          {
            for (int a = 0; a < na; a++)
              {
                const int k = act[a];
                src[a] = pass ? Y.p[k] : Rg.p[k];
                sol[a] = pass ? E.p[k] : Y.p[k];
                mu[a] = pass ? -masses[k] : masses[k];
              }
            const tms_status s = tms_cg_eoprec_batched(ctx, na, sol.data(), src.data(), kappa, has_anis, anis,
                                                       mu.data(), niter, rel.data(), precision, es.data());
            if (s != TMS_OK && s != TMS_ERR_NOT_CONVERGED) return s;
            if (s != TMS_OK) worst = s;
            for (int a = 0; a < na; a++)
              {
                sk[act[a]].iterations += es[a].iterations;
                sk[act[a]].seconds += es[a].seconds;
                ++ctx->launches;
                if (pass == 0) aos_g5_kernel<<<g5grid, blk, 0, ctx->stream>>>(V, Y.p[act[a]]);
                else aos_axpy_kernel<<<axgrid, blk, 0, ctx->stream>>>(V * 24, E.p[act[a]], X.p[act[a]]);
              }
            CU(cudaGetLastError());
          }
        for (int a = 0; a < na; a++)
          {
            const int k = act[a];
            TRY(lx_in(ctx, X.p[k], f[1]));
            TRY(set_params(ctx, kappa, masses[k], has_anis, anis));
            TRY(LxOp::true_residual(ctx, f[0], f[1], f[2], &rt[k]));
            TRY(lx_out(ctx, f[2], Rg.p[k]));
            ++ctx->launches;
            aos_g5_kernel<<<g5grid, blk, 0, ctx->stream>>>(V, Rg.p[k]);
            sk[k].reliable_updates++;
          }
        CU(cudaGetLastError());
      }
    ctx->ptr_mode = saved_mode;
    for (int k = 0; k < nmass; k++)
      {
        const tms_status sk_st = (rt[k] >= residues[k] * b2) ? TMS_ERR_NOT_CONVERGED : (worst == TMS_ERR_NOT_CONVERGED ? TMS_OK : worst);
        sk[k].true_rel_res2 = rt[k] / b2;
        sk[k].iterated_rel_res2 = rt[k] / b2;
        sk[k].status = sk_st;
        if (sk_st != TMS_OK) worst = TMS_ERR_NOT_CONVERGED;
        if (stats) stats[k] = sk[k];
        if (saved_mode == TMS_PTR_HOST)
          {
            CU(cudaMemcpyAsync(sols[k], X.p[k], bytes, cudaMemcpyDeviceToHost, ctx->stream));
            CU(cudaStreamSynchronize(ctx->stream));
          }
        else
          CU(cudaMemcpyAsync(sols[k], X.p[k], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
      }
    CU(cudaStreamSynchronize(ctx->stream));
    return worst;
  }
}

extern "C" {

tms_status tms_cg_tmQ2(tms_ctx* ctx, double* sol_lx, const double* guess_lx, const double* src_lx, double kappa,
                       int has_anis, double anis, double m, int niter, double residue, int precision,
                       tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (!sol_lx || !src_lx || niter <= 0 || !(residue > 0)) return fail(ctx, TMS_ERR_BAD_ARG, "bad solver arguments");
  TRY(set_params(ctx, kappa, m, has_anis, anis));
  Field* f = ctx->lx64;
  TRY(lx_in(ctx, src_lx, f[0]));
  if (guess_lx) TRY(lx_in(ctx, guess_lx, f[1]));
  const tms_status st = cg_dispatch<LxOp>(ctx, precision, niter, residue, guess_lx != nullptr, stats);
  if (st == TMS_OK || st == TMS_ERR_NOT_CONVERGED) TRY(lx_out(ctx, f[1], sol_lx));
  TRY(finish(ctx));
  return st;
}

tms_status tms_cgm_tmQ2(tms_ctx* ctx, double* const* sols, const double* src_lx, double kappa, int has_anis,
                        double anis, const double* masses, int nmass, int niter, const double* residues,
                        int precision, tms_stats* stats)
{
  TRY(check_conf(ctx));
  if (!sols || !src_lx || !masses || !residues || nmass <= 0 || nmass > CGM_MAX_SHIFTS || niter <= 0)
    return fail(ctx, TMS_ERR_BAD_ARG, "bad multi-shift arguments (1 <= nmass <= %d)", CGM_MAX_SHIFTS);
  if (precision != TMS_PREC_DOUBLE && precision != TMS_PREC_MIXED_SINGLE && precision != TMS_PREC_MIXED_HALF)
    return fail(ctx, TMS_ERR_BAD_ARG, "unknown precision %d", precision);
  for (int k = 0; k < nmass; k++)
    if (!sols[k] || !(residues[k] > 0) || !std::isfinite(masses[k]))
      return fail(ctx, TMS_ERR_BAD_ARG, "bad shift %d", k);
  TRY(set_params(ctx, kappa, 0.0, has_anis, anis, 1)); // the CGM operator Q(0)^2
  Field* f = ctx->lx64;
  const int stride = 2 * ctx->g.stride;
  for (int i = 1; i <= 6; i++) TRY(alloc_field(ctx, f[i], PREC_F64, stride));
  TRY(lx_in(ctx, src_lx, f[0]));
  double b2;
  TRY(norm2<PREC_F64>(ctx, f[0], &b2, stride));
  if (b2 == 0.0 || std::isnan(b2)) return fail(ctx, TMS_ERR_INVALID_SOURCE, "invalid norm: %g", b2);
  double sigma[CGM_MAX_SHIFTS], target[CGM_MAX_SHIFTS];
  // the FP32 multi-shift solve stops at the squared relative residue
  // cgm_floor_single at most; each shift is then brought to its target by the
  // mixed-precision CG from that guess
  const double floor32 = ctx->cgm_floor32;
  for (int k = 0; k < nmass; k++)
    {
      sigma[k] = masses[k] * masses[k];
      target[k] = (precision == TMS_PREC_DOUBLE) ? residues[k] : std::max(residues[k], floor32);
    }
  int iters = 0;
  float ms = 0;
  tms_status st;
  if (precision == TMS_PREC_DOUBLE)
    st = cgm_run<PREC_F64>(ctx, links64(ctx), nmass, sigma, target, niter, b2, &iters, &ms);
  else
    st = ctx->su3 ? cgm_run<PREC_F32>(ctx, links32r(ctx), nmass, sigma, target, niter, b2, &iters, &ms)
                  : cgm_run<PREC_F32>(ctx, links32f(ctx), nmass, sigma, target, niter, b2, &iters, &ms);
  if (st != TMS_OK && st != TMS_ERR_NOT_CONVERGED) return st;
  if (precision != TMS_PREC_DOUBLE && ctx->cgm_refine_batched)
    {
      // all shifts' corrections as batched e/o solves (tuning "cgm_refine_batched")
      tms_status worst = st;
      const tms_status s2 = cgm_refine_batched(ctx, kappa, has_anis, anis, masses, nmass, niter, residues, precision,
                                               b2, st, iters, ms, sols, stats);
      if (s2 != TMS_OK && s2 != TMS_ERR_NOT_CONVERGED) return s2;
      if (s2 != TMS_OK) worst = s2;
      TRY(finish(ctx));
      if (worst != TMS_OK) return fail(ctx, worst, "exit without converging");
      return TMS_OK;
    }
  tms_status worst = st;
  for (int k = 0; k < nmass; k++)
    {
      if (precision == TMS_PREC_DOUBLE) cgm_solution<PREC_F64>(ctx, k, f[1]);
      else cgm_solution<PREC_F32>(ctx, k, f[1]);
      // final true residue of the shift (cgm_invert_template_threaded.hpp:266-279)
      TRY(set_params(ctx, kappa, masses[k], has_anis, anis));
      double rt;
      TRY(LxOp::true_residual(ctx, f[0], f[1], f[2], &rt));
      tms_stats sk{};
      fill_stats(&sk, st, iters, 0, ctx->cgm_h->res[k], rt / b2, ms);
      if (precision != TMS_PREC_DOUBLE && rt >= residues[k] * b2)
        {
          // defect correction through the e/o solver, FP64 residuals in between:
          // (Q_W^2 + m^2)^-1 = Q(-m)^-1 Q(+m)^-1 and Q(mu)^-1 = D(mu)^-1 g5, so
          // e = D(-m)^-1 g5 D(+m)^-1 g5 r ; x += e ; r = b - (Q_W^2 + m^2) x
          Field* ex = ctx->ex;
          for (auto& e : ctx->ex) TRY(alloc_field(ctx, e, PREC_F64));
          const int n = (int)ctx->g.Vh;
          tms_status s2 = TMS_OK;
          int corrections = 0;
          while (rt >= residues[k] * b2 && corrections < 4)
            {
              // each e/o solve to a tenth of the remaining factor (squared residues):
              // one correction per shift at 32^3x64 with the true residual a third
              // of its target (a hundredth took 4 % longer; 0.3 needed a second one)
              const double rel = std::min(1e-2, std::max(1e-22, 1e-1 * residues[k] * b2 / rt));
              for (int p = 0; p < 2; p++)
                {
                  ++ctx->launches;
                  g5_copy_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
                    n, view_par<PREC_F64>(f[2], p), view<PREC_F64>(ex[p]));
                }
              for (int pass = 0; pass < 2; pass++)
                {
                  const double sg = pass ? -1.0 : +1.0;
                  TRY(set_params(ctx, kappa, sg * masses[k], has_anis, anis));
                  tms_stats es{};
                  s2 = eo_full_solve(ctx, niter, rel, precision, &es);
                  if (s2 != TMS_OK && s2 != TMS_ERR_NOT_CONVERGED) return s2;
                  sk.iterations += es.iterations;
                  sk.seconds += es.seconds;
                  for (int p = 0; p < 2; p++)
                    {
                      ++ctx->launches;
                      if (sg > 0)
                        g5_copy_kernel<<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0, ctx->stream>>>(
                          n, view<PREC_F64>(ex[2 + p]), view<PREC_F64>(ex[p]));
                      else
                        axpby_kernel<PREC_F64, PREC_F64, PREC_F64><<<div_up(n, BLAS_THREADS), BLAS_THREADS, 0,
                                                                     ctx->stream>>>(
                          n, 1.0, view_par<PREC_F64>(f[1], p), 1.0, view<PREC_F64>(ex[2 + p]),
                          view_par<PREC_F64>(f[1], p));
                    }
                }
              CU(cudaGetLastError());
              TRY(set_params(ctx, kappa, masses[k], has_anis, anis));
              TRY(LxOp::true_residual(ctx, f[0], f[1], f[2], &rt));
              corrections++;
            }
          if (s2 == TMS_OK && rt >= residues[k] * b2) s2 = TMS_ERR_NOT_CONVERGED;
          if (s2 != TMS_OK) worst = s2;
          sk.reliable_updates = corrections;
          sk.true_rel_res2 = rt / b2;
          sk.iterated_rel_res2 = rt / b2;
          sk.status = s2;
        }
      if (stats) stats[k] = sk;
      TRY(lx_out(ctx, f[1], sols[k]));
    }
  TRY(finish(ctx));
  if (worst != TMS_OK) return fail(ctx, worst, "exit without converging");
  return TMS_OK;
}

} // extern "C"
