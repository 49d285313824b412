// Direction-parallel hops for lattices too small to fill the GPU with one
// thread per site: a block takes 32 sites, its warp d computes direction d
// of all of them (one neighbour and one link per thread, so the eight gathers
// of a site are in flight at once), the products meet in shared memory and
// warp 0 adds them in the order of hop_site and runs the epilogue.
//
// Bound by latency, not by bytes.  With one thread per site a launch on a small
// lattice is eight dependent rounds of loads and products deep, here it is
// one.  The direction is a run-time value: eight unrolled directions are 40 KB
// of code, and fetching it was the leading stall (8.1 of 9.6 warps per issue
// waited for instructions with a code path per direction).  The links, which
// nothing in a stream of solver kernels writes, are loaded before the wait for
// the preceding kernel.
#pragma once

#include <type_traits>

#include "tms_kernels.cuh"
#include "tms_pipe.cuh"

namespace tms
{
  constexpr int HOP_DP_SITES = 32;
  constexpr int HOP_DP_THREADS = 8 * HOP_DP_SITES;

  // epilogues with a clover term
  template <class E, class = void>
  struct HasClover : std::false_type
  {
  };
  template <class E>
  struct HasClover<E, decltype((void)E::cl)> : std::true_type
  {
  };

  // direction d = 2 mu (forward), 2 mu + 1 (backward): lx index of the neighbour
  __device__ __forceinline__ int dp_neighbour(const Lattice& g, const Site& s, int d)
  {
    const int mu = d >> 1;
    const int c = mu == 0 ? s.t : mu == 1 ? s.x : mu == 2 ? s.y : s.z;
    const int n = mu == 0 ? g.T : mu == 1 ? g.LX : mu == 2 ? g.LY : g.LZ;
    const int st = mu == 0 ? g.LX * g.LY * g.LZ : mu == 1 ? g.LY * g.LZ : mu == 2 ? g.LZ : 1;
    if (d & 1) return c == 0 ? s.lx + (n - 1) * st : s.lx - st;
    return c == n - 1 ? s.lx - (n - 1) * st : s.lx + st;
  }

  // whether the projection of a direction pairs spin 0 with 3 (x, y) or with 2 (t, z)
  __device__ __forceinline__ bool dp_cross(int d) { return ((d >> 1) ^ (d >> 2)) & 1; }

  // the products U h (forward) or U^+ h (backward) of the two rows of the
  // projected neighbour, times f: `project` and `link_mul` with the direction a
  // run-time value.  a, b: the spins paired with spins 0, 1.
  template <typename R>
  __device__ __forceinline__ void dp_products(int d, const C<R> s0[3], const C<R> s1[3], const C<R> a[3],
                                              const C<R> b[3], const C<R> L[9], R f, C<R> u0[3], C<R> u1[3])
  {
    const bool bwd = d & 1, imag = (d >> 1) & 1;     // phases +-1 (t, y) or +-i (x, z)
    const R p0 = bwd ? R(-1) : R(1), p1 = (d >= 4) ? -p0 : p0;
    const R q0 = imag ? -p0 : p0, q1 = imag ? -p1 : p1; // on the real parts
    C<R> h0[3], h1[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
      {
        h0[c] = {s0[c].re + q0 * (imag ? a[c].im : a[c].re), s0[c].im + p0 * (imag ? a[c].re : a[c].im)};
        h1[c] = {s1[c].re + q1 * (imag ? b[c].im : b[c].re), s1[c].im + p1 * (imag ? b[c].re : b[c].im)};
      }
    // (a branch for the two forms: with the link transposed and conjugated into one
    // form, products contract to FMAs differently than in the other hops)
    if (bwd)
      {
        link_mul<false>(L, h0, u0, f);
        link_mul<false>(L, h1, u1, f);
      }
    else
      {
        link_mul<true>(L, h0, u0, f);
        link_mul<true>(L, h1, u1, f);
      }
  }

  // The reconstruction of one component (FP64): spin `spin` of direction d's
  // products is row dp_row of them times a phase +-1 or +-i and the hop factor f,
  // added by FMAs as the compiler contracts `reconstruct` to, so that the results
  // are the same bits.
  __device__ __forceinline__ int dp_row(int d, int spin) { return spin < 2 ? spin : dp_cross(d) ? 3 - spin : spin - 2; }
  __device__ __forceinline__ void dp_accumulate(int d, int spin, C<double> u, double f, C<double>& acc)
  {
    const int mu = d >> 1;
    // the lower spins' phase: t sg, x -i sg, y -sg (spin 2) or sg (spin 3), z -i sg (spin 2) or i sg (spin 3)
    const bool lower = spin >= 2, imag = lower && (mu & 1);
    const bool minus = lower && ((bool)(d & 1) != (mu == 1 || (mu >= 2 && spin == 2)));
    const double k = minus ? -f : f;
    acc.re = fma_rn(imag ? u.im : u.re, imag ? -k : k, acc.re);
    acc.im = fma_rn(imag ? u.re : u.im, k, acc.im);
  }

  // colour col (and the next, if two) of spin `spin` of the hop of a site, from the
  // products get(direction, product)
  template <class Get>
  __device__ __forceinline__ void dp_gather(const Get& get, const Lattice& g, const Site& s, double anis, int spin, int col,
                                            bool two, C<double> acc[2])
  {
    acc[0] = acc[1] = {0.0, 0.0};
#pragma unroll
    for (int d = 0; d < 8; d++)
      {
        const double f = d == 0 ? ((s.t == g.T - 1) ? g.bc_t : 1.0) : d == 1 ? ((s.t == 0) ? g.bc_t : 1.0) : anis;
        const int k = 3 * dp_row(d, spin) + col;
        dp_accumulate(d, spin, get(d, k), f, acc[0]);
        if (two) dp_accumulate(d, spin, get(d, k + 1), f, acc[1]);
      }
  }

  template <typename R>
  struct DpShare
  {
    C<R> u[8][6][HOP_DP_SITES]; // direction, product (row 0 colours, row 1 colours), site
  };

  // adds direction D's products times the hop factor f
  template <int D, typename R>
  __device__ __forceinline__ void dp_add(const DpShare<R>& sh, int lane, R f, C<R> acc[12])
  {
    C<R> u0[3], u1[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
      {
        u0[c] = cscale(sh.u[D][c][lane], f);
        u1[c] = cscale(sh.u[D][3 + c][lane], f);
      }
    reconstruct<D / 2, !(D & 1)>(acc, u0, u1);
  }

  // direction d of a site (parity p, neighbour n): its products into the share
  template <int P, int LF>
  __device__ __forceinline__ void dp_direction(DpShare<typename SpinorT<P>::R>& sh, int d, int lane, int n, const SpinorT<P>& in,
                                               const C<typename SpinorT<P>::R> L[9], typename SpinorT<P>::R ls)
  {
    using R = typename SpinorT<P>::R;
    R ss;
    C<R> v[12], a[3], b[3], u0[3], u1[3];
    in.load_raw(n, v, ss);
    const bool cross = dp_cross(d);
#pragma unroll
    for (int c = 0; c < 3; c++)
      {
        a[c] = {cross ? v[9 + c].re : v[6 + c].re, cross ? v[9 + c].im : v[6 + c].im};
        b[c] = {cross ? v[6 + c].re : v[9 + c].re, cross ? v[6 + c].im : v[9 + c].im};
      }
    dp_products<R>(d, v, v + 3, a, b, L, ss * ls, u0, u1);
#pragma unroll
    for (int c = 0; c < 3; c++)
      {
        sh.u[d][c][lane] = u0[c];
        sh.u[d][3 + c][lane] = u1[c];
      }
  }

  template <typename R>
  __device__ __forceinline__ void dp_sum(const DpShare<R>& sh, const Lattice& g, const Site& s, int lane, R anis,
                                         C<R> acc[12])
  {
#pragma unroll
    for (int c = 0; c < 12; c++) acc[c] = {R(0), R(0)};
    dp_add<0>(sh, lane, (s.t == g.T - 1) ? R(g.bc_t) : R(1), acc);
    dp_add<1>(sh, lane, (s.t == 0) ? R(g.bc_t) : R(1), acc);
    dp_add<2>(sh, lane, anis, acc);
    dp_add<3>(sh, lane, anis, acc);
    dp_add<4>(sh, lane, anis, acc);
    dp_add<5>(sh, lane, anis, acc);
    dp_add<6>(sh, lane, anis, acc);
    dp_add<7>(sh, lane, anis, acc);
  }

  template <int P, int LF, class Epi, class Fin>
  __global__ void __launch_bounds__(HOP_DP_THREADS, 2)
    hop_dp_kernel(Lattice g, int par_out, int npar, SpinorT<P> in_e, SpinorT<P> in_o, LinkT<LF> U, const OpParams* prm,
                  Epi epi, Reducer red, Fin fin, const int* __restrict__ stop)
  {
    using R = typename SpinorT<P>::R;
    __shared__ DpShare<R> sh;
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    const int chunk = (npar == 2) ? blockIdx.x >> 1 : blockIdx.x;
    const int p = (npar == 2) ? blockIdx.x & 1 : par_out;
    const bool active = chunk * HOP_DP_SITES + lane < g.Vh;
    const int ieo = active ? chunk * HOP_DP_SITES + lane : (int)g.Vh - 1;
    const Site s = eo_site(g, p, ieo);
    const int n = dp_neighbour(g, s, d) >> 1;
    C<R> L[9];
    R ls;
    U.template load_scaled<false>((d & 1) ? 1 - p : p, d >> 1, (d & 1) ? n : ieo, L, ls);
    pdl_enter();
    if (stop && *stop) return; // the same for the whole grid: this kernel writes it after its last block's hop
    dp_direction<P, LF>(sh, d, lane, n, p ? in_e : in_o, L, ls);
    __syncthreads();
    double part = 0.0;
    if (d == 0 && active)
      {
        C<R> acc[12];
        dp_sum(sh, g, s, lane, R(prm->anis), acc);
        part = epi(p, ieo, acc);
      }
    if (Epi::kReduce) grid_reduce<HOP_DP_THREADS>(part, red, fin);
  }
}
