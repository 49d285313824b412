// The FP64 hop between fields in the caller's own layout (sites of 24
// consecutive doubles), for the operators of the C ABI: one launch per hop
// straight on the caller's arrays, instead of converting to planes and back
// around a hop on planes.
//
// The directions of a site are spread over the eight warps of a block
// (tms_hop_dp.cuh), which suits small lattices and costs large ones little.
// A warp copies the 32 neighbour records of its direction together (12
// cp.async of 16 bytes per lane, consecutive lanes along a record) into shared
// memory and each lane reads its own record back at a pitch of 208 bytes, free
// of bank conflicts; the output leaves as whole lines.
// Whole calls, before (conversions around a hop on planes) / after: 8^3x16 hop
// 46 / 20.8 us, 32^3x64 563 / 425 us; 24^3x48 Q 453 / 281 us.  (One warp for the
// eight directions of 32 sites, three directions ahead, took 404 us a launch at
// 32^3x64 too, with eight warps per SM: the copies' address exchange and the
// reads back queue on the shared-memory pipe.  Three blocks per SM instead of
// two took 474 us, their shared memory being L1's.)
#pragma once

#include <type_traits>

#include "tms_hop_dp.cuh"
#include "tms_kernels.cuh"
#include "tms_pipe.cuh"

namespace tms
{
  constexpr int AOS_PITCH = 208;                // bytes of a staged record
  constexpr int AOS_SLOT = 32 * AOS_PITCH;      // a warp's records
  constexpr int AOS_DP_SMEM = 10 * AOS_SLOT;    // warp 0's operand and output, then a slot per direction

  // The epilogues' view of a field in the caller's layout (A64): the operand
  // they read is staged before they run, and what they write leaves afterwards.
  __device__ __forceinline__ double2* aos_record(int slot)
  {
    extern __shared__ __align__(16) char aos_smem[];
    return reinterpret_cast<double2*>(aos_smem + slot * AOS_SLOT + (threadIdx.x & 31) * AOS_PITCH);
  }
  template <> struct SpinorT<PREC_A64>
  {
    using R = double;
    double2* d;
    float* n; // unused
    int stride;
    __device__ __forceinline__ C<double> load1(int, int c) const
    {
      const double2 w = aos_record(0)[c];
      return {w.x, w.y};
    }
    __device__ __forceinline__ void store1(int, int c, C<double> v) const { aos_record(1)[c] = make_double2(v.re, v.im); }
  };

  // which word of which record a lane copies: word j of the warp's 384 for lane
  // l is q = 32 j + l, and three steps of j move on by eight records
  struct AosLane
  {
    int r[3], c[3];
    __device__ __forceinline__ AosLane()
    {
#pragma unroll
      for (int j = 0; j < 3; j++)
        {
          const int q = 32 * j + (int)(threadIdx.x & 31);
          r[j] = q / 12;
          c[j] = q % 12;
        }
    }
  };

  // the records `row` of the warp's lanes into a slot (cp.async, not committed)
  __device__ __forceinline__ void aos_fetch(const AosLane& a, char* slot, const double2* src, int row)
  {
#pragma unroll
    for (int j = 0; j < 12; j++)
      {
        const int r = a.r[j % 3] + 8 * (j / 3), c = a.c[j % 3];
        const size_t from = (size_t)__shfl_sync(0xffffffffu, row, r) * 12 + c;
        cp_async16(slot + r * AOS_PITCH + c * 16, src + from);
      }
  }

  // epilogues with an operand x, and with operator parameters
  template <class E, class = void>
  struct AosOperand
  {
    static constexpr bool has = false;
    __device__ static const double2* get(const E&, int) { return nullptr; }
  };
  template <class E>
  struct AosOperand<E, decltype((void)E::x)>
  {
    static constexpr bool has = true;
    __device__ static const double2* get(const E& e, int p) { return pick(e.x[0], e.x[1], p).d; }
  };
  template <class E>
  __device__ __forceinline__ auto aos_set_params(E& e, const OpParams* prm, int) -> decltype((void)(e.prm = prm))
  {
    e.prm = prm;
  }
  template <class E>
  __device__ __forceinline__ void aos_set_params(E&, const OpParams*, long)
  {
  }

  // FULL: both parities, in lx order; otherwise the e/o order of parity par_out
  template <class Epi, bool FULL>
  __global__ void __launch_bounds__(HOP_DP_THREADS, 2)
    hop_aos_dp_kernel(Lattice g, int par_out, const double2* __restrict__ in, LinkT<LINK_F64_18> U,
                      const __grid_constant__ OpParams prm, Epi epi)
  {
    extern __shared__ __align__(16) char aos_smem[];
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    const int nsite = (int)(FULL ? g.V : g.Vh);
    const int first = blockIdx.x * HOP_DP_SITES;
    const int idx = min(first + lane, nsite - 1);
    const int ieo = FULL ? idx >> 1 : idx;
    const int p = FULL ? lx_parity(g, (unsigned)idx) : par_out;
    const Site s = eo_site(g, p, ieo);
    const int n = dp_neighbour(g, s, d);
    C<double> L[9];
    U.load<false>((d & 1) ? 1 - p : p, d >> 1, (d & 1) ? n >> 1 : ieo, L);
    const AosLane al;
    char* slot = aos_smem + (2 + d) * AOS_SLOT;
    pdl_enter();
    aos_set_params(epi, &prm, 0);
    aos_fetch(al, slot, in, FULL ? n : n >> 1);
    if (AosOperand<Epi>::has && d == 0) aos_fetch(al, aos_smem, AosOperand<Epi>::get(epi, p), idx);
    cp_async_commit();
    C<double> z = {};
    if constexpr (!HasClover<Epi>::value) z = epi.pre();
    cp_async_wait<0>();
    __syncwarp();
    {
      // the products replace the lane's own record
      double2* rec = aos_record(2 + d);
      const int ka = dp_cross(d) ? 9 : 6;
      C<double> v[6], a[3], b[3], u0[3], u1[3];
#pragma unroll
      for (int c = 0; c < 6; c++) v[c] = {rec[c].x, rec[c].y};
#pragma unroll
      for (int c = 0; c < 3; c++)
        {
          a[c] = {rec[ka + c].x, rec[ka + c].y};
          b[c] = {rec[15 - ka + c].x, rec[15 - ka + c].y};
        }
      dp_products<double>(d, v, v + 3, a, b, L, 1.0, u0, u1);
#pragma unroll
      for (int c = 0; c < 3; c++)
        {
          rec[c] = make_double2(u0[c].re, u0[c].im);
          rec[3 + c] = make_double2(u1[c].re, u1[c].im);
        }
    }
    __syncthreads();
    {
      const int spin = d >> 1, col = (d & 1) ? 2 : 0;
      C<double> acc[2];
      dp_gather(
        [&](int dir, int k) {
          const double2 w = aos_record(2 + dir)[k];
          return C<double>{w.x, w.y};
        },
        g, s, prm.anis, spin, col, !(d & 1), acc);
      if constexpr (HasClover<Epi>::value)
        {
          // the clover terms mix the components of a chirality: they meet in slot 1
          aos_record(1)[3 * spin + col] = make_double2(acc[0].re, acc[0].im);
          if (!(d & 1)) aos_record(1)[3 * spin + 1] = make_double2(acc[1].re, acc[1].im);
          __syncthreads();
          acc[0] = epi.comp(p, ieo, 3 * spin + col, aos_record(1), aos_record(0));
          if (!(d & 1)) acc[1] = epi.comp(p, ieo, 3 * spin + 1, aos_record(1), aos_record(0));
          __syncthreads();
          aos_record(1)[3 * spin + col] = make_double2(acc[0].re, acc[0].im);
          if (!(d & 1)) aos_record(1)[3 * spin + 1] = make_double2(acc[1].re, acc[1].im);
        }
      else
        {
          epi.comp(p, ieo, 3 * spin + col, acc[0], z);
          if (!(d & 1)) epi.comp(p, ieo, 3 * spin + 1, acc[1], z);
        }
    }
    __syncthreads();
    // the block's records leave as whole lines, 48 words a warp
    double2* out = pick(epi.out[0], epi.out[1], 0).d;
#pragma unroll
    for (int j = 0; j < 2; j++)
      {
        const int q = j * HOP_DP_THREADS + threadIdx.x, r = q / 12;
        if (q < 32 * 12 && first + r < nsite)
          out[(size_t)first * 12 + q] = *reinterpret_cast<const double2*>(aos_smem + AOS_SLOT + r * AOS_PITCH + (q % 12) * 16);
      }
  }
}
