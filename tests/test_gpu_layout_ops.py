"""The operators on the caller's layout (one launch per hop) against the
oracle: lattices on both sides of the size up to which a site's directions are
spread over a block's warps, with ragged last warps and blocks, and every form
of caller buffer (host, device, device off a 16-byte boundary, output over the
input, output overlapping it)."""
import numpy as np
import pytest

import oracle
from nissa_b200 import Lattice
from nissa_b200 import workload as wl
from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-14


def _place(x, form):
    """(input, output) of the form: device tensors, or numpy arrays for host."""
    import torch
    n = x.size
    if form == "host":
        return x, np.empty_like(x)
    pool = torch.zeros(2 * n + 8, dtype=torch.float64, device="cuda")
    i0, o0 = {"device": (0, n), "off8": (1, n + 3), "in_place": (0, 0), "overlap": (0, 48)}[form]
    i = pool[i0:i0 + n].view(x.shape)
    i.copy_(torch.from_numpy(x))
    return i, pool[o0:o0 + n].view(x.shape)


@pytest.mark.parametrize("form", ["host", "device", "off8", "in_place", "overlap"])
@pytest.mark.parametrize("T,L", [(2, 4), (4, 6), (10, 10), (20, 10)])
def test_operators_on_the_callers_layout(cuda_device, T, L, form):
    # V and Vh of 128, 64; 864, 432; 10000 (whole-lattice: a warp per 32 sites), 5000 (e/o: split); 20000, 10000
    k, mu, anis, csw = 0.14, 0.02, 1.15, 1.3
    conf = wl.gauge_conf(T, L, 0.35, seed=T + L)
    cbc = wl.apply_time_bc(conf, T, L, -1.0)
    geo = oracle.Geom(T, L)
    ceo = geo.split(cbc)
    x, xl = wl.random_spinor(geo.Vh, 71), wl.random_spinor(geo.V, 72)
    Cl = geo.clover_term(cbc, csw)
    inv = geo.inv_clover_term(Cl, k, mu)
    Clo = geo.split(Cl.reshape(geo.V, -1)).reshape(2, geo.Vh, 4, 3, 3, 2)[1]
    inve = geo.split(inv.reshape(geo.V, -1)).reshape(2, geo.Vh, 2, 6, 6, 2)[0]
    with Lattice(T, L) as lat:
        lat.upload_conf(conf)
        lat.clover_term(csw)

        def check(op, v, want):
            i, o = _place(v, form)
            got = op(i, o)
            assert rel(got if form == "host" else got.cpu().numpy(), want) < TOL

        for par in (0, 1):
            check(lambda i, o: lat.tmn2Deo_or_tmn2Doe_eos(par, i, anis=anis, out=o), x, geo.hop(ceo, par, x, anis=anis))
        check(lambda i, o: lat.tmDee_or_oo_eos(k, mu, i, out=o), x, geo.tmDee(k, mu, x))
        check(lambda i, o: lat.inv_tmDee_or_oo_eos(k, mu, i, out=o), x, geo.inv_tmDee(k, mu, x))
        check(lambda i, o: lat.tmDkern_eoprec_eos(k, -mu, i, out=o), x, geo.kern(ceo, k, -mu, x))
        check(lambda i, o: lat.tmDkern_eoprec_square_eos(k, mu, i, anis=anis, out=o), x,
              geo.kern2(ceo, k, mu, x, anis=anis))
        check(lambda i, o: lat.apply_tmQ(k, mu, i, anis=anis, out=o), xl, geo.tmQ(cbc, k, mu, xl, anis=anis))
        check(lambda i, o: lat.apply_tmQ2(k, mu, i, out=o), xl, geo.tmQ2(cbc, k, mu, xl))
        for dag in (0, 1):
            check(lambda i, o: lat.tmclovDkern_eoprec_eos(k, mu, dag, i, out=o), x,
                  geo.tmclov_kern(ceo, k, Clo, inve, dag, mu, x))
        check(lambda i, o: lat.tmclovDkern_eoprec_square_eos(k, mu, i, anis=anis, out=o), x,
              geo.tmclov_kern2(ceo, k, Clo, inve, mu, x, anis=anis))
        check(lambda i, o: lat.apply_tmclovQ(k, mu, i, out=o), xl, geo.tmclovQ(cbc, k, Cl, mu, xl))


def test_the_callers_layout_gives_the_bits_of_the_planes(cuda_device):
    """The same operators from hops on planes (small_lattice 0): the components' forms of the epilogues round as the
    sites' forms do, FMA for FMA.  (Q alone has no form on planes; Q^2 is made of it.)  The clover terms' sums of 6 to 12 products are
    contracted differently: rounding, 1e-15."""
    T, L = 10, 8
    x, xl = wl.random_spinor(T * L ** 3 // 2, 73), wl.random_spinor(T * L ** 3, 74)
    with Lattice(T, L) as lat:
        lat.upload_conf(wl.gauge_conf(T, L, 0.35, seed=5))
        lat.clover_term(1.3)
        got = []
        for small in (1, 0):
            lat.set_tuning("small_lattice", small)
            got.append([lat.tmDkern_eoprec_eos(0.14, 0.021, x, anis=1.15),
                        lat.tmDkern_eoprec_square_eos(0.16, -0.5, x),
                        lat.apply_tmQ2(0.14, 0.021, xl, anis=1.15), lat.apply_tmQ2(0.16, -0.5, xl),
                        lat.tmclovDkern_eoprec_square_eos(0.13, 0.02, x, anis=1.15), lat.apply_tmclovQ(0.13, 0.02, xl)])
        for k, (a, b) in enumerate(zip(*got)):
            assert np.array_equal(a, b) if k < 4 else rel(a, b) < 1e-15, k
