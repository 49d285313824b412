"""The operators on the caller's layout (one launch per hop) and on planes against
the oracle: lattices on both sides of the size rules that choose between them,
with ragged last warps and blocks, and every form of caller buffer (host, device,
device off a 16-byte boundary, output over the input, output overlapping it)."""
import functools

import numpy as np
import pytest

import oracle
from nissa_b200 import Lattice
from nissa_b200 import workload as wl
from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-14
K, MU, ANIS, CSW = 0.14, 0.02, 1.15, 1.3


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


@functools.lru_cache(maxsize=1)
def _oracle(T, L):
    """conf, inputs and the oracle's outputs of every operator"""
    conf = wl.gauge_conf(T, L, 0.35, seed=T + L)
    cbc = wl.apply_time_bc(conf, T, L, -1.0)
    geo = oracle.Geom(T, L)
    ceo = geo.split(cbc)
    x, xl = wl.random_spinor(geo.Vh, 71), wl.random_spinor(geo.V, 72)
    Cl = geo.clover_term(cbc, CSW)
    inv = geo.inv_clover_term(Cl, K, MU)
    Clo = geo.split(Cl.reshape(geo.V, -1)).reshape(2, geo.Vh, 4, 3, 3, 2)[1]
    inve = geo.split(inv.reshape(geo.V, -1)).reshape(2, geo.Vh, 2, 6, 6, 2)[0]
    want = [geo.hop(ceo, 0, x, anis=ANIS), geo.hop(ceo, 1, x, anis=ANIS), geo.tmDee(K, MU, x), geo.inv_tmDee(K, MU, x),
            geo.kern(ceo, K, -MU, x), geo.kern2(ceo, K, MU, x, anis=ANIS), geo.tmQ(cbc, K, MU, xl, anis=ANIS),
            geo.tmQ2(cbc, K, MU, xl), geo.tmclov_kern(ceo, K, Clo, inve, 0, MU, x),
            geo.tmclov_kern(ceo, K, Clo, inve, 1, MU, x), geo.tmclov_kern2(ceo, K, Clo, inve, MU, x, anis=ANIS),
            geo.tmclovQ(cbc, K, Cl, MU, xl)]
    return conf, x, xl, want


# the largest is above every size rule, so its operators of several hops work on planes, as small_lattice 0 makes
# them do at every size; the others are below, with ragged last blocks (432, 5000, 864 sites) among them
@pytest.mark.parametrize("T,L,small,form", [(T, L, s, f) for T, L, s in
                                            [(2, 4, 1), (4, 6, 1), (4, 6, 0), (10, 10, 1), (10, 10, 0), (20, 10, 1),
                                             (32, 16, 1)]
                                            for f in ("host", "device", "off8", "in_place", "overlap")])
def test_operators_on_the_callers_layout(cuda_device, T, L, small, form):
    conf, x, xl, want = _oracle(T, L)
    with Lattice(T, L) as lat:
        lat.upload_conf(conf)
        lat.clover_term(CSW)
        lat.set_tuning("small_lattice", small)
        ops = [lambda i, o: lat.tmn2Deo_or_tmn2Doe_eos(0, i, anis=ANIS, out=o),
               lambda i, o: lat.tmn2Deo_or_tmn2Doe_eos(1, i, anis=ANIS, out=o),
               lambda i, o: lat.tmDee_or_oo_eos(K, MU, i, out=o),
               lambda i, o: lat.inv_tmDee_or_oo_eos(K, MU, i, out=o),
               lambda i, o: lat.tmDkern_eoprec_eos(K, -MU, i, out=o),
               lambda i, o: lat.tmDkern_eoprec_square_eos(K, MU, i, anis=ANIS, out=o),
               lambda i, o: lat.apply_tmQ(K, MU, i, anis=ANIS, out=o),
               lambda i, o: lat.apply_tmQ2(K, MU, i, out=o),
               lambda i, o: lat.tmclovDkern_eoprec_eos(K, MU, 0, i, out=o),
               lambda i, o: lat.tmclovDkern_eoprec_eos(K, MU, 1, i, out=o),
               lambda i, o: lat.tmclovDkern_eoprec_square_eos(K, MU, i, anis=ANIS, out=o),
               lambda i, o: lat.apply_tmclovQ(K, MU, i, out=o)]
        for n, (op, w) in enumerate(zip(ops, want)):
            i, o = _place(x if w.size == x.size else xl, form)
            got = op(i, o)
            assert rel(got if form == "host" else got.cpu().numpy(), w) < TOL, n


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


def test_planes_operators_stage_one_buffer(cuda_device):
    """K^2 on planes between host arrays, 65536 sites a parity: four work fields and one staging buffer, which holds
    the input and then the output."""
    import torch
    T, L = 32, 16
    unit = T * L ** 3 // 2 * 192
    x = wl.random_spinor(T * L ** 3 // 2, 75)
    with Lattice(T, L) as lat:
        # from the device: the staging buffer of a host conf would hide the operator's
        lat.upload_conf(torch.from_numpy(wl.gauge_conf(T, L, 0.35, seed=6, device="cuda")).to("cuda:0"))
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        lat.tmDkern_eoprec_square_eos(0.16, 0.01, x)
        used = free0 - torch.cuda.mem_get_info()[0]
    assert used <= 5 * unit + (6 << 20), used / unit
