"""Multi-shift CGM on the tm Q^2 operator and the full-lattice CG of Q(+m)Q(-m)
through the C ABI, against the reference's fixture (FP64) and the oracle."""
import numpy as np
import pytest

import oracle
from nissa_b200 import Lattice, TmError
from nissa_b200 import workload as wl
from conftest import rel

pytestmark = pytest.mark.gpu


def test_cgm_double_matches_reference_fixture(cuda_device, golden_small):
    g = golden_small
    T, L = int(g["T"]), int(g["L"])
    with Lattice(T, L) as lat:
        lat.upload_conf(g["conf"])
        sols, st = lat.inv_tmQ2_cgm(float(g["kappa"]), g["masses"], g["in_lx"], 10000, g["residues"])
        for k in range(len(g["masses"])):
            assert abs(st[k]["iterations"] - int(g["cgm_iters"])) <= 1
            assert rel(sols[k], g["cgm"][k]) < 1e-9, k
            assert st[k]["true_rel_res2"] < 2e-20


@pytest.mark.parametrize("precision,batched", [("single", 0), ("half", 0), ("half", 1)])
def test_cgm_mixed_reaches_every_target(cuda_device, precision, batched):
    """Both forms of the mixed solver's per-shift correction (shift after shift,
    or all shifts as batched e/o solves) reach every target."""
    T, L = 16, 8
    kappa = 0.1632
    masses = np.array([0.005, 0.02, 0.08, 0.2])
    conf = wl.gauge_conf(T, L, 0.35, seed=41)
    src = wl.z2_source(T, L, 5, col=1)
    geo = oracle.Geom(T, L)
    ref, _, _ = geo.cgm(wl.apply_time_bc(conf, T, L), kappa, masses, np.full(4, 1e-24), src, 100000)
    with Lattice(T, L) as lat:
        lat.upload_conf(conf)
        lat.set_tuning("cgm_refine_batched", batched)
        sols, st = lat.inv_tmQ2_cgm(kappa, masses, src, 100000, 1e-20, precision=precision)
        for k in range(len(masses)):
            assert st[k]["true_rel_res2"] < 1e-20, (k, st[k])
            assert rel(sols[k], ref[k]) < 1e-8, k


def test_cg_tmQ2_matches_single_shift(cuda_device):
    T, L = 8, 4
    kappa, m = 0.16, 0.03
    conf = wl.gauge_conf(T, L, 0.4, seed=43)
    src = wl.random_spinor(T * L ** 3, 44)
    geo = oracle.Geom(T, L)
    ref, _, _ = geo.cgm(wl.apply_time_bc(conf, T, L), kappa, [m], [1e-26], src, 100000)
    with Lattice(T, L) as lat:
        lat.upload_conf(conf)
        for prec in ("double", "single", "half"):
            sol, st = lat.inv_tmQ2_cg(kappa, m, src, 100000, 1e-22, precision=prec)
            assert st["true_rel_res2"] < 1e-22, prec
            assert rel(sol, ref[0]) < 1e-9, prec
        # the operator check: Q(+m)Q(-m) sol = src
        back = lat.apply_tmQ2(kappa, m, sol)
        assert rel(back, src) < 1e-10


def test_cgm_argument_errors(cuda_device):
    with Lattice(4, 4) as lat:
        lat.upload_conf(wl.gauge_conf(4, 4, 0.4, 1))
        src = wl.random_spinor(lat.V, 1)
        with pytest.raises(TmError) as e:
            lat.inv_tmQ2_cgm(0.16, np.linspace(0.01, 0.3, 33), src, 100, 1e-20)
        assert e.value.status == 3
        with pytest.raises(TmError) as e:
            lat.inv_tmQ2_cgm(0.16, [0.1], np.zeros_like(src), 100, 1e-20)
        assert e.value.status == 8
        with pytest.raises(TmError) as e:
            lat.inv_tmQ2_cgm(0.16, [0.01, 0.1], src, 3, 1e-24)
        assert e.value.status == 1


@pytest.mark.parametrize("graph_iters", [2, 5, 6, 7, 8, 24])
@pytest.mark.parametrize("precision,niter", [("double", 100000), ("double", 13), ("single", 100000)])
def test_cgm_window_lengths(cuda_device, graph_iters, precision, niter):
    """Shift updates applied by windows of 2 to 8 iterations, with shifts that stop inside a window and with a
    solve cut inside one (13 iterations), against one iteration at a time (windows of 1, replays of 11)."""
    T, L = 6, 4
    masses = [0.01, 0.05, 0.3]
    res = [1e-20, 1e-18, 1e-14]
    src = wl.random_spinor(T * L ** 3, 45)
    with Lattice(T, L) as lat:
        lat.upload_conf(wl.gauge_conf(T, L, 0.35, seed=46))
        got = []
        for n in (11, graph_iters):
            lat.set_tuning("graph_iters", n)
            got.append(lat.inv_tmQ2_cgm(0.16, masses, src, niter, res, precision=precision, raise_on_error=False))
        for k in range(3):
            assert got[0][1][k]["iterations"] == got[1][1][k]["iterations"]
            # FP64: the same operations per site in the same order, up to their contraction into FMAs.  FP32: two
            # solutions within their residues, |dx| <= 2 |A^-1| |r|, so 2 sqrt(res) cond(A) of |x|; here
            # A = Q_W^2 + m^2 has eigenvalues between m^2 and (1/2k + 4)^2, and a tenth of that bound is asked for
            cond = (0.5 / 0.16 + 4) ** 2 / masses[k] ** 2
            tol = 1e-12 if precision == "double" else 0.2 * np.sqrt(res[k]) * min(cond, 1e3)
            assert rel(got[1][0][k], got[0][0][k]) < tol, k


@pytest.mark.parametrize("precision", ["single", "half", "double"])
def test_a_window_keeps_no_memory(cuda_device, precision):
    """After a call a window of eight iterations holds what one of a single iteration does: the residuals lie in
    fields that are idle meanwhile.  FP64 needs four fields beyond them, and keeps them while they are a 64th of
    what is free at most."""
    import torch
    T, L = 24, 16  # FP64: 18.9 MB a field, seven besides the running one
    src = torch.from_numpy(wl.random_spinor(T * L ** 3, 47)).to("cuda:0")
    conf = wl.gauge_conf(T, L, 0.35, seed=48, device="cuda")
    used = []
    for n in (8, 1):
        with Lattice(T, L) as lat:
            lat.upload_conf(conf)
            lat.set_tuning("graph_iters", n)
            out = [torch.empty_like(src) for _ in range(2)]
            torch.cuda.synchronize()
            free0 = torch.cuda.mem_get_info()[0]
            lat.inv_tmQ2_cgm(0.15, [0.1, 0.5], src, 100000, [1e-16, 1e-16], precision=precision, out=out)
            used.append(free0 - torch.cuda.mem_get_info()[0])
    slack = 16 << 20  # the graphs' own memory
    more = 0
    if precision == "double" and 64 * 4 * T * L ** 3 * 192 <= torch.cuda.mem_get_info()[0]:
        more = 4 * T * L ** 3 * 192
    assert used[0] <= used[1] + more + slack, used


@pytest.mark.parametrize("precision", ["single", "double"])
def test_window_on_a_padded_lattice(cuda_device, precision):
    """216 sites a parity in planes of 256: fields used before in the caller's layout (Q^2) or for FP32 residuals
    leave nothing in the padding that a later reduction or solve could see."""
    T, L = 2, 6
    src = wl.random_spinor(T * L ** 3, 49)
    masses, res = [0.05, 0.4], [1e-20, 1e-18]
    with Lattice(T, L) as lat:
        lat.upload_conf(wl.gauge_conf(T, L, 0.35, seed=50))
        lat.apply_tmQ2(0.16, 0.1, src)
        got = []
        for n in (11, 8, 8):
            lat.set_tuning("graph_iters", n)
            got.append(lat.inv_tmQ2_cgm(0.16, masses, src, 100000, res, precision=precision))
            sol, st = lat.inv_tmQ2_cg(0.16, 0.05, src, 100000, 1e-20)
            assert st["true_rel_res2"] < 1e-20
            for k, m in enumerate(masses):
                r = lat.apply_tmQ2(0.16, m, got[-1][0][k]) - src
                assert np.vdot(r, r) / np.vdot(src, src) < 1.01 * res[k]
        for k in range(2):
            assert np.array_equal(got[1][0][k], got[2][0][k])
            assert rel(got[1][0][k], got[0][0][k]) < (1e-12 if precision == "double" else 1e-6)
