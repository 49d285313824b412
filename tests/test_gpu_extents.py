"""Unequal spatial extents, some with odd halves: the operators and solvers
against a plain numpy hop made of rolls of the lattice, with the kernels for
small lattices and without them."""
import numpy as np
import pytest

from nissa_b200 import Lattice
from nissa_b200 import workload as wl
from conftest import rel

pytestmark = pytest.mark.gpu

# partners of spins 0, 1 and their phase in 1 - gamma_mu: t, x, y, z
PAIR = [(2, 3, 1, 1), (3, 2, 1j, 1j), (3, 2, 1, -1), (2, 3, 1j, -1j)]


class Rolls:
    def __init__(self, dims, conf, anis):
        self.dims, self.anis = dims, anis
        U = conf.view(np.complex128).reshape(*dims, 4, 3, 3)
        self.U = [U[..., mu, :, :].copy() for mu in range(4)]
        self.U[0][-1] *= -1.0  # antiperiodic time
        self.par = sum(np.indices(dims)) & 1

    def hop(self, s):  # (*dims, 4, 3) complex
        acc = np.zeros_like(s)
        for mu in range(4):
            a, b, p0, p1 = PAIR[mu]
            f = self.anis if mu else 1.0
            for sg in (1, -1):
                v = np.roll(s, -1, mu) if sg > 0 else s
                h = np.stack([v[..., 0, :] + sg * p0 * v[..., a, :], v[..., 1, :] + sg * p1 * v[..., b, :]], -2)
                W = self.U[mu] if sg > 0 else np.conj(np.swapaxes(self.U[mu], -1, -2))
                u = f * np.einsum("...ij,...sj->...si", W, h)
                if sg < 0:
                    u = np.roll(u, 1, mu)
                acc[..., 0, :] += u[..., 0, :]
                acc[..., 1, :] += u[..., 1, :]
                acc[..., a, :] += np.conj(p0) * sg * u[..., 0, :]
                acc[..., b, :] += np.conj(p1) * sg * u[..., 1, :]
        return acc

    def spread(self, x, p):  # an e/o spinor as a full field
        f = np.zeros((*self.dims, 4, 3), np.complex128)
        f[self.par == p] = x.view(np.complex128).reshape(-1, 4, 3)
        return f

    def gather(self, f, p):
        return np.ascontiguousarray(f[self.par == p]).view(np.float64).reshape(-1, 4, 3, 2)

    def diag(self, f, kappa, mu, inverse=False):
        z = 1 / (2 * kappa) + 1j * mu * np.array([1, 1, -1, -1])[:, None]
        return f / z if inverse else f * z

    def g5(self, f):
        return f * np.array([1, 1, -1, -1])[:, None]

    def Q(self, f, kappa, mu):
        return self.g5(self.diag(f, kappa, mu) - 0.5 * self.hop(f))

    def K(self, f, kappa, mu):
        t = self.diag(self.hop(f), kappa, mu, inverse=True)
        return self.g5(self.diag(f, kappa, mu) - 0.25 * self.hop(t))


def _full(x, dims):
    return x.view(np.complex128).reshape(*dims, 4, 3)


@pytest.mark.parametrize("dims", [(6, 10, 14, 2), (4, 2, 6, 18), (10, 6, 4, 22), (20, 14, 10, 30)])
def test_operators_on_unequal_extents(cuda_device, dims):
    # the largest is above every size rule of the operators (42,000 sites a parity)
    V = int(np.prod(dims))
    kappa, mu, anis = 0.15, 0.03, 1.1
    conf = wl.gauge_conf(V, 1, 0.35, seed=3)  # independent links: any V of them
    x, xl = wl.random_spinor(V // 2, 4), wl.random_spinor(V, 5)
    R = Rolls(dims, conf, anis)
    want = {p: R.gather(R.hop(R.spread(x, 1 - p)), p) for p in (0, 1)}
    kern = R.gather(R.K(R.spread(x, 1), kappa, -mu), 1)
    kern2 = R.gather(R.K(R.spread(kern, 1), kappa, mu), 1)
    q = R.Q(_full(xl, dims), kappa, mu)
    q2 = R.Q(q, kappa, -mu)
    flat = lambda f: f.reshape(V, 4, 3).view(np.float64).reshape(V, 4, 3, 2)
    with Lattice(dims[0], 0, LX=dims[1], LY=dims[2], LZ=dims[3]) as lat:
        lat.upload_conf(conf)
        for small in (1, 0):
            lat.set_tuning("small_lattice", small)
            for p in (0, 1):
                assert rel(lat.tmn2Deo_or_tmn2Doe_eos(p, x, anis=anis), want[p]) < 1e-14
            assert rel(lat.tmDkern_eoprec_eos(kappa, -mu, x, anis=anis), kern) < 1e-14
            assert rel(lat.tmDkern_eoprec_square_eos(kappa, mu, x, anis=anis), kern2) < 1e-14
            assert rel(lat.apply_tmQ(kappa, mu, xl, anis=anis), flat(q)) < 1e-14
            assert rel(lat.apply_tmQ2(kappa, mu, xl, anis=anis), flat(q2)) < 1e-14


@pytest.mark.parametrize("precision", ["double", "single", "half"])
@pytest.mark.parametrize("dims", [(6, 10, 14, 2), (10, 6, 4, 22)])
def test_solves_on_unequal_extents(cuda_device, dims, precision):
    V = int(np.prod(dims))
    conf = wl.gauge_conf(V, 1, 0.35, seed=3)
    src = wl.random_spinor(V, 6)
    R = Rolls(dims, conf, 1.0)
    s = _full(src, dims)
    with Lattice(dims[0], 0, LX=dims[1], LY=dims[2], LZ=dims[3]) as lat:
        lat.upload_conf(conf)
        for small in (1, 0):
            lat.set_tuning("small_lattice", small)
            sol, _ = lat.inv_tmD_cg_eoprec(0.15, 0.02, src, 10000, 1e-22, precision=precision)
            r = R.g5(R.Q(_full(sol, dims), 0.15, 0.02)) - s
            # |varphi| and |src| differ by less than |D_ee^-1| and the hop, a factor of ten together
            assert np.linalg.norm(r) < 1e-10 * np.linalg.norm(s)
            q, _ = lat.inv_tmQ2_cg(0.15, 0.02, src, 10000, 1e-22, precision=precision)
            r = R.Q(R.Q(_full(q, dims), 0.15, -0.02), 0.15, 0.02) - s
            assert np.linalg.norm(r) < 1e-10 * np.linalg.norm(s)
