"""The work that programs have this library do, as cases that can be timed and checked.

A case is one call (or one loop over the columns of a propagator) of
``nissa_b200.Lattice``: an operator, a solve, a batch of solves, a multi-shift
solve, a twisted-clover operator or solve.  Sizes run from 4^4, where a call is
launches and latency, to 32^3x64; the lattices of the benchmark (8^3x16, 16^3x32,
24^3x48, 32^3x64) are listed, and lattices with unequal and odd half-extents are
drawn.  Inputs follow the benchmark's recipe: links exp(i eps H) with Gaussian
traceless Hermitian H and eps = 0.35, projected onto SU(3); point sources for
propagators, Z2 noise for the multi-shift solves, Gaussian spinors for the operators.

``exact`` computes the same in plain torch, in 64 bits, from the full-lattice
operator: rolls of the lattice instead of even/odd tables, and a conjugate gradient
on D^+ D run to 1e-14 instead of the Schur complement.
"""
import math

import numpy as np
import torch

from nissa_b200 import Lattice

EPS = 0.35
OPERATORS = ("hop", "kern2", "tmQ", "clov_kern2")
SOLVES = ("solve", "columns", "batched", "cgm", "clov_solve")


def _case(name, call, dims, kappa, mu, precision="double", anis=None, count=1, csw=0.0, residue=1e-20):
    T, LX, LY, LZ = dims
    c = dict(call=call, T=T, LX=LX, LY=LY, LZ=LZ, kappa=kappa, mu=mu, precision=precision, anis=anis, count=count,
             csw=csw, residue=residue)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call that the benchmark's lattices give: an even/odd hop at 8^3x16, as an
        # application that keeps its own solver calls it, thousands of times in a row
        _case("hop_8c16", "hop", (16, 8, 8, 8), 0.161, 0.005),
        # the same operator at production size
        _case("hop_32c64", "hop", (64, 32, 32, 32), 0.161, 0.005),
        # the matrix of an application's own CG, on a lattice with unequal and odd half-extents, anisotropic
        _case("kern2_14x10x12x20", "kern2", (20, 14, 10, 12), 0.15, 0.01, anis=1.15),
        # the full-lattice operator on lx fields: contractions, residual checks
        _case("tmQ_24c48", "tmQ", (48, 24, 24, 24), 0.161, 0.005),
        # the twisted-clover matrix of an application's own CG, at 16^3x32
        _case("clov_kern2_16c32", "clov_kern2", (32, 16, 16, 16), 0.135, 0.005, csw=1.6),
        # plain FP64 CG from a point source at 8^3x16 to 1e-12: the benchmark's smallest configuration
        _case("solve_double_8c16", "solve", (16, 8, 8, 8), 0.161, 0.005, residue=1e-24),
        # the drop-in shim's default: a FP64 solve, at 16^3x32
        _case("solve_double_16c32", "solve", (32, 16, 16, 16), 0.161, 0.005),
        # a propagator: twelve point columns through page-locked host buffers, FP32 inner solver, 16^3x32
        _case("columns_single_16c32", "columns", (32, 16, 16, 16), 0.161, 0.005, precision="single", count=12),
        # the benchmark's headline: one mixed-precision solve at 32^3x64
        _case("solve_half_32c64", "solve", (64, 32, 32, 32), 0.161, 0.005, precision="half"),
        # a propagator's twelve columns as one batch at 24^3x48
        _case("batched_half_24c48", "batched", (48, 24, 24, 24), 0.161, 0.005, precision="half", count=12),
        # the multi-shift solve of a rational approximation: eight masses, 24^3x48
        _case("cgm_single_24c48", "cgm", (48, 24, 24, 24), 0.1632, 0.002, precision="single", count=8),
        # a twisted-clover propagator column, FP16 inner solver, 24^3x48
        _case("clov_solve_half_24c48", "clov_solve", (48, 24, 24, 24), 0.135, 0.005, precision="half", csw=1.6),
    ]


def draw(rng):
    call = rng.choice(OPERATORS + OPERATORS + SOLVES)
    top = {"hop": 1 << 21, "kern2": 1 << 20, "tmQ": 1 << 20, "clov_kern2": 1 << 19, "solve": 1 << 19,
           "columns": 1 << 15, "batched": 1 << 16, "cgm": 1 << 17, "clov_solve": 1 << 18}[call]
    precision = "double" if call in OPERATORS else rng.choice(["double", "single", "half"])
    if precision == "double":
        top = min(top, 1 << 18) if call in SOLVES else top
    target = math.exp(rng.uniform(math.log(256), math.log(top)))
    while True:
        dims = [2 * int(round(math.exp(rng.uniform(math.log(2), math.log(b))))) for b in (32, 16, 16, 16)]
        v = math.prod(dims)
        if target / 2 <= v <= min(2 * target, top):
            break
    kappa = round(rng.uniform(0.12, 0.135 if call.startswith("clov") else 0.161), 4)
    mu = round(math.exp(rng.uniform(math.log(0.002), math.log(0.05))), 5) * rng.choice([1, -1])
    anis = round(rng.uniform(0.8, 1.2), 3) if call in OPERATORS and rng.random() < 0.5 else None
    count = {"columns": rng.choice([3, 12]), "batched": rng.randint(2, 16), "cgm": rng.randint(2, 10)}.get(call, 1)
    csw = round(rng.uniform(0.8, 2.0), 3) if call.startswith("clov") else 0.0
    if call == "cgm":
        mu = abs(mu)
    return _case(None, call, dims, kappa, mu, precision, anis, count, csw, rng.choice([1e-16, 1e-20, 1e-20, 1e-24]))


# ------------------------------------------------------------------- inputs

def _dims(c):
    return c["T"], c["LX"], c["LY"], c["LZ"]


def _volume(c):
    return math.prod(_dims(c))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _conf(c, seed):
    """Periodic SU(3) links exp(i eps H), complex128 (V, 4, 3, 3), on the GPU."""
    n = _volume(c) * 4
    g = _gen(seed)
    out = torch.empty((n, 3, 3), dtype=torch.complex128, device="cuda")
    for s in range(0, n, 1 << 21):
        m = min(1 << 21, n - s)
        r = torch.randn((8, m), dtype=torch.float64, device="cuda", generator=g) * math.sqrt(0.5)
        H = torch.zeros((m, 3, 3), dtype=torch.complex128, device="cuda")
        H[:, 0, 0] = r[2] + r[7] / math.sqrt(3)
        H[:, 1, 1] = -r[2] + r[7] / math.sqrt(3)
        H[:, 2, 2] = -2 * r[7] / math.sqrt(3)
        for (a, b), k in (((1, 0), 0), ((2, 0), 3), ((2, 1), 5)):
            H[:, a, b] = torch.complex(r[k], r[k + 1])
            H[:, b, a] = torch.complex(r[k], -r[k + 1])
        A = H * (1j * EPS / 8)
        U = torch.eye(3, dtype=torch.complex128, device="cuda") + A / 8
        for k in range(7, 0, -1):  # Horner's form of the exponential series, then three squarings
            U = torch.eye(3, dtype=torch.complex128, device="cuda") + (A @ U) / k
        for _ in range(3):
            U = U @ U
        a = U[:, 0] / U[:, 0].abs().square().sum(-1, keepdim=True).sqrt()
        b = U[:, 1] - (a.conj() * U[:, 1]).sum(-1, keepdim=True) * a
        b = b / b.abs().square().sum(-1, keepdim=True).sqrt()
        out[s:s + m, 0], out[s:s + m, 1] = a, b
        out[s:s + m, 2] = torch.linalg.cross(a, b, dim=-1).conj()
    return out.reshape(-1, 4, 3, 3)


def _gauss(n, seed):
    return torch.randn((n, 4, 3, 2), dtype=torch.float64, device="cuda", generator=_gen(seed + (1 << 20)))


def _z2(n, seed):
    bits = torch.randint(0, 2, (n, 4, 3, 2), device="cuda", generator=_gen(seed + (2 << 20)))
    return (2.0 * bits.double() - 1.0) / math.sqrt(2.0)


def _points(c, seed, count):
    """Point sources at one site of the seed's choice, the spin-colour columns in turn."""
    rng = np.random.default_rng(seed)
    site, first = int(rng.integers(_volume(c))), int(rng.integers(12))
    out = []
    for k in range(count):
        s = torch.zeros((_volume(c), 4, 3, 2), dtype=torch.float64, device="cuda")
        col = (first + k) % 12
        s[site, col // 3, col % 3, 0] = 1.0
        out.append(s)
    return out


def _masses(c):
    return [float(m) for m in np.geomspace(c["mu"], max(0.2, 2 * c["mu"]), c["count"])]


def _sources(c, seed):
    V = _volume(c)
    call = c["call"]
    if call in ("hop", "kern2", "clov_kern2"):
        return [_gauss(V // 2, seed)]
    if call == "tmQ":
        return [_gauss(V, seed)]
    if call == "cgm":
        return [_z2(V, seed)]
    return _points(c, seed, c["count"])


def prepare(case, seed):
    c = dict(case)
    lat = Lattice(c["T"], 0, device=torch.cuda.current_device(), LX=c["LX"], LY=c["LY"], LZ=c["LZ"])
    lat.upload_conf(torch.view_as_real(_conf(c, seed)).contiguous())
    if c["call"] == "clov_kern2":
        lat.clover_term(c["csw"])
    src = _sources(c, seed)
    if c["call"] == "columns":
        src = [s.cpu().pin_memory() for s in src]
        out = [torch.empty_like(s).pin_memory() for s in src]
    elif c["call"] == "cgm":
        out = [torch.empty_like(src[0]) for _ in range(c["count"])]
    else:
        out = [torch.empty_like(s) for s in src]
    return dict(c=c, lat=lat, src=src, out=out)


def run(state):
    c, lat, src, out = state["c"], state["lat"], state["src"], state["out"]
    call, kappa, mu = c["call"], c["kappa"], c["mu"]
    if call == "hop":
        return lat.tmn2Deo_or_tmn2Doe_eos(0, src[0], anis=c["anis"], out=out[0])
    if call == "kern2":
        return lat.tmDkern_eoprec_square_eos(kappa, mu, src[0], anis=c["anis"], out=out[0])
    if call == "tmQ":
        return lat.apply_tmQ(kappa, mu, src[0], anis=c["anis"], out=out[0])
    if call == "clov_kern2":
        return lat.tmclovDkern_eoprec_square_eos(kappa, mu, src[0], anis=c["anis"], out=out[0])
    kw = dict(niter=100000, precision=c["precision"])
    if call == "solve":
        return lat.inv_tmD_cg_eoprec(kappa, mu, src[0], residue=c["residue"], out=out[0], **kw)[0]
    if call == "clov_solve":
        return lat.inv_tmclovD_cg_eoprec(kappa, c["csw"], mu, src[0], residue=c["residue"], out=out[0], **kw)[0]
    if call == "columns":
        return lat.inv_tmD_cg_eoprec_columns(kappa, mu, src, residue=c["residue"], out=out, **kw)[0]
    if call == "batched":
        return lat.inv_tmD_cg_eoprec_batched(kappa, [mu] * len(src), src, residues=c["residue"], out=out, **kw)[0]
    return lat.inv_tmQ2_cgm(kappa, _masses(c), src[0], residues=c["residue"], out=out, **kw)[0]


# --------------------------------------------------------------- the measure

def _iterations(c):
    """About the iterations that the case's solves take: half the logarithm of the squared residue over
    the logarithm of the convergence per iteration, which follows the distance to the critical mass."""
    m = max(abs(c["mu"]), 0.02) if c["call"] == "cgm" else 0.5 / c["kappa"] - 0.5 / 0.1632 + abs(c["mu"])
    if c["call"] == "clov_solve":
        m = 0.5 / c["kappa"] - 0.5 / 0.139 + abs(c["mu"])
    return 0.5 * math.log(1 / c["residue"]) * (1.0 + 0.6 / math.sqrt(max(m, 0.01)))


def work(case):
    c = dict(case)
    Vh = _volume(c) // 2
    call = c["call"]
    spinor, link, clov = 192, 144, 72 * 16
    # each input once and each output once: 8 links per output site of a hop
    hop = (8 * link + 2 * spinor) * Vh
    hop_flops = 1320 * Vh
    if call == "hop":
        return dict(bytes=hop, flops=hop_flops)
    if call == "kern2":
        return dict(bytes=4 * hop + 2 * spinor * Vh, flops=4 * (hop_flops + 100 * Vh))
    if call == "tmQ":
        return dict(bytes=2 * (8 * link + 2 * spinor) * Vh, flops=2 * (hop_flops + 100 * Vh))
    if call == "clov_kern2":
        return dict(bytes=4 * hop + 2 * (spinor + 54 * 8 + clov) * Vh, flops=4 * (hop_flops + 500 * Vh))
    # one CG iteration: four hops, the vectors of the recurrence; at the inner precision
    sp, ln = {"double": (192, 144), "single": (96, 24), "half": (52, 24)}[c["precision"]]
    n = {"columns": c["count"], "batched": c["count"]}.get(call, 1)
    per = 4 * (8 * ln + 2 * sp) + 8 * sp
    if call == "clov_solve":
        per += 2 * (54 + 144) * (8 if c["precision"] == "double" else 4)
    if call == "cgm":  # full-lattice vectors, four per shift and iteration
        per = 2 * (2 * (8 * max(ln, 48) + 2 * max(sp, 96)) + (4 + 4 * c["count"]) * max(sp, 96))
    it = _iterations(c)
    if call == "batched":  # the links once for all right-hand sides
        per = 4 * (8 * ln / n + 2 * sp) + 8 * sp
    return dict(bytes=n * it * per * Vh, flops=n * it * 4 * 1500 * Vh)


def tolerance(case):
    # measured against exact(): 0.8e-16 (hop) to 2.5e-16 (twisted-clover square)
    if case["call"] in OPERATORS:
        return {"rel": 1e-15}
    # solutions agree as far as their residues say: 0.7 to 3.1 times the relative residue from exact()
    rel = 12 * math.sqrt(case["residue"]) + 2e-12
    return {"rel": rel, "max": 100 * rel}


# ------------------------------------------------- the same in plain torch, 64 bits

BC = -1.0


def _field(x, dims):
    """(V, 4, 3, 2) float64 -> (4, 3, T, X, Y, Z) complex128"""
    return torch.view_as_complex(x.contiguous()).permute(1, 2, 0).reshape(4, 3, *dims).contiguous()


def _unfield(f):
    return torch.view_as_real(f.reshape(4, 3, -1).permute(2, 0, 1).contiguous())


def _parity(dims, device="cuda"):
    g = torch.meshgrid(*[torch.arange(n, device=device) for n in dims], indexing="ij")
    return (g[0] + g[1] + g[2] + g[3]) & 1


def _project(s, mu, sg):
    """The two rows of (1 -+ gamma_mu) s, sg = +1 forward, -1 backward."""
    if mu == 0:
        return s[0] + sg * s[2], s[1] + sg * s[3]
    if mu == 1:
        return s[0] + 1j * sg * s[3], s[1] + 1j * sg * s[2]
    if mu == 2:
        return s[0] + sg * s[3], s[1] - sg * s[2]
    return s[0] + 1j * sg * s[2], s[1] - 1j * sg * s[3]


def _reconstruct(acc, u0, u1, mu, sg):
    acc[0] += u0
    acc[1] += u1
    if mu == 0:
        acc[2] += sg * u0
        acc[3] += sg * u1
    elif mu == 1:
        acc[2] -= 1j * sg * u1
        acc[3] -= 1j * sg * u0
    elif mu == 2:
        acc[2] -= sg * u1
        acc[3] += sg * u0
    else:
        acc[2] -= 1j * sg * u0
        acc[3] += 1j * sg * u1


class _Exact:
    def __init__(self, c, seed):
        self.c, self.dims = c, _dims(c)
        U = _conf(c, seed).reshape(*self.dims, 4, 3, 3)
        self.U = [U[..., mu, :, :].permute(4, 5, 0, 1, 2, 3).contiguous() for mu in range(4)]
        self.U[0][:, :, -1] *= BC  # the antiperiodic time boundary
        self.anis = 1.0 if c["anis"] is None else c["anis"]
        self.kcf = 1 / (2 * c["kappa"])
        self.clov = self._clover() if c["csw"] else None

    def hop(self, s):
        acc = torch.zeros_like(s)
        for mu in range(4):
            U, f = self.U[mu], (self.anis if mu else 1.0)
            h = torch.stack(_project(torch.roll(s, -1, mu + 2), mu, 1))
            u = sum(U[:, j] * h[:, j, None] for j in range(3)) * f
            _reconstruct(acc, u[0], u[1], mu, 1)
            h = torch.stack(_project(s, mu, -1))
            u = sum(U[j].conj() * h[:, j, None] for j in range(3)) * f
            u = torch.roll(u, 1, mu + 2)
            _reconstruct(acc, u[0], u[1], mu, -1)
        return acc

    def _clover(self):
        """The clover term's four 3x3 blocks, (4, 3, 3, T, X, Y, Z)."""
        def mm(a, b):
            return torch.stack([torch.stack([sum(a[i, k] * b[k, j] for k in range(3)) for j in range(3)])
                                for i in range(3)])

        def dag(a):
            return a.conj().transpose(0, 1)

        def sh(a, mu, k):
            return torch.roll(a, -k, mu + 2)

        U, P = self.U, []
        for mu in range(4):
            for nu in range(mu + 1, 4):
                p = mm(mm(U[mu], sh(U[nu], mu, 1)), mm(dag(sh(U[mu], nu, 1)), dag(U[nu])))
                # the plaquette seen from its four corners
                q = p
                a = mm(mm(U[nu], dag(sh(sh(U[mu], mu, -1), nu, 1))), mm(dag(sh(U[nu], mu, -1)), sh(U[mu], mu, -1)))
                q = q + a
                x = sh(U[mu], mu, -1)
                y = sh(sh(U[nu], mu, -1), nu, -1)
                z = sh(sh(U[mu], mu, -1), nu, -1)
                w = sh(U[nu], nu, -1)
                q = q + mm(mm(dag(x), dag(y)), mm(z, w))
                q = q + mm(mm(dag(w), sh(U[mu], nu, -1)), mm(sh(sh(U[nu], nu, -1), mu, 1), dag(U[mu])))
                P.append((q - dag(q)) / 4)
        f = -(self.c["csw"] + 1e-16) / 4
        A, B, C = P[3] - P[2], P[4] + P[1], P[5] - P[0]
        D, E, F = P[3] + P[2], P[4] - P[1], P[5] + P[0]
        return torch.stack([1j * A, B + 1j * C, 1j * D, E + 1j * F]) * f

    def clover(self, s):
        if self.clov is None:
            return torch.zeros_like(s)
        mv = lambda m, v: torch.stack([sum(m[i, j] * v[j] for j in range(3)) for i in range(3)])  # noqa: E731
        o = []
        for b in range(2):
            c0, c1, i0, i1 = self.clov[2 * b], self.clov[2 * b + 1], s[2 * b], s[2 * b + 1]
            o += [mv(c0, i0) + mv(c1.conj().transpose(0, 1), i1), mv(c1, i0) - mv(c0, i1)]
        return torch.stack(o)

    def diag(self, s, mu):
        o = self.kcf * s + self.clover(s)
        o[:2] += 1j * mu * s[:2]
        o[2:] -= 1j * mu * s[2:]
        return o

    def inv_diag(self, s, mu):
        if self.clov is None:
            z = complex(self.kcf, mu)
            return torch.cat([s[:2] / z, s[2:] / z.conjugate()])
        o = []
        for b in range(2):
            z = complex(self.kcf, -mu if b else mu)
            c0, c1 = self.clov[2 * b], self.clov[2 * b + 1]
            top = torch.cat([c0, c1.conj().transpose(0, 1)], 1)
            M = torch.cat([top, torch.cat([c1, -c0], 1)], 0).reshape(6, 6, -1).permute(2, 0, 1)
            M = M + z * torch.eye(6, dtype=torch.complex128, device=s.device)
            v = s[2 * b:2 * b + 2].reshape(6, -1).permute(1, 0)[..., None]
            o.append(torch.linalg.solve(M, v)[..., 0].permute(1, 0).reshape(2, 3, *self.dims))
        return torch.cat(o)

    def Q(self, s, mu):
        o = self.diag(s, mu) - self.hop(s) / 2
        o[2:] *= -1
        return o

    def kern(self, s, mu, odd):
        """The Schur operator on the odd sites of s."""
        te = self.inv_diag(self.hop(s) * (1 - odd), mu)
        o = self.diag(s, mu) - self.hop(te) / 4
        o[2:] *= -1
        return o * odd

    def cg(self, b, mu, m2=None, tol=1e-14):
        """(Q(-mu) Q(mu))^-1 b, or (Q(0)^2 + m2)^-1 b."""
        if m2 is None:
            op = lambda v: self.Q(self.Q(v, mu), -mu)  # noqa: E731
        else:
            op = lambda v: self.Q(self.Q(v, 0.0), 0.0) + m2 * v  # noqa: E731
        x, b2 = torch.zeros_like(b), float(b.abs().square().sum())
        for _ in range(3):  # restarted from the recomputed residue
            r = b - op(x)
            p, rr = r, float(r.abs().square().sum())
            for _ in range(3000):
                if rr <= (tol / 10) ** 2 * b2:
                    break
                Ap = op(p)
                a = rr / float((p.conj() * Ap).sum().real)
                x = x + a * p
                r = r - a * Ap
                new = float(r.abs().square().sum())
                p, rr = r + (new / rr) * p, new
        return x

    def solve(self, src, mu):
        """D^-1 src = (Q^+ Q)^-1 Q^+ g5 src"""
        s = src.clone()
        s[2:] *= -1
        return self.cg(self.Q(s, -mu), mu)


def exact(case, seed):
    c = dict(case)
    dims, call, mu = _dims(c), c["call"], c["mu"]
    src = _sources(c, seed)
    e = _Exact(c, seed)
    if call in ("hop", "kern2", "clov_kern2"):
        par = _parity(dims)
        full = torch.zeros((_volume(c), 4, 3, 2), dtype=torch.float64, device="cuda")
        full[par.reshape(-1) == 1] = src[0]
        s = _field(full, dims)
        if call == "hop":
            return _unfield(e.hop(s))[par.reshape(-1) == 0]
        first, second = (-mu, mu)
        return _unfield(e.kern(e.kern(s, first, par), second, par))[par.reshape(-1) == 1]
    if call == "tmQ":
        return _unfield(e.Q(_field(src[0], dims), mu))
    if call == "cgm":
        s, ms = _field(src[0], dims), _masses(c)
        some = {0, len(ms) // 2, len(ms) - 1}
        return [_unfield(e.cg(s, 0.0, m2=m * m)) if k in some else None for k, m in enumerate(ms)]
    some = 12 if _volume(c) <= 16384 else 2
    sols = [_unfield(e.solve(_field(s, dims), mu)) if k < some else None for k, s in enumerate(src)]
    if call in ("solve", "clov_solve"):
        return sols[0]
    return [None if s is None else s.cpu() for s in sols] if call == "columns" else sols
