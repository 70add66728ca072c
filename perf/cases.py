"""Performance cases: calls of the public Python entry points over the ranges
their users work in.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs and handles a program has before the call
    run(state)          one pass through the public entry points
    work(case)          bytes and flops one pass cannot do without (estimated
                        from the size parameters, not from a run)
    exact(case, seed)   the outputs from a plain torch evaluation in 64 bits

Kinds of case and what they stand for:

    batch    Context.tmatrix_batch: converged T-matrices of independent grains,
             the library's main path. One grain per call is the latency end
             (a caller that asks for one particle at a time), 4096 grains the
             batched benchmark; "download" cases also fetch every T-matrix,
             "graph" ones use the device-driven mode.
    fixed    Context.tmatrix_batch_fixed + observables: large grains at given
             orders (a program that knows its orders, or recomputes a batch).
    grad     autograd.extinction forward and backward: few grains and two
             directions (a gradient fit), or a batch at 32 angles.
    table    CosTuuM.get_table: the averaged coefficients of dust grids, with
             absorption, extinction, scattering matrices and the scattering
             subtraction.
    particle CosTuuM.TMatrix: one particle on the plain path, its averaged
             T-matrix and its scattering, extinction and absorption.
    plain    Context.tmatrix_batch_calculator + orientation_average +
             scattering_matrix: large elongated grains on the plain path (some
             of them do not converge, as with the reference).
"""
import functools
import math

import numpy as np
import torch

from costuum_b200 import CosTuuM
from costuum_b200.autograd import extinction
from costuum_b200.tmatrix import Context, tmatrix_size

LAM = 1e-6  # wavelength of the cases that take one (m)


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # one particle per call
        dict(name="batch one grain", kind="batch", n=1, xmin=0.1, xmax=10.0,
             graph=False),
        # the batched benchmark
        dict(name="batch 4096", kind="batch", n=4096, xmin=0.1, xmax=10.0,
             graph=False),
        # the device-driven mode on an ordinary batch
        dict(name="batch 1000 graph", kind="batch", n=1000, xmin=0.1, xmax=10.0,
             graph=True),
        # a few dozen grains whose T-matrices the caller wants back
        dict(name="fixed 53 download", kind="fixed", n=53, xmin=0.5, xmax=10.0,
             ntheta=0),
        # large grains at known orders (23 .. 50)
        dict(name="fixed large 96", kind="fixed", n=96, xmin=12.0, xmax=35.0,
             ntheta=16),
        # one step of a gradient fit
        dict(name="grad fit 16", kind="grad", n=16, xmin=0.6, xmax=3.2, ntheta=2,
             aligned=False),
        # forward and gradient of a batch
        dict(name="grad batch 1024", kind="grad", n=1024, xmin=0.1, xmax=10.0,
             ntheta=32, aligned=True),
        # averaged coefficients: radii x wavelengths x shapes, 32 angles
        dict(name="table averages", kind="table", nsizes=8, nlam=12, nshape=20,
             ntheta=32, rmin=0.01e-6, rmax=2e-6, lmin=0.25e-6, lmax=1e-4,
             alignment=2, absorption=True, extinction=True, scattering=False,
             account=False, nquad=20),
        # scattering matrices of a few cells
        dict(name="table scattering", kind="table", nsizes=3, nlam=4, nshape=5,
             ntheta=37, rmin=0.1e-6, rmax=0.5e-6, lmin=0.5e-6, lmax=2e-6,
             alignment=1, absorption=True, extinction=True, scattering=True,
             account=False, nquad=20),
        # absorption with the scattering subtracted
        dict(name="table subtraction", kind="table", nsizes=4, nlam=5, nshape=5,
             ntheta=9, rmin=0.05e-6, rmax=0.5e-6, lmin=0.5e-6, lmax=2e-6,
             alignment=2, absorption=True, extinction=False, scattering=False,
             account=True, nquad=20),
        # one particle on the plain path
        dict(name="plain particle", kind="particle", x=5.0, d=0.6, nout=181,
             nabs=5, nquad=20),
        # large elongated grains on the plain path
        dict(name="plain batch 40", kind="plain", n=40, xmin=10.0, xmax=30.0,
             nout=181),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["batch", "batch", "fixed", "grad", "table", "table",
                       "particle", "plain"])
    if kind == "batch":
        return dict(kind=kind, n=round(_log(rng, 1, 4096)), xmin=0.1,
                    xmax=rng.uniform(3.0, 10.0), graph=rng.random() < 0.2)
    if kind == "fixed":
        xmin = rng.uniform(0.5, 15.0)
        n = round(_log(rng, 4, 96))
        return dict(kind=kind, n=n, xmin=xmin, xmax=xmin + rng.uniform(2.0, 20.0),
                    ntheta=0 if n <= 53 and rng.random() < 0.5 else rng.randint(3, 19))
    if kind == "grad":
        n = round(_log(rng, 8, 1024))
        return dict(kind=kind, n=n, xmin=0.3, xmax=rng.uniform(3.0, 10.0),
                    ntheta=rng.randint(2, 32), aligned=rng.random() < 0.5)
    if kind == "table":
        form = rng.choice(["averages", "scattering", "account"])
        rmax = _log(rng, 0.2e-6, 1e-6 if form == "averages" else 0.5e-6)
        return dict(kind=kind, nsizes=rng.randint(1, 8 if form == "averages" else 3),
                    nlam=rng.randint(2, 12 if form == "averages" else 4),
                    nshape=rng.choice([1, 4, 5, 10, 20] if form == "averages"
                                      else [1, 4, 5]),
                    ntheta=rng.randint(5, 33 if form != "account" else 9),
                    rmin=0.05e-6, rmax=rmax, lmin=0.5e-6, lmax=_log(rng, 2e-6, 1e-4),
                    alignment=rng.choice([0, 1, 2]), absorption=form != "scattering",
                    extinction=rng.random() < 0.5 or form == "scattering",
                    scattering=form == "scattering", account=form == "account",
                    nquad=rng.randint(6, 20))
    if kind == "particle":
        return dict(kind=kind, x=rng.uniform(0.5, 12.0), d=_log(rng, 0.5, 2.0),
                    nout=rng.randint(19, 181), nabs=rng.randint(1, 5),
                    nquad=rng.randint(8, 20))
    xmin = rng.uniform(4.0, 12.0)
    return dict(kind=kind, n=round(_log(rng, 2, 40)), xmin=xmin,
                xmax=xmin + rng.uniform(2.0, 16.0), nout=rng.randint(31, 181))


# ----------------------------------------------------------------- inputs --

@functools.lru_cache(maxsize=None)
def _context(graph=False):
    """The program's context: one per batch mode, kept across calls."""
    ctx = Context(0)
    if graph:
        ctx.set_batch_mode(Context.BATCH_GRAPH)
    return ctx


@functools.lru_cache(maxsize=None)
def _alignment(kind, order):
    t = (CosTuuM.DISABLE_ALIGNMENT, CosTuuM.MISHCHENKO_ALIGNMENT,
         CosTuuM.DAVIS_GREENSTEIN_ALIGNMENT)[kind]
    return CosTuuM.SizeBasedAlignmentDistribution(0.1e-6, t, maximum_order=order)


@functools.lru_cache(maxsize=None)
def _shapes(n):
    return (CosTuuM.SingleShapeShapeDistribution(1.5) if n == 1
            else CosTuuM.DraineHensleyShapeDistribution(n))


@functools.lru_cache(maxsize=None)
def _random_orientation(order):
    return CosTuuM.RandomOrientationDistribution(order).coefficients


def _grains(n, seed, xmin, xmax, dmin=0.5, dmax=2.0):
    """Spheroids as the benchmark draws them: (r_ev, m, axis ratio)."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(xmin, xmax, n)
    d = np.exp(rng.uniform(math.log(dmin), math.log(dmax), n))
    m = rng.uniform(1.3, 2.0, n) + 1j * np.exp(rng.uniform(math.log(1e-3), 0.0, n))
    return x * LAM / (2 * np.pi), m, d


def _fixed_grains(case, seed):
    """Grains of evenly spaced size parameters, a little shifted by the seed,
    and the orders that go with the unshifted ones."""
    rng = np.random.default_rng(seed)
    x = np.linspace(case["xmin"], case["xmax"], case["n"])
    _, m, d = _grains(case["n"], seed, 1.0, 2.0, 0.67, 1.5)
    r = x * np.exp(rng.uniform(-0.02, 0.02, x.size)) * LAM / (2 * np.pi)
    return (r, m, d), (x + 4.05 * np.cbrt(x) + 2).astype(np.int32)


def _grid(case, seed):
    """Radii and wavelengths of a table: logarithmic grids, a little shifted
    by the seed."""
    rng = np.random.default_rng(seed)
    sizes = np.geomspace(case["rmin"], case["rmax"], case["nsizes"] + 2)[1:-1]
    lams = np.geomspace(case["lmin"], case["lmax"], case["nlam"] + 2)[1:-1]
    return (sizes * np.exp(rng.uniform(-0.05, 0.05, sizes.size)),
            lams * np.exp(rng.uniform(-0.05, 0.05, lams.size)))


def _dielectric(lam):
    """Refractive index with resonances at 9.7, 18 and 25 um, the model of the
    averaged-grid benchmark plus an absorbing continuum."""
    w = 1.0 / (lam * 1e6)
    eps = 2.5 + 0.1j
    for lj, f in ((9.7, 0.8), (18.0, 0.4), (25.0, 0.2)):
        eps += f / lj ** 2 / (1.0 / lj ** 2 - w * w - 0.1j * w / lj)
    return complex(np.sqrt(eps))


def _thetas(n):
    return np.arccos(np.linspace(-1, 1, n)) if n > 2 else np.array([0.3, 1.2])[:n]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "batch":
        s["ctx"] = _context(case["graph"])
        s["grains"] = _grains(case["n"], seed, case["xmin"], case["xmax"])
    elif kind == "fixed":
        s["ctx"] = _context()
        s["grains"], s["nmax"] = _fixed_grains(case, seed)
        s["coeffs"] = _random_orientation(2 * 64)
        s["thetas"] = _thetas(case["ntheta"])
    elif kind == "grad":
        r, m, d = _grains(case["n"], seed, case["xmin"], case["xmax"])
        s["params"] = torch.tensor(np.stack([m.real, m.imag, r, d], 1),
                                   dtype=torch.float64, requires_grad=True)
        s["thetas"] = _thetas(case["ntheta"])
        rng = np.random.default_rng(seed + 1)
        s["upstream"] = torch.tensor(rng.normal(size=(case["n"], case["ntheta"], 3)))
        s["coeffs"] = _alignment(2, 100).prolate.coefficients if case["aligned"] else None
    elif kind == "table":
        s["ctx"] = _context()
        s["sizes"], s["lams"] = _grid(case, seed)
        s["kw"] = dict(
            types=np.array([0]), sizes=s["sizes"], wavelengths=s["lams"],
            thetas=_thetas(case["ntheta"]),
            shape_distribution=_shapes(case["nshape"]),
            alignment_distribution=_alignment(case["alignment"], 100),
            dust_properties=CosTuuM.CustomDustProperties(lambda w, a, t: _dielectric(w)),
            do_absorption=case["absorption"], do_extinction=case["extinction"],
            do_scattering=case["scattering"],
            account_for_scattering=case["account"],
            number_of_quadrature_angles=case["nquad"], context=s["ctx"])
    elif kind == "particle":
        rng = np.random.default_rng(seed)
        s["r"] = case["x"] * math.exp(rng.uniform(-0.02, 0.02)) * LAM / (2 * math.pi)
        s["m"] = complex(rng.uniform(1.3, 1.7), 10 ** rng.uniform(-3, -1))
        s["out"] = np.linspace(0.0, np.pi, case["nout"])
        s["abs"] = np.linspace(0.2, 1.4, case["nabs"])
    else:
        s["ctx"] = _context()
        s["grains"] = _grains(case["n"], seed, case["xmin"], case["xmax"], 0.33, 3.0)
        s["out"] = np.linspace(0.0, np.pi, case["nout"])
        s["coeffs"] = _random_orientation(400)
    return s


# -------------------------------------------------------------------- run --

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        r, m, d = s["grains"]
        res = s["ctx"].tmatrix_batch(r, LAM, m, d)
        return dict(nmax=res.nmax, ngauss=res.ngauss, status=res.status, q=res.q)
    if kind == "fixed":
        r, m, d = s["grains"]
        res = s["ctx"].tmatrix_batch_fixed(r, LAM, m, d, s["nmax"], 2 * s["nmax"])
        out = dict(status=res.status, q=res.q[:, 2:4])
        if case["ntheta"]:
            out["obs"] = s["ctx"].observables(s["thetas"], s["coeffs"])
        else:
            flat, off = s["ctx"].tmatrices()
            out["T"] = [flat[o:o + tmatrix_size(k)] for o, k in zip(off, s["nmax"])]
        return out
    if kind == "grad":
        p = s["params"]
        p.grad = None
        q = extinction(p, LAM, s["thetas"], s["coeffs"])
        q.backward(s["upstream"])
        return dict(q=q.detach(), grad=p.grad)
    if kind == "table":
        out = CosTuuM.get_table(return_status=True, **s["kw"])
        return list(out)
    if kind == "particle":
        t = CosTuuM.TMatrix(s["r"], case["d"], LAM, s["m"])
        return dict(order=t.get_nmax(), ngauss=t.get_ngauss(),
                    Z=t.get_scattering_matrix(0.3, 0.0, s["out"], 0.5),
                    K=t.get_extinction_matrix(s["abs"], 0.0),
                    C=t.get_absorption_cross_sections(s["abs"], case["nquad"]))
    r, m, d = s["grains"]
    n, no = case["n"], case["nout"]
    res = s["ctx"].tmatrix_batch_calculator(r, LAM, m, d)
    s["ctx"].orientation_average(s["coeffs"], np.where(res.nmax > 0, 0, -1))
    Z = s["ctx"].scattering_matrix(np.repeat(np.arange(n), no), 0.0, 0.0,
                                   np.tile(s["out"], n), 0.0)
    return dict(nmax=res.nmax, ngauss=res.ngauss, status=res.status, Z=Z)


# ------------------------------------------------------------------- work --

def _order(x):
    return int(max(11, x + 4.05 * x ** (1 / 3) + 1))


def _blocks_flops(N, ng):
    """Assembly, factors and solves of every parity class at order N."""
    f = 4 * (16 * (N / 2) ** 2 * ng + 10.7 * (N / 2) ** 3)
    for m in range(1, N + 1):
        nb = N + 1 - m
        f += 2 * (32 * nb ** 2 * ng + 10.7 * nb ** 3)
    return f


def _converge_flops(N, first=10):
    return sum(4 * (16 * (k / 2) ** 2 * 2 * k + 10.7 * (k / 2) ** 3)
               for k in range(first, N + 1))


def _average_flops(N):
    return sum(8 * (min(a, b) + 1) ** 2 for a in range(1, N + 1) for b in range(1, N + 1))


def _angle_flops(N):
    """One incoming angle: T v for both polarisations."""
    return 16 * (N * N + sum((N + 1 - m) ** 2 for m in range(1, N + 1)))


def work(case):
    kind = case["kind"]
    f, nbytes = 0.0, 0.0
    if kind in ("batch", "fixed", "grad", "plain"):
        n = case["n"]
        for i in range(16):
            x = case["xmin"] + (i + 0.5) / 16 * (case["xmax"] - case["xmin"])
            N = _order(x)
            g = _blocks_flops(N, 2 * N)
            t_bytes = 16.0 * tmatrix_size(N)
            if kind != "fixed":
                g += _converge_flops(N)
            na = case.get("ntheta", case.get("nout", 0))
            nbytes += n / 16 * 8 * (9 + 3 * na + 16 * case.get("nout", 0))
            if kind == "fixed" and na == 0:
                nbytes += n / 16 * t_bytes
            if na and (kind != "grad" or case["aligned"]):
                g += _average_flops(N)
            g += na * _angle_flops(N)
            f += n / 16 * (3 * g if kind == "grad" else g)
    elif kind == "table":
        ncell = case["nsizes"] * case["nlam"] * case["nshape"]
        for a in np.geomspace(case["rmin"], case["rmax"], case["nsizes"] + 2)[1:-1]:
            for lam in np.geomspace(case["lmin"], case["lmax"], case["nlam"] + 2)[1:-1]:
                N = _order(2 * math.pi * a / lam)
                nin = case["ntheta"] + (case["nquad"] if case["account"] else 0)
                g = (_blocks_flops(N, 2 * N) + _converge_flops(N) + _average_flops(N)
                     + nin * _angle_flops(N))
                if case["scattering"]:
                    g += 2 * case["ntheta"] ** 2 * 8 * 4 * N
                if case["account"]:
                    g += case["ntheta"] * case["nquad"] ** 2 * 8 * 4 * N
                f += case["nshape"] * g
        nout = ((2 if case["absorption"] else 0) + (3 if case["extinction"] else 0)
                + (32 * case["ntheta"] if case["scattering"] else 0))
        nbytes = 8.0 * (5 * ncell + ncell / case["nshape"] * case["ntheta"] * nout)
    else:
        N = _order(case["x"])
        f = (_blocks_flops(N, 2 * N) + _converge_flops(N) + _average_flops(N)
             + (case["nout"] + case["nabs"] + case["nquad"]) * _angle_flops(N)
             + case["nabs"] * case["nquad"] ** 2 * 8 * 4 * N)
        nbytes = 8.0 * (5 + 16 * case["nout"] + 18 * case["nabs"])
    return dict(bytes=nbytes, flops=f)


# ------------------------------------------------------------------ exact --
#
# Extended-boundary-condition T-matrices of spheroids and their observables
# in double precision with torch: full blocks, dense solves, Clebsch-Gordan
# rows as eigenvectors of J^2.

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=None)
def _nodes(ng):
    x, w = np.polynomial.legendre.leggauss(2 * ng)
    return torch.tensor(x[:ng], device=_dev()), torch.tensor(w[:ng], device=_dev())


def _wigner(x, N, m):
    """d^n_{0m} and its derivative in theta at cos(theta) = x, n = 1..N (last
    axis), by upward recurrence in n."""
    s = torch.sqrt((1 - x) * (1 + x))
    prev, cur = torch.zeros_like(x), torch.ones_like(x)
    for i in range(1, m + 1):
        cur = cur * math.sqrt((2 * i - 1) / (2 * i)) * s
    d, dd = [], []
    for n in range(m, N + 1):
        a, b = math.sqrt(n * n - m * m), math.sqrt((n + 1) ** 2 - m * m)
        nxt = ((2 * n + 1) * x * cur - a * prev) / b
        if n > 0:
            d.append(cur)
            dd.append((n * b * nxt - (n + 1) * a * prev) / ((2 * n + 1) * s))
        prev, cur = cur, nxt
    return torch.stack(d, -1), torch.stack(dd, -1)


def _bessel_j(z, N):
    """j_n and [z j_n]'/z, n = 1..N on a new last axis."""
    start = N + int(z.detach().abs().max()) + 60
    rho, ratios = z / (2 * start + 1), {}
    for k in range(start - 1, 0, -1):
        rho = 1 / ((2 * k + 1) / z - rho)
        if k <= N:
            ratios[k] = rho
    prev = torch.sin(z) / z
    j, dj = [], []
    for k in range(1, N + 1):
        cur = ratios[k] * prev
        j.append(cur)
        dj.append(prev - k * cur / z)
        prev = cur
    return torch.stack(j, -1), torch.stack(dj, -1)


def _bessel_y(z, N):
    prev, cur = -torch.cos(z) / z, -torch.cos(z) / z ** 2 - torch.sin(z) / z
    y, dy = [], []
    for k in range(1, N + 1):
        y.append(cur)
        dy.append(prev - k * cur / z)
        prev, cur = cur, (2 * k + 1) / z * cur - prev
    return torch.stack(y, -1), torch.stack(dy, -1)


class _Surface:
    """Node data and Bessel functions of grains (r, m, d) at one (N, ngauss);
    real tensors of shape [grains]."""

    def __init__(self, r, mr, mi, d, lam, N, ng):
        x, w = _nodes(ng)
        self.N, self.x = N, x
        sn = torch.sqrt((1 - x) * (1 + x))
        q = 1 / (sn ** 2 + d[:, None] ** 2 * x ** 2)
        r2 = d[:, None] ** (2 / 3) * q
        self.drr = (q * x * sn * (d[:, None] ** 2 - 1))[..., None]
        self.kr = 2 * math.pi / lam[:, None] * r[:, None] * torch.sqrt(r2)
        self.m = torch.complex(mr, mi)
        self.mkr = self.m[:, None] * self.kr
        self.wr2 = (w * r2)[..., None]
        self.sin = sn
        self.j, self.dj = _bessel_j(self.kr, N)
        self.y, self.dy = _bessel_y(self.kr, N)
        self.jm, self.djm = _bessel_j(self.mkr, N)

    def block(self, m):
        """T-matrix block m, [grains, 2 nb, 2 nb]."""
        N, lo = self.N, max(m, 1)
        n = torch.arange(lo, N + 1, device=self.x.device, dtype=torch.float64)
        nb = n.numel()
        d, dd = _wigner(self.x, N, m)
        nn = n * (n + 1)
        a = torch.sqrt((2 * n + 1) / nn)
        sl = slice(lo - 1, N)
        j, dj = self.j[..., sl], self.dj[..., sl]
        h, dh = torch.complex(j, self.y[..., sl]), torch.complex(dj, self.dy[..., sl])
        jm, djm = self.jm[..., sl], self.djm[..., sl]
        kr, mkr, mu = self.kr[..., None], self.mkr[..., None], (m / self.sin)[:, None] ** 2
        be = (m / self.sin)[:, None] * self.wr2
        G1 = d * djm * a
        G2 = (dd * djm + self.drr / mkr * nn * d * jm) * a
        G3, G4 = d * jm * a, dd * jm * a
        k = self.m[:, None, None]

        def fold(f, g):
            f = [(v * a).to(torch.complex128) for v in f]
            return sum(torch.einsum("bgi,bgj->bij", u, v) for u, v in zip(f, g))

        W11 = (k * self.wr2 * mu * G1, k * self.wr2 * G2, -self.wr2 * mu * G3,
               -self.wr2 * G4)
        W22 = (self.wr2 * mu * G1, self.wr2 * G2, -k * self.wr2 * mu * G3,
               -k * self.wr2 * G4)
        W12 = [1j * be * v for v in (k * G4, k * G3, G2, G1)]
        W21 = [1j * be * v for v in (G4, G3, k * G2, k * G1)]

        def assemble(f, df):
            F = (d * f, dd * f, d * df, dd * df + nn * self.drr / kr * d * f)
            top = torch.cat([fold(F, W11), fold(F, W12)], 2)
            return torch.cat([top, torch.cat([fold(F, W21), fold(F, W22)], 2)], 1)

        lab = torch.cat([n, n + 1]).to(torch.int64)
        mask = ((lab[:, None] + lab[None, :]) % 2 == 0).to(torch.float64)
        Rg, Q = assemble(j, dj) * mask, assemble(h, dh) * mask
        return torch.linalg.solve(Q, -Rg, left=False)


def _sums(T, N):
    """m = 0 (Qsca, Qext) from the diagonal of block 0."""
    w = 2 * torch.arange(1, N + 1, device=T.device, dtype=torch.float64) + 1
    dg = torch.diagonal(T, dim1=1, dim2=2)
    a, b = dg[:, :N], dg[:, N:]
    return ((w * (a.abs() ** 2 + b.abs() ** 2)).sum(1), (w * (a + b).real).sum(1))


def _tensors(r, m, d, lam):
    lam = np.broadcast_to(lam, r.shape)
    return [torch.tensor(np.ascontiguousarray(v), dtype=torch.float64, device=_dev())
            for v in (r, m.real, m.imag, d, lam)]


def _converge(p, tol=1e-4, first=10, last=99):
    """(orders, dQsca, dQext, Qsca, Qext) by the task-based schedule."""
    n = p[0].numel()
    order = np.zeros(n, np.int64)
    q = np.zeros((4, n))
    old = None
    active = np.arange(n)
    for k in range(first, last + 1):
        idx = torch.tensor(active, device=_dev())
        s = _Surface(*[v[idx] for v in p], k, 2 * k)
        qs, qe = (v.cpu().numpy() for v in _sums(s.block(0), k))
        order[active] = k
        q[2, active], q[3, active] = qs, qe
        done = np.zeros(len(active), bool)
        if old is not None:
            ds, de = np.abs((old[0] - qs) / qs), np.abs((old[1] - qe) / qe)
            ok = ds > 0
            q[0, active[ok]], q[1, active[ok]] = ds[ok], de[ok]
            done = ok & (ds <= tol) & (de <= tol)
        active, old = active[~done], (qs[~done], qe[~done])
        if len(active) == 0:
            break
    return order, q


def _groups(order):
    for N in np.unique(order):
        for part in np.array_split(np.flatnonzero(order == N),
                                   1 + np.sum(order == N) * int(N) ** 3 // 4000000):
            if part.size:
                yield int(N), torch.tensor(part, device=_dev())


def _full_sums(blocks, N):
    qs = qe = 0.0
    for m, T in enumerate(blocks):
        nb = T.shape[1] // 2
        f = 1 if m == 0 else 2
        qs = qs + f * (T.abs() ** 2).sum((1, 2))
        qe = qe + f * sum(torch.diagonal(T[:, i:i + nb, j:j + nb], dim1=1, dim2=2).real
                          .sum(1) for i in (0, nb) for j in (0, nb))
    return qs, qe


@functools.lru_cache(maxsize=None)
def _clebsch(n1, n2):
    """<n1 m n2 -m | N 0> for N = |n1 - n2| .. n1 + n2 (rows, up to a sign
    each) and m = 0 .. min(n1, n2): eigenvectors of J^2 in the m basis."""
    M = min(n1, n2)
    m = np.arange(-M, M + 1)
    diag = n1 * (n1 + 1) + n2 * (n2 + 1) - 2.0 * m * m
    off = np.sqrt((n1 * (n1 + 1) - m[:-1] * m[1:]) * (n2 * (n2 + 1.0) - m[:-1] * m[1:]))
    _, v = np.linalg.eigh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))
    return v.T[:, M:].copy()


def _average(blocks, N, p):
    """Orientation-averaged blocks for expansion coefficients p."""
    out = [torch.zeros_like(b) for b in blocks]
    for n1 in range(1, N + 1):
        for n2 in range(1, N + 1):
            M, lo = min(n1, n2), abs(n1 - n2)
            C = _clebsch(n1, n2)
            # T of -m is that of m up to the parity, so only the rows of one
            # parity are left, twice
            f = np.where(np.arange(M + 1) == 0, 1.0, 2.0)
            sg = (-1.0) ** np.arange(M + 1)
            pN = p[lo:lo + 2 * M + 1] * (np.arange(2 * M + 1) % 2 == (n1 + n2) % 2)
            K = torch.tensor((sg[:, None] * (C.T * pN)) @ (C * (f * sg)),
                             dtype=torch.complex128, device=_dev())
            for i1 in (0, 1):
                for i2 in (0, 1):
                    if (n1 + i1 + n2 + i2) % 2:
                        continue
                    at = [(slice(None), i1 * (b.shape[1] // 2) + n1 - max(m, 1),
                           i2 * (b.shape[1] // 2) + n2 - max(m, 1))
                          for m, b in enumerate(blocks[:M + 1])]
                    t = torch.stack([b[i] for b, i in zip(blocks, at)], 1)
                    for m, (i, v) in enumerate(zip(at, (t @ K.T).unbind(1))):
                        out[m][i] = v
    return out


def _angular(cost, N, m):
    """(pi, tau) = (m d / sin, d') for n = max(m, 1) .. N, [angles, n]."""
    poles = torch.abs(1 - cost.abs()) <= 1e-10
    c = torch.where(poles, torch.zeros_like(cost), cost)
    d, dd = _wigner(c, N, m)
    p, t = m * d / torch.sqrt((1 - c) * (1 + c))[:, None], dd
    n = torch.arange(max(m, 1), N + 1, device=cost.device, dtype=torch.float64)
    lim = 0.5 * torch.sqrt(n * (n + 1)) * (1 if m == 1 else 0)
    alt = torch.where(n.to(torch.int64) % 2 == 0, -1.0, 1.0)
    up = (cost > 0)[:, None]
    return (torch.where(poles[:, None], torch.where(up, lim, lim * alt), p),
            torch.where(poles[:, None], torch.where(up, lim, -lim * alt), t))


def _amplitudes(blocks, N, k, cin, cout, eiphi, pairwise=False):
    """2 x 2 amplitudes S for incoming cosines cin, outgoing cosines cout and
    azimuth factors eiphi: [grains, in, out, phi, 4], or [grains, in, phi, 4]
    for pairs (cin[i], cout[i])."""
    S = 0
    n0 = torch.arange(1, N + 1, device=_dev())
    turns = torch.tensor([1, 1j, -1, -1j], dtype=torch.complex128, device=_dev())
    for m, T in enumerate(blocks):
        n = n0[max(m, 1) - 1:]
        nf = n.to(torch.float64)
        a = torch.sqrt((2 * nf + 1) / (nf * (nf + 1)))
        c = turns[(n[None, :] - n[:, None] - 1) % 4] * (a[:, None] * a[None, :])
        Tc = T * c.repeat(2, 2)
        pi, ti = _angular(cin, N, m)
        po, to = _angular(cout, N, m)
        v = [torch.cat([x, y], 1).to(torch.complex128) for x, y in ((pi, ti), (ti, pi))]
        u = [torch.cat([x, y], 1).to(torch.complex128) for x, y in ((po, to), (to, po))]
        e = eiphi ** m
        f = (2.0 if m else 1.0) * e.real
        g = (2.0 if m else 0.0) * e.imag
        fac = torch.stack([f, g, -g, f], 1)
        sub = "ax,bxy,ay->ba" if pairwise else "ox,bxy,ay->bao"
        X = torch.stack([torch.einsum(sub, uu, Tc, vv) for uu in u for vv in v], -1)
        S = S + X[..., None, :] * fac
    return S / k.reshape((-1,) + (1,) * (S.dim() - 1))


def _extinction(S, k, r):
    f = 2 / (k * r * r)
    a, b = S[..., 0, 0], S[..., 0, 3]
    return torch.stack([(a + b).imag, (a - b).imag, (b - a).real], -1) * f[:, None, None]


def _mueller(S):
    """4 x 4 scattering matrix of (S11, S12, S21, S22)."""
    a, b, c, d = S.unbind(-1)
    x = lambda u, v: u * v.conj()  # noqa: E731
    aa, bb, cc, dd = (v.abs() ** 2 for v in (a, b, c, d))
    rows = [0.5 * (aa + bb + cc + dd), 0.5 * (aa - bb + cc - dd),
            -(x(a, b) + x(d, c)).real, -(x(a, b) - x(d, c)).imag,
            0.5 * (aa + bb - cc - dd), 0.5 * (aa - bb - cc + dd),
            (x(d, c) - x(a, b)).real, -(x(a, b) + x(d, c)).imag,
            -(x(a, c) + x(d, b)).real, (x(d, b) - x(a, c)).real,
            (x(a, d) + x(b, c)).real, (x(a, d) + x(c, b)).imag,
            -(x(c, a) + x(d, b)).imag, -(x(c, a) - x(d, b)).imag,
            (x(d, a) - x(b, c)).imag, (x(d, a) - x(b, c)).real]
    return torch.stack(rows, -1).reshape(S.shape[:-1] + (4, 4))


def _cos(theta):
    return torch.tensor(np.cos(np.asarray(theta, float)), device=_dev())


def _one():
    return torch.ones(1, dtype=torch.complex128, device=_dev())


def _exact_batch(case, seed):
    r, m, d = _grains(case["n"], seed, case["xmin"], case["xmax"])
    p = _tensors(r, m, d, LAM)
    order, dq = _converge(p)
    q = np.zeros((case["n"], 6))
    q[:, 0], q[:, 1], q[:, 4], q[:, 5] = dq[2], dq[3], dq[0], dq[1]
    for N, idx in _groups(order):
        s = _Surface(*[v[idx] for v in p], N, 2 * N)
        qs, qe = _full_sums([s.block(k) for k in range(N + 1)], N)
        at = idx.cpu().numpy()
        q[at, 2], q[at, 3] = qs.cpu().numpy(), qe.cpu().numpy()
    return dict(nmax=None, ngauss=None, status=None, q=q)


def _exact_fixed(case, seed):
    (r, m, d), order = _fixed_grains(case, seed)
    p = _tensors(r, m, d, LAM)
    q = np.zeros((case["n"], 2))
    T = [None] * case["n"]
    obs = np.zeros((case["n"], case["ntheta"], 3))
    coeffs = _random_orientation(2 * 64)
    th = _cos(_thetas(case["ntheta"]))
    for N, idx in _groups(order):
        sub = [v[idx] for v in p]
        s = _Surface(*sub, N, 2 * N)
        blocks = [s.block(k) for k in range(N + 1)]
        at = idx.cpu().numpy()
        qs, qe = _full_sums(blocks, N)
        q[at, 0], q[at, 1] = qs.cpu().numpy(), qe.cpu().numpy()
        if not case["ntheta"]:
            flat = torch.cat([b.reshape(len(at), -1) for b in blocks], 1).cpu().numpy()
            for i, row in zip(at, flat):
                T[i] = row
            continue
        k = 2 * math.pi / sub[4]
        S = _amplitudes(_average(blocks, N, coeffs), N, k, th, th, _one(), True)
        obs[at] = _extinction(S, k, sub[0]).cpu().numpy()
    return dict(status=None, q=q, **(dict(obs=obs) if case["ntheta"] else dict(T=T)))


def _exact_grad(case, seed):
    if case["n"] > 64:
        return None
    s = prepare(case, seed)
    base = s["params"].detach().to(_dev())
    lam = torch.full((case["n"],), LAM, dtype=torch.float64, device=_dev())
    order, _ = _converge([base[:, 2], base[:, 0], base[:, 1], base[:, 3], lam])
    q = np.zeros((case["n"], case["ntheta"], 3))
    grad = np.zeros((case["n"], 4))
    th = _cos(s["thetas"])
    for N, idx in _groups(order):
        x = base[idx].clone().requires_grad_(True)
        surf = _Surface(x[:, 2], x[:, 0], x[:, 1], x[:, 3], lam[idx], N, 2 * N)
        blocks = [surf.block(k) for k in range(N + 1)]
        if case["aligned"]:
            blocks = _average(blocks, N, s["coeffs"])
        k = 2 * math.pi / lam[idx]
        out = _extinction(_amplitudes(blocks, N, k, th, th, _one(), True), k, x[:, 2])
        at = idx.cpu().numpy()
        (out * s["upstream"].to(_dev())[idx]).sum().backward()
        q[at], grad[at] = out.detach().cpu().numpy(), x.grad.cpu().numpy()
    return dict(q=q, grad=grad)


def _gauss(n, a, b):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (b - a) * x + 0.5 * (b + a), 0.5 * (b - a) * w


def _exact_table(case, seed):
    if case["nsizes"] * case["nlam"] * case["nshape"] > 300:
        return None
    sizes, lams = (np.sort(v) for v in _grid(case, seed))
    sh = _shapes(case["nshape"])
    al = _alignment(case["alignment"], 100)
    i, j, s = (v.ravel() for v in np.meshgrid(np.arange(sizes.size),
               np.arange(lams.size), np.arange(len(sh.shapes)), indexing="ij"))
    m = np.array([_dielectric(w) for w in lams])[j]
    p = _tensors(sizes[i], m, np.asarray(sh.shapes)[s], lams[j])
    order, _ = _converge(p)
    thetas = _thetas(case["ntheta"])
    th, nt = _cos(thetas), case["ntheta"]
    q = np.zeros((i.size, nt, 5))
    Z = np.zeros((i.size, nt, 2 * nt, 4, 4)) if case["scattering"] else None
    for N, idx in _groups(order):
        sub = [v[idx] for v in p]
        surf = _Surface(*sub, N, 2 * N)
        blocks = [surf.block(k) for k in range(N + 1)]
        at = idx.cpu().numpy()
        sets = {}
        for row, g in enumerate(at):
            dist = al.get_distribution(sizes[i[g]], sh.shapes[s[g]])
            sets.setdefault(id(dist), (dist, []))[1].append(row)
        for dist, rows in sets.values():
            part = [b[rows] for b in blocks]
            if dist.compute_alignment:
                part = _average(part, N, dist.coefficients)
            k, r = 2 * math.pi / sub[4][rows], sub[0][rows]
            ext = _extinction(_amplitudes(part, N, k, th, th, _one(), True), k, r)
            absn = ext[..., :2].clone()
            if case["account"]:
                cx, cw = np.polynomial.legendre.leggauss(case["nquad"])
                ph, pw = _gauss(case["nquad"], 0, 2 * np.pi)
                S = _amplitudes(part, N, k, torch.tensor(cx, device=_dev()), th,
                                torch.tensor(np.exp(-1j * ph), device=_dev()))
                a = (S.abs() ** 2) * 0.5
                wt = torch.tensor(cw[:, None, None] * pw, device=_dev())
                norm = (math.pi * r * r)[:, None]
                absn[..., 0] -= (a.sum(-1) * wt).sum((1, 3)) / norm
                absn[..., 1] -= ((a[..., 0] + a[..., 1] - a[..., 2] - a[..., 3])
                                 * wt).sum((1, 3)) / norm
            q[at[rows]] = torch.cat([absn, ext], -1).cpu().numpy()
            if case["scattering"]:
                cx, _ = np.polynomial.legendre.leggauss(nt)
                ph, _ = _gauss(2 * nt, 0, 2 * np.pi)
                S = _amplitudes(part, N, k, torch.zeros(1, dtype=torch.float64, device=_dev()),
                                torch.tensor(cx, device=_dev()),
                                torch.tensor(np.exp(1j * ph), device=_dev()))
                Z[at[rows]] = _mueller(S[:, 0]).cpu().numpy()
    w = np.asarray(sh.weights) / np.sum(sh.weights)

    def mean(v):
        v = v.reshape((1, sizes.size, lams.size, w.size) + v.shape[1:])
        return np.squeeze(np.tensordot(v, w, axes=([3], [0])))

    cols = ([0, 1] if case["absorption"] else []) + ([2, 3, 4] if case["extinction"] else [])
    out = []
    if cols:
        out.append(mean(q[..., cols]))
    if case["scattering"]:
        out.append(mean(Z))
    return out + [None]


def _exact_particle(case, seed):
    s = prepare(case, seed)
    p = _tensors(np.array([s["r"]]), np.array([s["m"]]), np.array([case["d"]]), LAM)
    x = 2 * math.pi * s["r"] / LAM
    N = int(max(4.0, x + 4.05 * x ** (1 / 3)))
    tol, old = 1e-4, None

    def moves(N, ng):  # whether the m = 0 sums still change from step to step
        nonlocal old
        qs, qe = (float(v[0]) for v in _sums(_Surface(*p, N, ng).block(0), N))
        last, old = old, (qs, qe)
        return last is None or abs((last[0] - qs) / qs) > tol or \
            abs((last[1] - qe) / qe) > tol

    while moves(N, 2 * N):
        N += 1
    ng = 2 * N + 1
    while moves(N, ng):
        ng += 1
    surf = _Surface(*p, N, ng)
    blocks = _average([surf.block(k) for k in range(N + 1)], N,
                      _random_orientation(2 * N))
    k = 2 * math.pi / p[4]
    S = _amplitudes(blocks, N, k, _cos([0.3]), _cos(s["out"]), _one() * np.exp(0.5j))
    th = _cos(s["abs"])
    F = _amplitudes(blocks, N, k, th, th, _one(), True)[0, :, 0]
    pf = 2 * math.pi / k
    K = torch.zeros(F.shape[0], 4, 4, dtype=torch.float64, device=_dev())
    for i in range(4):
        K[:, i, i] = pf * (F[:, 0] + F[:, 3]).imag
    K[:, 0, 1] = K[:, 1, 0] = pf * (F[:, 0] - F[:, 3]).imag
    K[:, 2, 3] = pf * (F[:, 3] - F[:, 0]).real
    K[:, 3, 2] = -K[:, 2, 3]
    cx, cw = np.polynomial.legendre.leggauss(case["nquad"])
    ph, pw = _gauss(case["nquad"], 0, 2 * np.pi)
    A = _amplitudes(blocks, N, k, torch.tensor(cx, device=_dev()), th,
                    torch.tensor(np.exp(-1j * ph), device=_dev()))[0].abs() ** 2 * 0.5
    wt = torch.tensor(cw[:, None, None] * pw, device=_dev())
    C = torch.stack([K[:, 0, 0] - (A.sum(-1) * wt).sum((0, 2)),
                     K[:, 0, 1] - ((A[..., 0] + A[..., 1] - A[..., 2] - A[..., 3])
                                   * wt).sum((0, 2))], 1)
    return dict(order=None, ngauss=None, Z=np.squeeze(_mueller(S[0, 0, :, 0]).cpu().numpy()),
                K=np.squeeze(K.cpu().numpy()), C=np.squeeze(C.cpu().numpy()))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "fixed":
        return _exact_fixed(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "table":
        return _exact_table(case, seed)
    if kind == "particle":
        return _exact_particle(case, seed)
    # some grains of the plain batch do not converge and run to order 200: no
    # plain evaluation in a few seconds
    return None
