"""Timed cases of the boost-factor solvers: what users of the package run, by use.

The families, each through the package's public API:

  propagate    one call of a `prop=` propagator on a host field (the drop-in for
               code that runs its own bounce loop): the smallest call there is
  dancer       the legacy bounce loop (one-shot call or resident stack)
  cheerleader  the current bounce loop (one-shot call, resident stack with host
               fields, or with the fields left on the device)
  transformer  mode matching, one-shot drop-in call
  step         one optimiser step: a resident stack moved and solved by the server
  group        one step of several optimisers of one booster design at once
  pgrid        one optimiser cost on an interpolated propagation-matrix grid
  batch1d      the 1D model for many spacing configurations

A resident solver's pass moves the disks first (`set_distance`, or the request's
`distance`), as every step of an optimiser does.  Mixed-precision solves compute
in single precision, and their results are kept in single precision here, as a
program that asks for them would.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "boostfractor.jl_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

C0 = 299792458.0


def listed():
    return [
        # the reference's default 101 x 101 grid, one propagation with a tilted, rough disk
        dict(name="propagate-101", kind="propagate", n=101, prop="propagator", precision="fp64", rough=True),
        # the reference's CPU-runnable case: one disk, 64 x 64, one frequency per call
        dict(name="dancer-64-1f", kind="dancer", n=64, ndisk=1, eps=24.0, nf=1, nmax=200, precision="fp64",
             how="oneshot", tilts=False),
        # the single-disk notebook: default odd grid, eps 9, part of its frequency sweep as one batch
        dict(name="cheerleader-101-32f", kind="cheerleader", n=101, ndisk=1, eps=9.0, nf=32, nmax=100,
             precision="fp64", how="oneshot", tilts=False),
        # a small tilted booster at an odd number of frequencies, the exit fields to the host
        dict(name="cheerleader-64-37f", kind="cheerleader", n=64, ndisk=5, eps=9.4, nf=37, nmax=100,
             precision="mixed", how="host", tilts=True),
        # the headline booster, 20 tilted disks at 256 frequencies, for the solver's default number of bounces; the
        # fields stay on the device
        dict(name="cheerleader-128-256f", kind="cheerleader", n=128, ndisk=20, eps=24.0, nf=256, nmax=100,
             precision="mixed", how="device", tilts=True),
        # a dancer of the uneven batch's larger grid
        dict(name="dancer-256-64f", kind="dancer", n=256, ndisk=12, eps=9.4, nf=64, nmax=100, precision="mixed",
             how="host", tilts=False),
        # the 20-disk notebook: 51 x 51, 28 Bessel modes, 29 frequencies, double precision
        dict(name="transformer-51-28m", kind="transformer", n=51, ndisk=20, eps=24.0, nf=29, M=4, L=3,
             precision="fp64", rough=False),
        # one interactive optimiser step: 8 modes, 256 frequencies
        dict(name="step-128-8m-256f", kind="step", n=128, ndisk=20, eps=24.0, nf=256, M=8, rough=False),
        # sixteen optimisers of one design stepping together
        dict(name="group-128-8m-16x256f", kind="group", n=128, ndisk=20, eps=24.0, nf=256, M=8, nreq=16),
        # the large spectrum: 64 modes, rough disks on a 256 x 256 grid, 1024 frequencies
        dict(name="step-256-64m-1024f", kind="step", n=256, ndisk=20, eps=24.0, nf=1024, M=64, rough=True),
        # one cost evaluation of an optimiser on interpolated matrices
        dict(name="pgrid-128-8m-256f", kind="pgrid", n=128, ndisk=20, eps=24.0, nf=256, M=8, nsp=9),
        # 4096 spacing configurations of the 20-disk booster in the 1D limit
        dict(name="batch1d-4096x256", kind="batch1d", ndisk=20, eps=24.0, nconf=4096, nf=256),
    ]


# --------------------------------------------------------------------------
# drawing
# --------------------------------------------------------------------------
def _logint(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _grid(rng, lo, hi):
    """Half powers of two (what large solves use), half any size, odd ones among them."""
    if rng.random() < 0.5:
        return rng.choice([n for n in (32, 64, 128, 256) if lo <= n <= hi])
    return _logint(rng, lo, hi)


def _props(kind, ndisk, nmax):
    """Propagations of one frequency's bounce loop."""
    nd = 2 * ndisk + 2
    return (nmax + 1) * 2 * (nd - 1 if kind == "dancer" else nd - 2) + (0 if kind == "dancer" else nd - 2)


def draw(rng):
    kind = rng.choice(["propagate", "dancer", "cheerleader", "cheerleader", "transformer", "step", "group", "pgrid",
                       "batch1d"])
    eps = rng.choice([9.0, 9.4, 24.0])
    if kind == "propagate":
        prop = rng.choice(["propagator", "propagatorNoTilts", "propagatorMomentumSpace"])
        return dict(kind=kind, n=_grid(rng, 32, 256), prop=prop, precision=rng.choice(["fp64", "mixed"]),
                    rough=prop == "propagator" and rng.random() < 0.5)
    if kind in ("dancer", "cheerleader"):
        precision = rng.choice(["fp64", "mixed", "mixed"])
        n, ndisk = _grid(rng, 48, 256), _logint(rng, 1, 24)
        nmax = _logint(rng, 20, 400 if precision == "fp64" else 80)
        # about 0.3 s of propagations: grids that are no power of two are the dear ones
        if n & (n - 1):
            rate = 1.5e10 / n ** 3
        else:
            rate = (1.5e7 if precision == "mixed" else 1.5e6) * (128 / n) ** 2
        most = 0.3 * rate
        nmax = max(5, min(nmax, int(most / _props(kind, ndisk, 0))))
        ndisk = max(1, min(ndisk, int(most / _props(kind, 1, nmax))))
        nf = _logint(rng, 1, max(1, min(256, int(most / _props(kind, ndisk, nmax)))))
        return dict(kind=kind, n=n, ndisk=ndisk, eps=eps, nf=nf, nmax=nmax, precision=precision,
                    how=rng.choice(["oneshot", "host"] + (["device"] if kind == "cheerleader" else [])),
                    tilts=rng.random() < 0.5)
    if kind == "transformer":
        M, L = rng.choice([(4, 3), (5, 0), (10, 0), (3, 1), (6, 2)])
        precision = rng.choice(["fp64", "mixed"])
        n = _grid(rng, 48, 128)
        ndisk = _logint(rng, 1, 24)
        nm = M * (2 * L + 1)
        most = (2e11 if precision == "fp64" else 2e12) / (8 * nm * nm * n * n / 8 * 2 * ndisk)
        return dict(kind=kind, n=n, ndisk=ndisk, eps=eps, nf=_logint(rng, 1, max(1, min(512, int(most)))), M=M, L=L,
                    precision=precision, rough=rng.random() < 0.3)
    if kind in ("step", "group", "pgrid"):
        M = _logint(rng, 1, 64 if kind == "step" else 24)
        n, ndisk = _grid(rng, 48, 256 if kind == "step" else 128), _logint(rng, 2, 40 if kind == "step" else 20)
        case = dict(kind=kind, n=n, ndisk=ndisk, eps=eps, M=M)
        if kind == "step":
            case.update(nf=_logint(rng, 16, 1024 if M <= 32 and ndisk <= 20 else 256), rough=rng.random() < 0.3)
        elif kind == "group":
            case.update(nf=_logint(rng, 16, 256), nreq=rng.randint(2, 16))
        else:
            case.update(nf=_logint(rng, 16, 256), nsp=rng.choice([5, 9, 12]))
        return case
    return dict(kind=kind, ndisk=_logint(rng, 1, 40), eps=eps, nconf=_logint(rng, 1, 4096), nf=_logint(rng, 1, 256))


# --------------------------------------------------------------------------
# inputs, from the seed alone
# --------------------------------------------------------------------------
def _axis(n):
    """n points over 1 m, antisymmetric about 0."""
    i = np.arange(n, dtype=np.float64)
    return (2 * i - (n - 1)) / (2.0 * (n - 1))


def _inputs(case, seed):
    """The booster (regions mirror, gap, disk, ..., gap, disk, exit) and what else a case takes, as host arrays."""
    rng = np.random.default_rng([seed, 20240521])
    kind, ndisk = case["kind"], case.get("ndisk", 1)
    g = dict(rng=rng, diskR=0.15, freqs=np.linspace(19.5e9, 20.5e9, case.get("nf", 1)) + rng.uniform(0, 1e6))
    nd = 2 * ndisk + 2
    g["distance"], g["eps"] = np.zeros(nd), np.ones(nd, dtype=np.complex128)
    g["eps"][0] = np.nan
    g["eps"][2:-1:2] = case.get("eps", 9.0)
    g["distance"][1:-1:2] = rng.uniform(7.5e-3, 8.5e-3, ndisk)
    g["distance"][2:-1:2] = 1e-3
    g["tx"], g["ty"] = np.zeros(nd), np.zeros(nd)
    if case.get("tilts"):
        g["tx"][2:-1:2], g["ty"][2:-1:2] = rng.uniform(-5e-4, 5e-4, (2, ndisk))
    # the step that an optimiser takes from there
    g["moved"] = g["distance"].copy()
    g["moved"][1:-1:2] += rng.normal(0.0, 10e-6, ndisk)
    if "n" in case:
        g["X"] = _axis(case["n"])
    g["surf"] = _rough(g["X"], nd, rng, g["diskR"]) if case.get("rough") else None
    if kind == "propagate":
        n = case["n"]
        r2 = g["X"][:, None] ** 2 + g["X"][None, :] ** 2
        g["E"] = np.exp(-r2 / 0.1 ** 2) * (1 + 0.1 * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))))
        g["dz"], g["lam"] = rng.uniform(7.5e-3, 8.5e-3), C0 / 20e9
        g["tilt"] = rng.uniform(-5e-4, 5e-4, 2)
    if kind == "group":
        g["all"] = np.repeat(g["distance"][None], case["nreq"], 0)
        g["all"][:, 1:-1:2] += rng.normal(0.0, 50e-6, (case["nreq"], ndisk))
    if kind == "pgrid":
        g["grid"] = np.linspace(-2e-4, 2e-4, case["nsp"])
        g["shift"] = np.clip(rng.normal(0.0, 4e-5, ndisk), -1e-4, 1e-4)
        g["antenna"] = rng.normal(size=case["M"]) + 1j * rng.normal(size=case["M"])
    if kind == "batch1d":
        g["confs"] = np.repeat(g["distance"][None], case["nconf"], 0)
        g["confs"][:, 1:-1:2] += rng.normal(0.0, 10e-6, (case["nconf"], ndisk))
    return g


def _rough(X, nd, rng, diskR):
    """Surface maps of the disks: white noise of 10 um smoothed over 2 cm, zero off the disk."""
    n = len(X)
    out = np.zeros((nd, n, n))
    d = X[:, None] ** 2 + X[None, :] ** 2
    k = np.fft.fftfreq(n, X[1] - X[0]) * 2 * np.pi
    smooth = np.exp(-(k[:, None] ** 2 + k[None, :] ** 2) * 0.02 ** 2 / 4)
    for j in range(2, nd - 1, 2):
        s = np.fft.ifft2(np.fft.fft2(rng.standard_normal((n, n))) * smooth).real
        out[j] = np.where(d <= diskR ** 2, np.clip(s * (1e-5 / np.sqrt(np.mean(s ** 2))), -1e-4, 1e-4), 0.0)
    return out


def _lg(X, count, diskR, waist=0.03):
    """The `count` lowest Laguerre-Gauss modes LG_p^l exp(-i l phi), cut to the disk and normalised, and their
    transverse wavenumbers 2 sqrt(2p + |l| + 1) / waist."""
    r2 = X[:, None] ** 2 + X[None, :] ** 2
    phi = np.arctan2(*np.broadcast_arrays(X[None, :], X[:, None]))
    u = 2.0 * r2 / waist ** 2
    pats, kt, order = [], [], 0
    while len(pats) < count:
        for l in range(-order, order + 1, 2):
            p, a = (order - abs(l)) // 2, abs(l)
            poly = sum((-1) ** i * math.comb(p + a, p - i) / math.factorial(i) * u ** i for i in range(p + 1))
            f = u ** (a / 2) * poly * np.exp(-u / 2) * np.exp(-1j * l * phi)
            f[np.sqrt(r2) > diskR] = 0.0
            pats.append(f / np.sqrt(np.sum(np.abs(f) ** 2)))
            kt.append(2.0 * math.sqrt(order + 1.0) / waist)
        order += 1
    return np.array(pats[:count]), np.array(kt[:count], dtype=np.complex128)


# --------------------------------------------------------------------------
# prepare and run: the package
# --------------------------------------------------------------------------
class _Server:
    """A server and what it serves, closed in the order that the server wants."""

    def __init__(self, B, handle, stack, modes):
        self.handle, self.stack, self.modes = handle, stack, modes
        self.server = B.Server(n_workers=1)

    def __del__(self):
        for part in (self.server, self.stack, self.modes, self.handle):
            part.close()


def prepare(case, seed):
    import bfgb300 as B
    g, kind = _inputs(case, seed), case["kind"]
    s = dict(B=B, kind=kind, case=case, g=g)
    if kind == "batch1d":
        return s
    s["coords"] = B.SeedCoordinateSystem(X=g["X"], Y=g["X"])
    if kind == "propagate":
        s["surface"] = None if g["surf"] is None else g["surf"][2]
        return s
    bdry = B.SeedSetupBoundaries(s["coords"], diskno=case["ndisk"], distance=g["distance"], epsilon=g["eps"],
                                 relative_tilt_x=g["tx"], relative_tilt_y=g["ty"], relative_surfaces=g["surf"])
    s["bdry"] = bdry
    if kind in ("dancer", "cheerleader"):
        if case["how"] != "oneshot":
            s["stack"] = B.Stack(bdry, s["coords"], g["diskR"])
        if case["how"] == "device":
            n, nf = case["n"], case["nf"]
            s["right"] = torch.empty(nf, n, n, dtype=torch.complex128, device="cuda")
            s["beta2"] = torch.empty(nf, dtype=torch.float64, device="cuda")
        return s
    bdry.eps[np.isnan(bdry.eps)] = 1e30   # as the transformer call itself does
    if kind == "transformer":
        s["modes"] = B.SeedModes(s["coords"], ThreeDim=True, Mmax=case["M"], Lmax=case["L"], diskR=g["diskR"])
        return s
    h = B.Handle(0)
    pats, kt = _lg(g["X"], case["M"], g["diskR"])
    modes = B.SeedModes(s["coords"], ThreeDim=True, Mmax=case["M"], Lmax=0, diskR=g["diskR"],
                        pattern_input=pats[:, None, :, :, None], kT_arr=kt[:, None], handle=h)
    s["modes"], s["handle"] = modes, h
    if kind == "step":
        s["service"] = _Server(B, h, B.Stack(bdry, s["coords"], g["diskR"], handle=h), modes)
    elif kind == "group":
        s["stacks"] = [B.Stack(bdry, s["coords"], g["diskR"], handle=h) for _ in range(case["nreq"])]
    else:
        s["pgrid"] = B.PGrid(bdry, s["coords"], modes, g["freqs"], g["grid"], diskR=g["diskR"], precision="mixed")
    return s


def _single(case, *out):
    """Results in the precision they were computed in."""
    if case.get("precision", "mixed") == "fp64":
        return list(out)
    to = {np.dtype("c16"): np.complex64, np.dtype("f8"): np.float32}
    return [o.astype(to[o.dtype]) for o in out]


def run(s):
    B, g, case = s["B"], s["g"], s["case"]
    kind, precision = s["kind"], case.get("precision", "mixed")
    if kind == "propagate":
        E = getattr(B, case["prop"])(g["E"], g["dz"], g["diskR"], 1.0, g["tilt"][0], g["tilt"][1], s["surface"],
                                     g["lam"], s["coords"], precision=precision)
        return _single(case, E)
    if kind in ("dancer", "cheerleader"):
        if case["how"] == "oneshot":
            solve = B.dancer if kind == "dancer" else B.cheerleader
            return _single(case, solve(0, case["nmax"], s["bdry"], s["coords"], f=g["freqs"], diskR=g["diskR"],
                                       precision=precision))
        s["stack"].set_distance(g["moved"])
        if kind == "dancer":
            return _single(case, *s["stack"].dancer(g["freqs"], nmax=case["nmax"], precision=precision))
        if case["how"] == "host":
            right, _, beta2 = s["stack"].cheerleader(g["freqs"], nmax=case["nmax"], precision=precision)
            return _single(case, right, beta2)
        s["stack"].cheerleader_device(g["freqs"], s["right"].data_ptr(), s["beta2"].data_ptr(), nmax=case["nmax"],
                                      precision=precision)
        if precision == "fp64":
            return [s["right"], s["beta2"]]
        return [s["right"].to(torch.complex64), s["beta2"].to(torch.float32)]
    if kind == "transformer":
        return _single(case, B.transformer(s["bdry"], s["coords"], s["modes"], f=g["freqs"], diskR=g["diskR"],
                                           precision=precision))
    if kind == "step":
        v = s["service"]
        r = v.server.wait(v.server.submit(v.stack, g["freqs"], solver="transformer", modes=v.modes,
                                          distance=g["moved"], want_boost=True))
        return _single(case, r["boost"], r["beta2"])
    if kind == "group":
        for st, d in zip(s["stacks"], g["all"]):
            st.set_distance(d)
        beta2, boost = B.transformer_group(s["stacks"], s["modes"], g["freqs"], want_boost=True)
        return _single(case, boost, beta2)
    if kind == "pgrid":
        cost, coupled = s["pgrid"].cost(g["shift"], g["antenna"])
        return _single(case, np.array([cost]), coupled)
    boost, beta2 = B.transformer_1d_batch(g["confs"], g["eps"], g["freqs"])
    return [boost, beta2]


def work(case):
    """Bytes of inputs and outputs, and the flops of the propagations (two transforms each) or of the dense algebra."""
    kind, n, nf, ndisk = case["kind"], case.get("n", 1), case.get("nf", 1), case.get("ndisk", 1)
    nd = 2 * ndisk + 2
    if kind == "propagate":
        return dict(bytes=32.0 * n * n, flops=2 * 5.0 * n * n * math.log2(n * n))
    if kind in ("dancer", "cheerleader"):
        return dict(bytes=16.0 * nf * n * n,
                    flops=nf * _props(kind, ndisk, case["nmax"]) * 2 * 5.0 * n * n * math.log2(n * n))
    if kind == "batch1d":
        return dict(bytes=8.0 * case["nconf"] * nd + 24.0 * case["nconf"] * nf,
                    flops=60.0 * case["nconf"] * nf * (nd - 1))
    nm = case["M"] * (2 * case.get("L", 0) + 1)
    nreq = case.get("nreq", 1)
    chain = nreq * nf * ((nd - 1) * 8.0 * (2 + 1) * nm ** 3 + 8.0 * nm ** 3 / 3)
    if kind == "pgrid":   # four spline coefficients per matrix entry
        return dict(bytes=16.0 * nf * nm * nm * ((ndisk + 1) * 4 + ndisk), flops=chain)
    # overlaps of the upper triangle of mode pairs: an eighth of the k-grid for the gaps, the disk's pixels for the disks
    overlap = nf * 4.0 * nm * (nm + 1) * n * n * ((ndisk + 1) * nreq / 8 + ndisk * math.pi * 0.15 ** 2)
    return dict(bytes=16.0 * nm * n * n + 24.0 * nreq * nf * nm, flops=chain + overlap)


# --------------------------------------------------------------------------
# the same in 64 bits, from the formulas, in plain torch
# --------------------------------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV)


def _k0(eps, freqs):
    """2 pi sqrt(eps) / lambda with real eps taken as eps - 0i."""
    e = complex(eps)
    return 2 * np.pi * freqs / C0 * np.sqrt(complex(e.real, -0.0 if e.imag == 0 else e.imag))


def _kaxis(X):
    n = len(X)
    dk = 2 * np.pi / (2 * X.max())
    return (np.arange(n) - (n - 1) / 2) * dk


def _kz(eps, freqs, X):
    """sqrt(k0^2 - kx^2 - ky^2) per frequency on the shifted k-grid, evanescent bins decaying."""
    k0 = _t(_k0(eps, freqs))[:, None, None]
    k2 = _t(_kaxis(X) ** 2)
    q = k0 * k0 - (k2[:, None] + k2[None, :])
    r = torch.sqrt(q)
    return torch.where((q.imag == 0) & (q.real < 0), torch.complex(torch.zeros_like(r.real), -r.abs()), r)


def _phasor(eps, dz, freqs, X):
    """exp(-i kz dz) in the order of fft2's bins."""
    n = len(X)
    return torch.roll(torch.exp(-1j * _kz(eps, freqs, X) * dz), (-(n // 2), -(n // 2)), (1, 2))


def _map(eps, tx, ty, surf, freqs, X):
    """The tilt and surface factor of a region, or None."""
    if tx == 0 and ty == 0 and (surf is None or not surf.any()):
        return None
    path = tx * X[:, None] + ty * X[None, :] + (0.0 if surf is None else surf)
    return torch.exp(-1j * _t(_k0(eps, freqs))[:, None, None] * _t(path))


def _mask(X, R):
    return _t((np.abs(X[:, None] ** 2 + X[None, :] ** 2) < R ** 2).astype(np.float64))


class _Prop:
    def __init__(self, g, regions):
        X, f = g["X"], g["freqs"]
        self.mask = _mask(X, g["diskR"])
        self.D, self.M = {}, {}
        for j in regions:
            self.D[j] = _phasor(g["eps"][j], g["use"][j], f, X)
            self.M[j] = _map(g["eps"][j], g["tx"][j], g["ty"][j], None if g["surf"] is None else g["surf"][j], f, X)

    def __call__(self, j, E):
        E = torch.fft.ifft2(torch.fft.fft2(E * self.mask) * self.D[j])
        return E if self.M[j] is None else E * self.M[j]


def _emission(g):
    """Right- and left-moving amplitudes of the field that the axions induce at the sides of region 1, 2, ..."""
    eps = [complex(e) for e in g["eps"][1:]]
    amp = lambda a, b: (1 - b / a) * np.sqrt(a) / (a * np.sqrt(b) + b * np.sqrt(a))   # noqa: E731
    right = [-1.0] + [amp(eps[i], eps[i - 1]) for i in range(1, len(eps))]
    left = [amp(eps[i], eps[i + 1] if i + 1 < len(eps) else 1.0) for i in range(len(eps))]
    r = [1.0] + [(np.sqrt(a) - np.sqrt(b)) / (np.sqrt(a) + np.sqrt(b)) for a, b in zip(eps[:-1], eps[1:])]
    X = g["X"]
    disk = _t((X[:, None] ** 2 + X[None, :] ** 2 <= g["diskR"] ** 2).astype(np.complex128))
    return right, left, [complex(v) for v in r], disk


def _exact_cheerleader(g, nmax):
    nd, nf = len(g["eps"]), len(g["freqs"])
    p = _Prop(g, range(1, nd - 1))
    right, left, r, disk = _emission(g)
    n = disk.shape[0]
    F = [None] + [(right[j - 1] * disk).expand(nf, n, n) for j in range(1, nd)]
    for i in range(1, nd - 1):
        F[i] = p(i, F[i])
        F[i + 1] = F[i + 1] + (1 + r[i]) * F[i]
        F[i] = F[i] * r[i]
    for j in range(1, nd - 1):
        F[j] = F[j] + left[j - 1] * disk
    last = nd - 2
    F[last] = F[last] + (1 - r[last]) * left[-1] * disk
    F[last + 1] = F[last + 1] - r[last] * left[-1] * disk
    for _ in range(nmax + 1):
        F[1] = p(1, F[1]) * -r[0]
        for i in range(1, nd - 2):
            a, b = p(i, F[i]), p(i + 1, F[i + 1])
            F[i], F[i + 1] = r[i] * a + (1 - r[i]) * b, (1 + r[i]) * a - r[i] * b
        F[last] = p(last, F[last])
        F[last + 1] = F[last + 1] + (1 + r[last]) * F[last]
        F[last] = F[last] * r[last]
    return F[last + 1]


def _exact_dancer(g, nmax):
    nd, nf = len(g["eps"]), len(g["freqs"])
    p = _Prop(g, range(1, nd))
    right, left, r, disk = _emission(g)
    n = disk.shape[0]
    R = [(a * disk).expand(nf, n, n) for a in right]
    L = [(a * disk).expand(nf, n, n) for a in left]
    out = torch.zeros_like(R[0])
    r = r + [0.0]
    for _ in range(nmax + 1):
        # every field crosses its region and meets the boundary there; the directions then change names
        pR = [p(j + 1, R[j]) for j in range(nd - 1)]
        pL = [p(j + 1, L[j]) for j in range(nd - 1)]
        out = out + pR[-1]
        R2, L2 = [None] * (nd - 1), [None] * (nd - 1)
        for i in range(nd):
            if i > 0:
                L2[i - 1] = r[i] * pR[i - 1] + ((1 - r[i]) * pL[i] if i < nd - 1 else 0.0)
            if i < nd - 1:
                R2[i] = -r[i] * pL[i] + ((1 + r[i]) * pR[i - 1] if i > 0 else 0.0)
        R, L = R2, L2
    return out


def _besselj(l, x):
    """J_l(x) by the trapezoidal rule on its integral over a period, which converges past the last digit."""
    k = 2 * (int(np.max(np.abs(x))) + abs(l) + 40)
    t = 2 * np.pi * np.arange(k) / k
    return np.mean(np.cos(l * t - np.asarray(x, dtype=np.float64)[..., None] * np.sin(t)), axis=-1)


def _bessel_zeros(l, m):
    x = np.arange(l + 0.5, l + 4 * m + 20, 0.05)
    y = _besselj(l, x)
    at = np.nonzero(y[:-1] * y[1:] < 0)[0][:m]
    lo, hi = x[at], x[at + 1]
    s = np.sign(y[at])
    for _ in range(60):
        mid = (lo + hi) / 2
        same = np.sign(_besselj(l, mid)) == s
        lo, hi = np.where(same, mid, lo), np.where(same, hi, mid)
    return (lo + hi) / 2


def _bessel_modes(X, M, L, diskR):
    r = np.sqrt(X[:, None] ** 2 + X[None, :] ** 2)
    phi = np.arctan2(*np.broadcast_arrays(X[None, :], X[:, None]))
    zeros = {l: _bessel_zeros(l, M) for l in range(L + 1)}
    pats, kt = [], []
    for m in range(M):
        for l in range(-L, L + 1):
            k = zeros[abs(l)][m] / diskR
            f = np.where(r > diskR, 0.0, _besselj(l, k * np.minimum(r, diskR))) * np.exp(-1j * l * phi)
            pats.append(f / np.sqrt(np.sum(np.abs(f) ** 2)))
            kt.append(complex(k))
    return np.array(pats), np.array(kt)


class _Overlaps:
    """Mode-mixing matrices [frequency, mode, mode'] of a booster's regions."""

    def __init__(self, g, pats, kt, freqs):
        self.g, self.f, self.kt = g, freqs, _t(kt)
        nm, n = len(pats), len(g["X"])
        self.pat = _t(pats)
        mask = _mask(g["X"], g["diskR"])
        self.kz = _kz(1.0, freqs, g["X"])
        shift = lambda a: torch.roll(a, (n // 2, n // 2), (1, 2)).reshape(nm, -1)   # noqa: E731
        self.left = shift(torch.fft.fft2(self.pat)).conj()
        self.right = shift(torch.fft.fft2(self.pat * mask)).T / n ** 2

    def gap(self, dz):
        D = torch.exp(-1j * self.kz * dz).reshape(len(self.f), 1, -1)
        return torch.cat([(self.left * d) @ self.right for d in D.split(16)])

    def disk(self, j):
        g, nm = self.g, len(self.pat)
        diag = torch.exp(-1j * torch.sqrt(_t(_k0(g["eps"][j], self.f))[:, None] ** 2 - self.kt ** 2) * g["distance"][j])
        m = _map(g["eps"][j], g["tx"][j], g["ty"][j], None if g["surf"] is None else g["surf"][j], self.f, g["X"])
        flat = self.pat.reshape(nm, -1)
        if m is None:
            return diag[:, :, None] * (flat.conj() @ flat.T)
        m = m.reshape(len(self.f), 1, -1)
        return diag[:, :, None] * torch.cat([(flat.conj() * d) @ flat.T for d in m.split(16)])


def _chain(g, pats, mats, nf):
    """The boundary solve of the transfer chain with the regions' matrices mats(j)."""
    nm, X = len(pats), g["X"]
    B = (np.sqrt(X[:, None] ** 2 + X[None, :] ** 2) <= g["diskR"]).astype(np.float64)
    emit = _t(np.sum(np.conj(pats) * B / np.sqrt(B.sum()), axis=(1, 2)))[:, None]
    n = np.sqrt(np.where(np.isnan(g["eps"]), 1e30, g["eps"]))
    T2 = torch.eye(nm, dtype=torch.complex128, device=DEV).expand(nf, nm, nm)
    T1 = torch.zeros_like(T2)
    beam = torch.zeros(nf, nm, 1, dtype=torch.complex128, device=DEV)
    for j in range(1, len(n)):
        a, b, P = complex(n[j - 1] + n[j]), complex(n[j - 1] - n[j]), mats(j)
        beam = beam + complex(1 / n[j - 1] ** 2 - 1 / n[j] ** 2) / 2 * ((T1 + T2) @ emit)
        s = complex(1 / (2 * n[j - 1]))
        T1, T2 = s * (a * T1 + b * T2) @ P, s * (b * T1 + a * T2) @ torch.linalg.inv(P)
    boost = -torch.linalg.solve(T2, beam)[:, :, 0]
    return boost, (boost.abs() ** 2).sum(1)


def _exact_modes(g, pats, kt, distance):
    o = _Overlaps(g, pats, kt, g["freqs"])
    disks = {j: o.disk(j) for j in range(2, len(g["eps"]) - 1, 2)}
    got = [_chain(g, pats, lambda j, d=d: disks[j] if j in disks else o.gap(d[j]), len(g["freqs"])) for d in distance]
    return torch.stack([x for x, _ in got]), torch.stack([y for _, y in got])


def _exact_pgrid(g, pats, kt, case):
    """Natural cubic spline (zero second derivative half a cell beyond the ends) of the gaps' matrices at the shifts."""
    o, sg, nsp = _Overlaps(g, pats, kt, g["freqs"]), g["grid"], case["nsp"]
    step = sg[1] - sg[0]
    A = np.zeros((nsp + 2, nsp + 2))
    for row, i, t in ((0, 1, -0.5), (nsp + 1, nsp - 1, 1.5)):
        A[row, i - 1:i + 3] = np.convolve([1, -2, 1], [1 - t, t])
    for j in range(1, nsp + 1):
        A[j, j - 1:j + 2] = np.array([1, 4, 1]) / 6
    inv = np.linalg.inv(A)[:, 1:nsp + 1]

    def mats(j):
        if j % 2 == 0:
            return o.disk(j)
        x = 0.0 if j == len(g["eps"]) - 1 else g["shift"][(j - 1) // 2]
        u = 1 + (x - sg[0]) / step
        i = min(max(int(math.floor(u)), 1), nsp - 1)
        t = u - i
        w = np.array([(1 - t) ** 3, 3 * t ** 3 - 6 * t ** 2 + 4, -3 * t ** 3 + 3 * t ** 2 + 3 * t + 1, t ** 3]) / 6
        return sum(float(c) * o.gap(g["distance"][j] + d) for c, d in zip(w @ inv[i - 1:i + 3], sg))

    boost, _ = _chain(g, pats, mats, case["nf"])
    coupled = (boost.conj() @ _t(g["antenna"])).abs() ** 2
    lo, hi = sg[0] - step / 2, sg[-1] + step / 2
    depth = 0.05 * (hi - lo)
    ext = np.append(g["shift"], g["shift"].sum())
    penalty = 1 - (max(ext.max() - (hi - depth), lo + depth - ext.min(), 0.0) / depth) ** 6
    top = coupled.max()
    norm = top * ((coupled / top) ** -20.0).mean() ** (-1 / 20)
    return (-norm * penalty).reshape(1), coupled


def exact(case, seed):
    g, kind, n, nf = _inputs(case, seed), case["kind"], case.get("n", 1), case.get("nf", 1)
    if kind == "propagate":
        X, f = g["X"], np.array([C0 / g["lam"]])
        E, D = _t(g["E"]), _phasor(1.0, g["dz"], f, X)[0]
        tx, ty = (g["tilt"] if case["prop"] != "propagatorNoTilts" else (0.0, 0.0))
        m = _map(1.0, tx, ty, None if g["surf"] is None else g["surf"][2], f, X)
        m = 1.0 if m is None else m[0]
        if case["prop"] == "propagatorMomentumSpace":
            back = lambda a: torch.roll(a, (-(n // 2), -(n // 2)), (0, 1))   # noqa: E731
            E = torch.fft.ifft2(back(E) * D) * _mask(X, g["diskR"]) * m
            return [torch.roll(torch.fft.fft2(E), (n // 2, n // 2), (0, 1))]
        return [torch.fft.ifft2(torch.fft.fft2(E * _mask(X, g["diskR"])) * D) * m]
    if kind in ("dancer", "cheerleader"):
        points = float(nf) * n * n * _props(kind, case["ndisk"], case["nmax"])
        if points * (2.4e-10 if n & (n - 1) == 0 else 1e-9) > 10:
            return None
        g["use"] = g["distance"] if case["how"] == "oneshot" else g["moved"]
        E = (_exact_cheerleader if kind == "cheerleader" else _exact_dancer)(g, case["nmax"])
        dx = g["X"][1] - g["X"][0]
        beta2 = (E.abs() ** 2).sum((1, 2)) * dx * dx / (math.pi * g["diskR"] ** 2)
        if case["how"] == "oneshot":
            return [E]
        if case["how"] == "device":   # the device buffer holds [y][x]
            E = E.transpose(1, 2).contiguous()
        return [E, beta2]
    if kind == "batch1d":
        if case["nconf"] * nf * case["ndisk"] > 4e7:
            return None
        return list(_exact_1d(g))
    nm = case["M"] * (2 * case.get("L", 0) + 1)
    gaps = case.get("nreq", 1) * (case["ndisk"] + 1) * case.get("nsp", 1)
    if 8.0 * nm * nm * n * n * nf * (gaps + case["ndisk"] * bool(case.get("rough"))) > 2e12:
        return None
    if kind == "transformer":
        pats, kt = _bessel_modes(g["X"], case["M"], case["L"], g["diskR"])
        return [_exact_modes(g, pats, kt, [g["distance"]])[0][0]]
    pats, kt = _lg(g["X"], case["M"], g["diskR"])
    if kind == "pgrid":
        return list(_exact_pgrid(g, pats, kt, case))
    boost, beta2 = _exact_modes(g, pats, kt, [g["moved"]] if kind == "step" else g["all"])
    return [boost, beta2] if kind == "group" else [boost[0], beta2[0]]


def _exact_1d(g):
    n = np.sqrt(np.where(np.isnan(g["eps"]), 1e30, g["eps"]))
    d, f = _t(g["confs"]), _t(g["freqs"])
    t2 = torch.ones(len(d), len(f), dtype=torch.complex128, device=DEV)
    t1, beam = torch.zeros_like(t2), torch.zeros_like(t2)
    for j in range(1, len(n)):
        a, b, s = complex(n[j - 1] + n[j]), complex(n[j - 1] - n[j]), complex(1 / (2 * n[j - 1]))
        P = torch.exp(-2j * math.pi / C0 * complex(n[j]) * (d[:, j, None] * f[None, :]))
        beam = beam + complex(1 / n[j - 1] ** 2 - 1 / n[j] ** 2) / 2 * (t1 + t2)
        t1, t2 = s * (a * t1 + b * t2) * P, s * (b * t1 + a * t2) / P
    boost = -beam / t2
    return boost, boost.abs() ** 2
