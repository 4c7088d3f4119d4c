"""The transformer's chain and boundary solve at the mode counts where their
kernels change: 1 to 16 modes (warps of 8 or 16 columns, double-float), 17 to 32
(a warp's FP64 boundary solve), above (a CTA's), against the oracle."""
import numpy as np
import pytest

from bfgb300 import workloads as W
from oracle import bf_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    import build
    build.build()
    import bfgb300
    return bfgb300


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


# the FP64 chain spreads rows over CTAs by the frequency count; complex
# permittivities take the general (not the real) double-float factors
@pytest.mark.parametrize("nm,nf,eps", [(1, 3, 9.4), (2, 1, 24.0), (7, 5, 9.4 + 0.01j), (8, 4, 24.0), (9, 3, 9.4),
                                       (16, 2, 9.4 + 0.01j), (17, 3, 9.4), (31, 2, 9.4), (32, 1, 9.4), (33, 2, 9.4),
                                       (5, 160, 9.4)])
def test_mode_counts_vs_oracle(B, nm, nf, eps):
    # 48 points: the 33 lowest modes are resolved (cond(P) ~ 1; on 24 points it
    # is 3e3 and a 1e-14 change of P moves the result by 66 %)
    n, ndisk = 48, 3
    rng = np.random.default_rng(nm)
    X = W.symmetric_grid(n)
    distance, e, _, _ = W.booster(ndisk, rng.uniform(7.5e-3, 8.5e-3, ndisk), eps_disk=eps)
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    freqs = np.linspace(19.7e9, 20.3e9, nf)
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    geo = dict(diskno=ndisk, distance=distance, epsilon=e)
    refl = rng.standard_normal(nm) + 1j * rng.standard_normal(nm)
    check = sorted({0, nf // 2, nf - 1})
    ref = [O.transformer(O.seed_setup_boundaries(co, **geo), co, mo, f=freqs[k], diskR=0.3, reflect=refl) for k in check]
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-4)):
        boost, back = B.transformer(B.SeedSetupBoundaries(c, **geo), c, m, f=freqs, diskR=0.3, reflect=refl,
                                    precision=precision)
        alone = B.transformer(B.SeedSetupBoundaries(c, **geo), c, m, f=freqs, diskR=0.3, precision=precision)
        for i, k in enumerate(check):
            assert rel(boost[k], ref[i][0]) < tol and rel(back[k], ref[i][1]) < tol, (precision, k)
            assert rel(alone[k], ref[i][0]) < tol, (precision, k)


@pytest.mark.parametrize("nm,ndisk,eps", [(17, 6, 24.0), (32, 6, 24.0), (33, 6, 9.4 + 0.01j), (64, 6, 24.0),
                                          (17, 10, 60.0), (40, 10, 60.0), (64, 10, 60.0)])
def test_refined_boundary_solve(B, nm, ndisk, eps):
    """The mixed boundary solve by refinement (17 to 64 modes) on injected
    matrices that complex64 holds, and inverts, exactly (permutations times
    powers of i), so that its result is as exact as the double-float residual:
    6 disks refine (cond(T22) ~ 3e3), 10 disks of eps 60 have a cond(T22) of ~1e7,
    beyond complex64, and fall back to the double-float chain.  Double-float
    carries ~48 bits: 1e-14 times cond(T22), 1e-7 here."""
    n = 24
    rng = np.random.default_rng([nm, ndisk])
    X = W.symmetric_grid(n)
    distance, e, _, _ = W.booster(ndisk, np.full(ndisk, 8e-3), eps_disk=eps)
    nd = len(e)
    pm = np.zeros((nd, nm, nm), dtype=complex)
    for j in range(nd):
        pm[j, np.arange(nm), rng.permutation(nm)] = 1j ** rng.integers(0, 4, nm)
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    geo = dict(diskno=ndisk, distance=distance, epsilon=e)
    emit, refl = rng.standard_normal((2, nm)) + 1j * rng.standard_normal((2, nm))
    args = dict(f=20e9, diskR=0.3, emit=emit, reflect=refl, propagation_matrices=pm)
    ref = O.transformer(O.seed_setup_boundaries(co, **geo), co, mo, **args)
    got = B.transformer(B.SeedSetupBoundaries(c, **geo), c, m, precision="mixed", **args)
    for x, y in zip(got, ref):
        assert rel(x, y) < 1e-6
