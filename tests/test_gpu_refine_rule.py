"""Which form of the mixed boundary solve a stack takes from 17 modes on: the same result either way."""
import numpy as np
import pytest

from bfgb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    import build
    build.build()
    import bfgb300
    return bfgb300


# 20 disks of eps 24 are refined, 36 take the chain in double-float at once (plane waves grow 1e4 and 1e8 times); the
# same matrices injected are tried by refinement first.  Double-float's 46 bits through 73 regions, times the change of the
# amplitudes per change of the matrices: at most the growth, 1e8 for single frequencies of 36 disks (1e-4), 1e5 for 20
# (1e-7).
@pytest.mark.parametrize("nm,ndisk,tol", [(17, 20, 1e-7), (17, 36, 1e-4), (33, 20, 1e-7), (33, 36, 1e-4)])
def test_chain_and_refinement_agree(B, nm, ndisk, tol):
    n = 48
    rng = np.random.default_rng(ndisk)
    X = W.symmetric_grid(n)
    distance, e, _, _ = W.booster(ndisk, rng.uniform(7.5e-3, 8.5e-3, ndisk), eps_disk=24.0)
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    c = B.SeedCoordinateSystem(X=X, Y=X)
    m = B.SeedModes(c, ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    freqs = np.linspace(19.5e9, 20.5e9, 5)
    refl = rng.standard_normal(nm) + 1j * rng.standard_normal(nm)
    bdry = lambda: B.SeedSetupBoundaries(c, diskno=ndisk, distance=distance, epsilon=e.copy())  # noqa: E731
    P = np.asarray(B.calc_propagation_matrices(bdry(), c, m, f=freqs, diskR=0.3, precision="mixed"))
    got = B.transformer(bdry(), c, m, f=freqs, diskR=0.3, reflect=refl, precision="mixed")
    ref = B.transformer(bdry(), c, m, f=freqs, diskR=0.3, reflect=refl, precision="mixed", propagation_matrices=P)
    for x, y in zip(got, ref):
        for k in range(len(freqs)):
            assert np.linalg.norm(x[k] - y[k]) < tol * np.linalg.norm(y[k]), k
