"""Disks without tilt and surface map (one matrix and one inverse for all that are equal) against the general route,
which a tilt too small to change a number takes."""
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


# 1e-300 of tilt leaves every phase factor at exactly 1 but not the region's class; mixed: the same Gram sums, so the
# same float32 matrices; fp64: sums in another order, 1e-16 times the chain's amplification at 5 disks (~1e2)
@pytest.mark.parametrize("nm,nf,precision,tol", [(1, 1, "fp64", 1e-12), (5, 3, "fp64", 1e-12), (17, 40, "fp64", 1e-12),
                                                 (8, 1, "mixed", 1e-6), (9, 300, "mixed", 1e-6), (33, 2, "mixed", 1e-6)])
def test_flat_disks_equal_general_route(B, nm, nf, precision, tol):
    n, ndisk = 40, 5
    rng = np.random.default_rng(nm)
    X = W.symmetric_grid(n)
    distance, eps, _, _ = W.booster(ndisk, rng.uniform(7.5e-3, 8.5e-3, ndisk), eps_disk=9.4)
    nd = len(eps)
    distance[6], eps[8] = 1.2e-3, 12.0 + 0.01j     # three types: two equal to none, three equal
    tx = np.zeros(nd)
    tx[2] = 2e-4                                    # and one of those tilted
    flat = np.where(np.arange(nd) % 2 == 0, 1e-300, 0.0)
    flat[[0, -1]] = 0.0
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    c = B.SeedCoordinateSystem(X=X, Y=X)
    m = B.SeedModes(c, ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    freqs = np.linspace(19.7e9, 20.3e9, nf)
    got = [B.transformer(B.SeedSetupBoundaries(c, diskno=ndisk, distance=distance, epsilon=eps, relative_tilt_x=tx,
                                               relative_tilt_y=ty), c, m, f=freqs, diskR=0.3, precision=precision)
           for ty in (np.zeros(nd), flat)]
    assert np.linalg.norm(got[0] - got[1]) <= tol * np.linalg.norm(got[1])
