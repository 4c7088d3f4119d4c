"""The mixed boundary solve of 17 to 64 modes where T22's rows and columns differ widely in size."""
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


def evanescent_matrices(nm, nd, rng):
    """Modes that keep, halve, ... or lose 15/16 of their amplitude in every gap, and one that doubles it, times powers of i,
    with two couplings of 2^-10: complex64 holds them and their inverses exactly."""
    halvings = np.zeros(nm, dtype=int)
    halvings[nm // 3:] = rng.permutation(np.arange(nm - nm // 3) % 5)
    halvings[-1] = -1
    pm = np.zeros((nd, nm, nm), dtype=complex)
    for j in range(nd):
        pm[j][np.arange(nm), np.arange(nm)] = 2.0 ** (-halvings * (j % 2)) * 1j ** rng.integers(0, 4, nm)
        if j % 2:
            pm[j, 0, nm // 3 + 1] = pm[j, nm // 3 + 2, 1] = 2.0 ** -10
    return pm


# 20 disks of eps 2: T22's entries run from 1e-3 to 2e25, beyond the square root of the largest float32, and the modes
# that belong to the large ones have amplitudes like the others.  A relative change of the matrices changes an amplitude
# at most 1.6e4 times as much (from perturbed oracle solves) and double-float carries 46 bits through 41 regions: 9.3e-9.
@pytest.mark.parametrize("nm,seed", [(17, 1), (24, 0), (32, 1), (33, 2), (64, 0), (64, 1)])
def test_evanescent_modes_keep_their_amplitudes(B, nm, seed):
    n, ndisk = 24, 20
    X = W.symmetric_grid(n)
    distance, e, _, _ = W.booster(ndisk, np.full(ndisk, 8e-3), eps_disk=2.0)
    pm = evanescent_matrices(nm, len(e), np.random.default_rng([nm, ndisk, seed]))
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    geo = dict(diskno=ndisk, distance=distance, epsilon=e)
    rng = np.random.default_rng(1)
    emit, refl = rng.standard_normal((2, nm)) + 1j * rng.standard_normal((2, nm))
    args = dict(f=20e9, diskR=0.3, emit=emit, reflect=refl, propagation_matrices=pm)
    ref = O.transformer(O.seed_setup_boundaries(co, **geo), co, mo, **args)
    got = B.transformer(B.SeedSetupBoundaries(c, **geo), c, m, precision="mixed", **args)
    assert np.max(np.abs(got[0] - ref[0]) / np.abs(ref[0])) < 2e-8
    assert np.linalg.norm(got[1] - ref[1]) < 2e-8 * np.linalg.norm(ref[1])
