"""Where the mixed boundary solve of 17 to 64 modes stops."""
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


# Permutations times powers of i, which complex64 holds exactly: what is left is double-float's rounding, 46 bits through
# at most 17 regions, times a change of the result by at most 22 for a change of the matrices by 1 (from perturbed oracle
# solves): 5.3e-12.  T22 and its inverse in complex64 are off by 1e-6, so the corrections decide.
@pytest.mark.parametrize("nm,ndisk,eps", [(17, 8, 9.4), (32, 6, 16.0), (33, 8, 9.4), (64, 4, 24.0)])
def test_refined_solve_ends_at_double_float(B, nm, ndisk, eps):
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
        assert np.linalg.norm(x - y) < 8e-12 * np.linalg.norm(y)
