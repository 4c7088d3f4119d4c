"""Overlaps of modes whose patterns differ in size."""
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


# Each entry against its own two modes' sizes: an entry is linear in both patterns, so the tolerances are those of unit
# patterns (fp64 the transforms' rounding; mixed complex64 entries, products of split operands and float32 phases of up
# to k0 dz = 3.5), but for entries that cancel, which are compared at that size too.
@pytest.mark.parametrize("n,small", [(33, 1e-8), (32, 1e-8), (40, 1e-7), (33, 1e-12)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1.6e-6), ("mixed-simt", 1.6e-6)])
def test_small_patterns_keep_their_overlaps(B, n, small, precision, tol):
    nm, ndisk = 6, 2
    X = W.symmetric_grid(n)
    distance, eps, _, _ = W.booster(ndisk, [7.7e-3, 8.4e-3], eps_disk=9.4)
    pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
    scale = np.ones(nm)
    scale[[1, 2, 4]] = small
    pats = pats * scale.reshape((-1,) + (1,) * (pats.ndim - 1))
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    geo = dict(diskno=ndisk, distance=distance, epsilon=eps)
    f = 20e9
    ref = np.array(O.calc_propagation_matrices(O.seed_setup_boundaries(co, **geo), co, mo, f=f, diskR=0.3))[1:]
    got = np.asarray(B.calc_propagation_matrices(B.SeedSetupBoundaries(c, **geo), c, m, f=[f], diskR=0.3,
                                                 precision=precision))[0][1:]
    assert np.max(np.abs(got - ref) / np.outer(scale, scale)) < tol
    assert np.all(np.abs(got[:, range(nm), range(nm)]) > 0)
