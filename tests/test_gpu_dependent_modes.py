"""Mode sets that are not independent on their grid."""
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


# More modes than the disk has pixels: the overlaps' rank is lost to rounding, which is all that keeps the matrices from
# being singular.  Such a call solves (to numbers that mean nothing); leaving out the rows that cancel by symmetry made
# zeros of that rounding, and a matrix singular to the bit of 12 of these.
@pytest.mark.parametrize("n,R,nm,ndisk,waist", [(9, 0.15, 7, 4, 0.05), (51, 0.03, 17, 3, 0.05), (9, 0.2, 20, 3, 0.05),
                                                (51, 0.03, 40, 2, 0.05), (33, 0.05, 12, 2, 0.03), (17, 0.1, 10, 3, 0.08)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dependent_modes_are_accepted(B, n, R, nm, ndisk, waist, precision):
    X = (2 * np.arange(n) - (n - 1)) / (2.0 * (n - 1))
    distance, eps, _, _ = W.booster(ndisk, np.linspace(7.6e-3, 8.4e-3, ndisk), eps_disk=9.4)
    pats, kt = W.lg_modes(X, X, nm, waist, R)
    c = B.SeedCoordinateSystem(X=X, Y=X)
    m = B.SeedModes(c, ThreeDim=True, Mmax=nm, Lmax=0, diskR=R, pattern_input=pats, kT_arr=kt)
    for f in (18.5e9, 20e9, 21.5e9):
        B.transformer(B.SeedSetupBoundaries(c, diskno=ndisk, distance=distance, epsilon=eps.copy()), c, m, f=f, diskR=R,
                      precision=precision)
