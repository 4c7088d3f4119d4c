"""The gaps' overlaps over the range of the operand that is made in the multiplying kernel."""
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


# Random patterns weigh every bin, the corners (which decay at 18 GHz on 96 and 128 points over 1 m) like the centre.
# Phases up to 25 radians over 6 cm (several turns taken off), the stored operand beyond, growth in negative gaps, loss
# and gain.  Of the largest entry: complex64 entries, three of four products of split operands and float32 phases of up
# to k0 dz, 1.1e-6 + 2^-23 460 dz; fp64 the transforms' rounding.
@pytest.mark.parametrize("n,gaps,eps", [(96, (0.03, 0.05), 1.0), (96, (0.06, 8e-3), 1.0 - 1e-3j), (128, (-0.01, 0.02), 1.0),
                                        (101, (0.04, -0.005), 1.0 + 1e-3j), (96, (0.09, 0.03), 1.0)])
def test_long_and_negative_gaps_vs_oracle(B, n, gaps, eps):
    nm, ndisk, R = 4, 2, 0.3
    rng = np.random.default_rng([n, int(1e3 * gaps[0]) + 100])
    X = W.symmetric_grid(n)
    distance, e, _, _ = W.booster(ndisk, list(gaps), eps_disk=9.4)
    e[[1, 3]] = eps
    pats = rng.standard_normal((nm, 1, n, n, 1)) + 1j * rng.standard_normal((nm, 1, n, n, 1))
    pats[:, :, X[:, None] ** 2 + X[None, :] ** 2 >= R ** 2] = 0.0
    pats /= np.sqrt(np.sum(np.abs(pats) ** 2, axis=(1, 2, 3, 4), keepdims=True))
    kt = np.linspace(10.0, 60.0, nm).reshape(nm, 1).astype(complex)
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=R, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    geo = dict(diskno=ndisk, distance=distance, epsilon=e)
    freqs = np.array([18e9, 20e9])
    ref = np.array([O.calc_propagation_matrices(O.seed_setup_boundaries(co, **geo), co, mo, f=f, diskR=R)
                    for f in freqs])[:, 1:]
    for precision, tol in (("fp64", 1e-13), ("mixed", 1.1e-6 + 2.0 ** -23 * 460 * max(map(abs, gaps)))):
        got = B.calc_propagation_matrices(B.SeedSetupBoundaries(c, **geo), c, m, f=freqs, diskR=R, precision=precision)
        for j in range(ref.shape[1]):
            assert np.max(np.abs(got[:, 1 + j] - ref[:, j])) < tol * np.max(np.abs(ref[:, j])), (precision, j)
