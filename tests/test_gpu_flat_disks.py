"""Disks without tilt and surface map (one matrix and one inverse for all that are equal) against the general route,
which a tilt too small to change a number takes, and the overlaps between the disks against the oracle."""
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


# The overlaps between the disks.  On an odd grid the modes' symmetry makes most rows zero, which are left out: 28 Bessel
# modes leave 118; without symmetry 11 modes have 121 rows (one tile of the tensor cores, operand made in the kernel)
# and 12 have 144 (two tiles, stored operand).  Tolerances of the largest entry: fp64 the transforms' rounding; mixed
# complex64 entries (6e-8), three of four products of split operands (2^-21 of two terms), and float32 phases of up to
# k0 dz (2^-23 of it); 20 cm of air are beyond the range that makes the operand in the kernel.
@pytest.mark.parametrize("n,nm,nf,loss,gap", [
    (51, 28, 3, 0.0, 8.4e-3), (33, 3, 70, 0.0, 8.4e-3), (32, 1, 1, 0.0, 8.4e-3), (32, 11, 5, 0.0, 8.4e-3),
    (40, 12, 3, 0.0, 8.4e-3), (36, 8, 33, 1e-3, 8.4e-3), (41, 5, 2, 1e-3, 8.4e-3), (32, 6, 2, 0.0, 0.2)])
def test_overlaps_vs_oracle(B, n, nm, nf, loss, gap):
    from oracle import bf_oracle as O
    ndisk = 2
    X = W.symmetric_grid(n)
    distance, eps, _, _ = W.booster(ndisk, [7.7e-3, gap], eps_disk=9.4)
    eps[3] = 1.0 - 1j * loss
    c, co = B.SeedCoordinateSystem(X=X, Y=X), O.seed_coordinate_system(X=X, Y=X)
    if nm == 28:
        kw = dict(ThreeDim=True, Mmax=4, Lmax=3, diskR=0.15)
    else:
        pats, kt = W.lg_modes(X, X, nm, 0.05, 0.3)
        kw = dict(ThreeDim=True, Mmax=nm, Lmax=0, diskR=0.3, pattern_input=pats, kT_arr=kt)
    m, mo = B.SeedModes(c, **kw), O.seed_modes(co, **kw)
    freqs = np.linspace(18e9, 22e9, nf)
    geo = dict(diskno=ndisk, distance=distance, epsilon=eps)
    kf = [0, nf - 1]
    ref = np.array([O.calc_propagation_matrices(O.seed_setup_boundaries(co, **geo), co, mo, f=freqs[k],
                                                diskR=kw["diskR"]) for k in kf])[:, 1:]
    for precision, tol in (("fp64", 1e-13), ("mixed", 1.1e-6 + 2.0 ** -23 * 460 * gap)):
        got = B.calc_propagation_matrices(B.SeedSetupBoundaries(c, **geo), c, m, f=freqs, diskR=kw["diskR"],
                                          precision=precision)
        assert np.max(np.abs(got[kf][:, 1:] - ref)) < tol * np.max(np.abs(ref)), precision
