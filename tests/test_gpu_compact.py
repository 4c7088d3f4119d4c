"""Bounce stages with the truncated propagator kernel: transform lengths below
(or beside) the grid's own.  Every form that takes the path is compared with the
full-grid path (amin > 0 keeps a solve on it: 1e-300 never stops a bounce) and,
at a few sizes, with the oracle."""
import numpy as np
import pytest

from oracle import bf_oracle as O

pytestmark = pytest.mark.gpu

# FP64: both paths carry a few 1e-16 per propagation, ~60 propagations deep (at
# mixed precision too on grids without a complex64 transform of their own);
# mixed: the single-precision bar of the bounce solvers' beta^2, 1e-4, half of it
# on the field
FP64_TOL, MIXED_TOL = 1e-11, 5e-5


@pytest.fixture(scope="module")
def B():
    import build
    build.build()
    import bfgb300
    return bfgb300


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def booster(B, n, radius_px, ndisk=2, seed=0, surfaces=True):
    """A tilted, rough booster on an n x n grid over 1 m whose disk spans
    radius_px pixels from the axis."""
    rng = np.random.default_rng([seed, n, int(1000 * radius_px)])
    X = (2 * np.arange(n) - (n - 1)) / (2.0 * (n - 1))
    c = B.SeedCoordinateSystem(X=X, Y=X)
    nd = 2 * ndisk + 2
    distance, eps = np.zeros(nd), np.ones(nd, dtype=complex)
    eps[0], eps[2:-1:2] = np.nan, 9.4
    distance[1:-1:2], distance[2:-1:2] = rng.uniform(7.5e-3, 8.5e-3, ndisk), 1e-3
    tx, ty = np.zeros(nd), np.zeros(nd)
    tx[2:-1:2], ty[2:-1:2] = rng.uniform(-5e-4, 5e-4, (2, ndisk))
    surf = np.zeros((nd, n, n))
    if surfaces:
        surf[2] = 1e-5 * rng.standard_normal((n, n))
    b = B.SeedSetupBoundaries(c, diskno=ndisk, distance=distance, epsilon=eps, relative_tilt_x=tx,
                              relative_tilt_y=ty, relative_surfaces=surf)
    return c, b, radius_px / (n - 1)


def box_of(c, R):
    m = np.abs(c.X[:, None] ** 2 + c.Y[None, :] ** 2) < R ** 2
    return int(np.ptp(np.nonzero(m.any(1))[0])) + 1


# (grid, disk radius in pixels, box): at and just above the lengths' limits
# 2 box - 1 <= 8, 16, 32, 40, 64, 80, 128, 160, odd and even grids, grids whose
# own length is no power of two, and boxes beyond half of the grid
SIZES = [(41, 1.2, 3), (40, 3.7, 8), (64, 8.2, 16), (64, 10.2, 20), (65, 10.2, 21), (101, 15.2, 31), (75, 16.2, 33),
         (128, 20.2, 40), (97, 20.2, 41), (150, 32.2, 64), (129, 33.2, 67), (256, 40.2, 80), (51, 20.3, 41)]


@pytest.mark.parametrize("n,radius,box", SIZES)
def test_truncated_kernel_equals_full_grid(B, n, radius, box):
    c, b, R = booster(B, n, radius)
    assert box_of(c, R) == box
    f = np.array([19.7e9, 20.3e9])
    for solve in (B.cheerleader, B.dancer):
        for precision, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            full = solve(1e-300, 6, b, c, f=f, diskR=R, precision="fp64")
            got = solve(0, 6, b, c, f=f, diskR=R, precision=precision)
            assert rel(got, full) < tol, (solve.__name__, precision)


@pytest.mark.parametrize("precision,tol", [("fp64", FP64_TOL), ("mixed", MIXED_TOL)])
def test_truncated_kernel_options(B, precision, tol):
    """Given emission, reflection, both exits, no tilts, and a mirror that lets
    the left exit through, on an odd grid."""
    n = 101
    c, b, R = booster(B, n, 15.2)
    b.r[0] = 0.3
    rng = np.random.default_rng(5)
    emit = rng.standard_normal((6, 2, n, n)) + 1j * rng.standard_normal((6, 2, n, n))
    refl = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    for kw in (dict(emit=emit), dict(reflect=refl), dict(prop=B.propagatorNoTilts)):
        args = dict(f=20e9, diskR=R, returnboth=True, **kw)
        full = B.cheerleader(1e-300, 5, b, c, precision="fp64", **args)
        got = B.cheerleader(0, 5, b, c, precision=precision, **args)
        for x, y in zip(got, full):
            assert rel(x, y) < tol, kw.keys()


@pytest.mark.parametrize("n,radius", [(101, 15.2), (64, 10.2), (97, 20.2)])
def test_truncated_kernel_vs_oracle(B, n, radius):
    c, b, R = booster(B, n, radius)
    co = O.seed_coordinate_system(X=c.X, Y=c.Y)
    so = O.seed_setup_boundaries(co, diskno=2, distance=b.distance, epsilon=b.eps, relative_tilt_x=b.relative_tilt_x,
                                 relative_tilt_y=b.relative_tilt_y, relative_surfaces=b.relative_surfaces)
    for mine, ref in ((B.cheerleader, O.cheerleader), (B.dancer, O.dancer)):
        assert rel(mine(0, 4, b, c, f=20e9, diskR=R), ref(0, 4, so, co, f=20e9, diskR=R)) < FP64_TOL


def test_wavenumbers_without_symmetry_keep_the_grid_transform(B):
    """The truncated kernel's spectrum is folded to one quadrant, which takes
    antisymmetric kX and kY: other wavenumbers run as before."""
    for n in (64, 65):
        c, b, R = booster(B, n, 10.2)
        c.kX = c.kX + 0.3
        full = B.cheerleader(1e-300, 4, b, c, f=20e9, diskR=R)
        assert rel(B.cheerleader(0, 4, b, c, f=20e9, diskR=R), full) < FP64_TOL


def test_batch_equals_single_at_the_truncated_lengths(B):
    """One frequency (split-phase stages) and a batch (fused stages) agree bit
    for bit at lengths 40, 80 and 160."""
    for n, radius in ((64, 9.5), (128, 19.2), (256, 38.2)):
        c, b, R = booster(B, n, radius)
        st = B.Stack(b, c, R)
        freqs = np.linspace(19.5e9, 20.5e9, 160)
        many, _, beta = st.cheerleader(freqs, nmax=4, precision="mixed")
        for k in (0, 83, 159):
            one, _, beta1 = st.cheerleader(freqs[k:k + 1], nmax=4, precision="mixed")
            assert np.array_equal(one[0], many[k]) and beta1[0] == beta[k], (n, k)
        st.close()


def test_out_of_memory_falls_back_to_the_full_grid(B):
    """A budget that holds the full grid's fields but not the stages' buffers: a
    grid that took the full path before the truncated kernel still solves."""
    n = 51
    c, b, R = booster(B, n, 20.3, ndisk=1, surfaces=False)
    f = np.linspace(19.5e9, 20.5e9, 8)
    ref = B.dancer(0, 3, b, c, f=f, diskR=R)
    h = B.Handle(0, hbm_budget_bytes=3_000_000)
    with pytest.raises(B.BFError):   # neither path fits
        B.dancer(0, 3, b, c, f=np.linspace(19.5e9, 20.5e9, 64), diskR=R, handle=h)
    for budget in (3_200_000, 3_600_000, 4_400_000, 6_000_000):
        h2 = B.Handle(0, hbm_budget_bytes=budget)
        try:
            full = B.dancer(1e-300, 3, b, c, f=f, diskR=R, handle=h2)
        except B.BFError:
            continue
        got = B.dancer(0, 3, b, c, f=f, diskR=R, handle=h2)   # accepted whenever the full path is
        assert rel(got, ref) < FP64_TOL and rel(full, ref) < FP64_TOL
        h2.close()
    h.close()
