"""The 1D batch's rounding: the short forms of lossless regions give the bits of the general ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    import build
    build.build()
    import bfgb300
    return bfgb300


# Random spacings of 20 disks of eps 24 have resonances that amplify a unit of rounding more than 1e5 times, so beta^2 of
# two forms of one formula agree to 1e-9 at best; an imaginary part of 1e-300 takes the general form and changes no sum.
@pytest.mark.parametrize("ndisk,nconf,nf,emit", [(20, 300, 64, 1.0), (20, 60, 33, 0.3 - 0.7j), (1, 3, 1, 1.0),
                                                 (7, 40, 65, 0.3 - 0.7j)])
def test_lossless_regions_have_the_general_bits(B, ndisk, nconf, nf, emit):
    rng = np.random.default_rng([ndisk, nf])
    nd = 2 * ndisk + 2
    eps = np.ones(nd, dtype=complex)
    eps[0] = np.nan
    eps[2:-1:2] = 24.0
    conf = np.zeros((nconf, nd))
    conf[:, 1:-1:2] = rng.uniform(7.5e-3, 8.5e-3, (nconf, ndisk))
    conf[:, 2:-1:2] = 1e-3
    conf[nconf // 2:, 2:-1:2] = rng.uniform(-1e-3, 2e-3, (nconf - nconf // 2, ndisk))
    freqs = np.linspace(19.5e9, 20.5e9, nf)
    got = B.transformer_1d_batch(conf, eps, freqs, emit=emit)
    general = eps + 1e-300j
    general[0] = np.nan
    for a, b in zip(got, B.transformer_1d_batch(conf, general, freqs, emit=emit)):
        assert np.array_equal(a, b)


# lossy, absorbing and lossless regions side by side, equal ones among them, against the oracle: 1e-16 times 15 regions
# times a resonance below 1e2
def test_mixed_regions_vs_oracle(B):
    from oracle import bf_oracle as O
    ndisk, nf = 7, 5
    rng = np.random.default_rng(7)
    nd = 2 * ndisk + 2
    eps = np.ones(nd, dtype=complex)
    eps[0] = np.nan
    eps[2:-1:2] = [9.4, 9.4 - 0.02j, 9.4, 9.4, 24.0 - 0.1j, 24.0 - 0.1j, 2.0]
    eps[9] = 1.0 - 1e-3j
    conf = np.zeros((3, nd))
    conf[:, 1:-1:2] = rng.uniform(7.5e-3, 8.5e-3, (3, ndisk))
    conf[:, 2:-1:2] = 1e-3
    freqs = np.linspace(18e9, 22e9, nf)
    boost, beta2 = B.transformer_1d_batch(conf, eps, freqs)
    co = O.seed_coordinate_system(X=np.array([1e-7]), Y=np.array([1e-7]))
    mo = O.seed_modes(co, ThreeDim=False)
    for i, d in enumerate(conf):
        for k, f in enumerate(freqs):
            bdry = O.seed_setup_boundaries(co, diskno=ndisk, distance=d, epsilon=eps.copy())
            ref = O.transformer(bdry, co, mo, f=f, prop=O.propagator1d)[0]
            assert abs(boost[i, k] - ref) < 1e-12 * abs(ref), (i, k)
