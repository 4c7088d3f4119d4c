"""The lossless 1D chain against the general one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    import build
    build.build()
    import bfgb300
    return bfgb300


# an imaginary part of 1e-300 makes every |P| exactly 1 but not the chain lossless; the two round differently, 1e-16
# times regions (13 at most) times the resonance (< 1e2 at 6 disks)
@pytest.mark.parametrize("ndisk,nconf,nf,equal", [(0, 1, 1, True), (1, 3, 33, True), (2, 1, 300, False), (6, 17, 29, True),
                                                  (6, 5, 64, False)])
def test_1d_lossless_equals_general_route(B, ndisk, nconf, nf, equal):
    rng = np.random.default_rng([ndisk, nf])
    nd = max(3, 2 * ndisk + 2)
    eps = np.ones(nd, dtype=complex)
    eps[0] = np.nan
    eps[2:-1:2] = 9.4 if equal else rng.uniform(0.5, 24.0, len(eps[2:-1:2]))
    conf = rng.uniform(7.5e-3, 8.5e-3, (nconf, nd))
    conf[:, 2:-1:2] = 1e-3 if equal else rng.uniform(-1e-3, 2e-3, conf[:, 2:-1:2].shape)
    conf[0, 1], conf[:, -1] = 0.0, 0.0
    freqs, emit = np.linspace(18e9, 22e9, nf), 0.3 - 0.7j
    got = B.transformer_1d_batch(conf, eps, freqs, emit=emit)
    lossy = np.where(np.arange(nd) == 1, eps + 1e-300j, eps)
    for a, b in zip(got, B.transformer_1d_batch(conf, lossy, freqs, emit=emit)):
        assert np.max(np.abs(a - b) / np.abs(b)) < 1e-11
