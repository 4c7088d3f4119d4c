"""Bounce stages of a few frequencies in one launch."""
import numpy as np
import pytest

from .test_gpu_compact import B, booster  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,radius,nf", [(64, 9.5, 1), (64, 9.5, 4), (64, 30.0, 2), (49, 7.4, 3), (128, 19.2, 1)])
def test_run_of_split_stages_equals_batch(B, n, radius, nf):
    """Barriers between the phases in place of launches (FP64): bit for bit the batch's fused stages, on the first solve and
    on the captured ones, with bounces and with none."""
    c, b, R = booster(B, n, radius)
    st = B.Stack(b, c, R)
    freqs = np.linspace(19.5e9, 20.5e9, 160)
    for nmax in (0, 5):
        many, _, beta = st.cheerleader(freqs, nmax=nmax, precision="fp64")
        for _ in range(3):
            some, _, beta1 = st.cheerleader(freqs[:nf], nmax=nmax, precision="fp64")
            assert np.array_equal(some, many[:nf]) and np.array_equal(beta1, beta[:nf])
