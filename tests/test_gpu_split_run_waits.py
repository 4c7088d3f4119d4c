"""Runs of split stages in one launch: the dancer, the barriers' bounded wait, and two runs at once."""
import numpy as np
import pytest

from .test_gpu_compact import B, booster  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,radius,nf,nmax", [(64, 9.5, 1, 40), (64, 9.5, 2, 9), (64, 30.0, 1, 12), (128, 19.2, 1, 9)])
def test_dancer_run_equals_batch(B, n, radius, nf, nmax):  # noqa: F811
    """Bit for bit the batch's fused stages, on the first solve and on the captured ones; the run of stages is one launch, so
    the solve has fewer launches than stages (four each without it)."""
    c, b, R = booster(B, n, radius)
    st = B.Stack(b, c, R)
    freqs = np.linspace(19.5e9, 20.5e9, 160)
    many, beta = st.dancer(freqs, nmax=nmax, precision="fp64")
    for _ in range(3):
        some, beta1 = st.dancer(freqs[:nf], nmax=nmax, precision="fp64")
        assert np.array_equal(some, many[:nf]) and np.array_equal(beta1, beta[:nf])
    replays, launches = st.graph_stats()
    assert replays >= 1 and launches <= 4 < nmax
    st.close()


def test_barrier_wait_is_bounded(B):  # noqa: F811
    """With one arrival withheld (a test hook; nothing is read or written that a normal launch would not touch) the barrier
    gives up after ~0.1 s, the solve returns BF_ERR_TIMEOUT, and the next ones on the same stack are right again."""
    from bfgb300 import _lib
    c, b, R = booster(B, 64, 9.5)
    st = B.Stack(b, c, R)
    f = np.array([20e9])
    ok, beta = st.dancer(f, nmax=11, precision="fp64")
    L = _lib.lib()
    L.bf_test_run_withhold_arrival(1)
    try:
        with pytest.raises(B.BFError) as e:
            st.dancer(f, nmax=11, precision="fp64")
    finally:
        L.bf_test_run_withhold_arrival(0)
    assert e.value.code == _lib.BF_ERR_TIMEOUT and "barrier" in str(e.value)
    for _ in range(3):
        again, beta1 = st.dancer(f, nmax=11, precision="fp64")
        assert np.array_equal(again, ok) and np.array_equal(beta1, beta)
    st.close()


def test_two_workers_run_at_once(B):  # noqa: F811
    """One-frequency FP64 solves of two stacks on two server workers: two cooperative grids in flight, each bit for bit what
    the stack gives alone."""
    h = B.Handle(0)
    stacks, ref = [], []
    freqs = np.linspace(19.6e9, 20.4e9, 6)
    for seed in (0, 1):
        c, b, R = booster(B, 64, 9.5, seed=seed)
        st = B.Stack(b, c, R, handle=h)
        stacks.append(st)
        ref.append([st.cheerleader(freqs[k:k + 1], nmax=60, precision="fp64")[2][0] for k in range(len(freqs))])
    srv = B.Server(n_workers=2)
    try:
        ids = [(s, k, srv.submit(stacks[s], freqs[k:k + 1], "cheerleader", nmax=60, precision="fp64"))
               for k in range(len(freqs)) for s in (0, 1)]
        for s, k, i in ids:
            assert srv.wait(i, timeout_ms=60000)["beta2"][0] == ref[s][k], (s, k)
    finally:
        srv.close()
        for st in stacks:
            st.close()
        h.close()
