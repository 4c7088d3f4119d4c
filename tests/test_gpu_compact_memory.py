"""Bounce solves whose stage buffers do not fit the budget: they run on the full grid, and on the stages where they fit."""
import numpy as np
import pytest

from .test_gpu_compact import B, FP64_TOL, booster, rel  # noqa: F401

pytestmark = pytest.mark.gpu


def test_fallback_is_taken_between_the_two_budgets(B):  # noqa: F811
    """From the smallest budget that the full grid accepts (amin > 0 keeps a solve there) upwards in steps of 2 %: every one
    solves, the first ones without a captured stage graph, a generous one with it."""
    n = 51
    c, b, R = booster(B, n, 20.3, ndisk=1, surfaces=False)
    f = np.linspace(19.5e9, 20.5e9, 8)
    ref = B.dancer(0, 3, b, c, f=f, diskR=R)

    def solve(budget, amin, repeat=1):
        h = B.Handle(0, hbm_budget_bytes=int(budget))
        try:
            st = B.Stack(b, c, R, handle=h)
            try:
                for _ in range(repeat):
                    out = st.dancer(f, amin=amin, nmax=3, precision="fp64")[0]
                return out, st.graph_stats()[0]
            finally:
                st.close()
        finally:
            h.close()

    lo, hi = 1e5, 64e6   # refused, accepted
    while hi > 1.005 * lo:
        mid = (lo * hi) ** 0.5
        try:
            solve(mid, 1e-300)
            hi = mid
        except B.BFError:
            lo = mid
    fallbacks = 0
    for k in range(12):
        out, replays = solve(hi * 1.02 ** k, 0.0, repeat=3)
        assert rel(out, ref) < FP64_TOL
        fallbacks += replays == 0
    assert fallbacks >= 1
    assert solve(256e6, 0.0, repeat=3)[1] >= 1
