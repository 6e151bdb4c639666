"""A pixel without a finite cost: its chains' minima are not numbers, so neither is the bound, for every label count that
leaves no pad label among the lanes' (the oracle's bound is NaN too)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("H,W", [(9, 20), (1300, 4)])  # two warps per chain, one
def test_bound_is_no_number(cuda, oracle, D, value, H, W):
    torch = cuda
    from cnncrf.api import crf_solve
    rng = np.random.default_rng(D)
    cost = rng.random((H, W, D)).astype(np.float32)
    wx, wy = ((rng.random((H, W)) * 0.5).astype(np.float32) for _ in range(2))
    cost[H // 2, W // 2] = value
    for iters in (1, 3):
        if H < 100:
            assert np.isnan(oracle.crf(cost, wx, wy, 0.5, 1.5, 3, iters, shape=1)[1])
        _, lb = crf_solve(*(torch.from_numpy(x).cuda() for x in (cost, wx, wy)), L1=0.5, L2=1.5, delta=3, total_it=iters, shape=1)
        assert np.isnan(lb)
