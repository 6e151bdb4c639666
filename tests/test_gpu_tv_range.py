"""The fused TV iterations at values near the largest float, against the oracle: twice u overflows there before u is taken off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(6, 4), (92, 52)])
@pytest.mark.parametrize("iters", [1, 3])
def test_extrapolation_overflows(cuda, oracle, W, H, iters):
    torch = cuda
    from cnncrf import api
    rng = np.random.default_rng(W)
    u0 = rng.random((H, W)).astype(np.float32)
    big = u0[2::4, 2::4]  # no two beside each other: their difference would be no number
    big[...] = rng.choice([-1.0, 1.0], big.shape) * (1.8 + rng.random(big.shape)) * 1e38
    qf = np.stack([rng.standard_normal((H, W)), rng.random((H, W)) * 3], 2).astype(np.float32)
    wx, wy = (rng.random((H, W)).astype(np.float32) for _ in range(2))
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u0, u0, qf, wx, wy)]
    got = api.tv_iterate(*d, 1.5, 0.05, 1e37, iters)
    want = oracle.tv_iterate(u0, u0, qf, wx, wy, 1.5, 0.05, 1e37, iters)
    assert np.isinf(want[1]).any()
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w, equal_nan=True)
