"""The fused TV iterations with weights of any sign, against the oracle bit for bit: a zero stays a zero through the prox
operator whatever its weight's sign, and the short form of it may serve the tiles without negative weights only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(W, H, seed):
    rng = np.random.default_rng(seed)
    u0 = np.round(rng.random((H, W)) * 6).astype(np.float32)  # plateaus: zero gradients in the first iteration
    qf = np.stack([rng.standard_normal((H, W)), rng.random((H, W)) * 3], 2).astype(np.float32)
    wx, wy = (rng.random((H, W)).astype(np.float32) for _ in range(2))
    return u0, qf, wx, wy


def check(torch, oracle, u0, qf, wx, wy, C, step, iters):
    from cnncrf import api
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u0, u0, qf, wx, wy)]
    got = api.tv_iterate(*d, C, 0.05, step, iters)
    want = oracle.tv_iterate(u0, u0, qf, wx, wy, C, 0.05, step, iters)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)


@pytest.mark.parametrize("W,H", [(1, 1), (9, 5), (64, 32), (170, 90)])
@pytest.mark.parametrize("C", [1.5, 0.0, -0.25])
@pytest.mark.parametrize("share", ["all", "some", "one"])
def test_negative_weights(cuda, oracle, W, H, C, share):
    u0, qf, wx, wy = fields(W, H, W * 100 + H)
    rng = np.random.default_rng(7)
    for w in (wx, wy):
        if share == "one":
            w[H // 2, W // 2] = -0.5
        else:
            w[rng.random((H, W)) < (2.0 if share == "all" else 0.3)] *= -1.0
    check(cuda, oracle, u0, qf, wx, wy, C, 1.0, 6)
