"""The fused TV iterations against the oracle, bit for bit, where tiles begin and end: images smaller than a tile, with
interior blocks that just fit or just spill, with tiles that touch no border, one-pixel rows and columns; launches of
every iteration count and their splits; C at and below zero (the prox operator's other form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,iters", [(62, 30, 1), (63, 31, 1), (56, 24, 4), (57, 25, 4), (54, 22, 5), (55, 23, 5), (170, 90, 5),
                                       (193, 101, 11), (130, 130, 7), (1, 80, 6), (80, 1, 6), (2, 2, 3), (64, 32, 10)])
@pytest.mark.parametrize("C", [1.5, 0.0, -0.25])
def test_tv_forms_bitexact(cuda, oracle, W, H, iters, C):
    torch = cuda
    from cnncrf import api
    rng = np.random.default_rng(W * 1000 + H)
    u0 = np.round(rng.random((H, W)) * 30).astype(np.float32)
    qf = np.stack([rng.standard_normal((H, W)), rng.random((H, W)) * 3], 2).astype(np.float32)
    wx, wy = (np.where(rng.random((H, W)) < 0.1, 0.0, rng.random((H, W))).astype(np.float32) for _ in range(2))
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u0, u0, qf, wx, wy)]
    got = api.tv_iterate(*d, C, 0.05, 1.0, iters)
    want = oracle.tv_iterate(u0, u0, qf, wx, wy, C, 0.05, 1.0, iters)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)
