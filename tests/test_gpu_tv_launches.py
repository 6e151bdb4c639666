"""How many iterations a launch of the TV kernel takes: up to 8 where the field is at most a tile per SM, up to 5 beyond, with
the oracle's bits on both sides of the limit and at the longer launches' tile edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,iters,launches", [
    (40, 30, 6, 1), (40, 30, 8, 1), (40, 30, 12, 2), (1, 1, 16, 2), (48, 16, 8, 1), (49, 17, 8, 1), (96, 32, 7, 1), (97, 33, 24, 3),
    (384, 304, 8, 1), (385, 304, 8, 2), (384, 305, 16, 4)])
def test_iterations_per_launch(cuda, oracle, W, H, iters, launches):
    torch = cuda
    from cnncrf import _lib as L, api
    rng = np.random.default_rng(W + H)
    u0 = np.round(rng.random((H, W)) * 30).astype(np.float32)
    qf = np.stack([rng.standard_normal((H, W)), rng.random((H, W)) * 3], 2).astype(np.float32)
    wx, wy = (rng.random((H, W)).astype(np.float32) for _ in range(2))
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u0, u0, qf, wx, wy)]
    L.profile_reset()
    L.profile_enable(True)
    got = api.tv_iterate(*d, 1.5, 0.05, 1.0, iters)
    L.profile_enable(False)
    n = L.profile_query("tv")[0]
    L.profile_reset()
    assert n == launches
    for g, w in zip(got, oracle.tv_iterate(u0, u0, qf, wx, wy, 1.5, 0.05, 1.0, iters)):
        assert np.array_equal(g.cpu().numpy(), w)
