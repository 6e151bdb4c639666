"""The census volume's bit-string kernel against the oracle, bit for bit: every
number of words per string, rows around its 64-pixel tiles, label counts around
the warp, lists that start or end outside the image, and the lists that stay
with the general kernel (fractional, or too wide a range)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,dmin,dstep,D,fs", [(40, 7, 0.0, 1.0, 5, fs) for fs in range(1, 17)] + [
    (63, 3, 0.0, 1.0, 31, 7), (64, 3, 1.0, 1.0, 32, 7), (65, 3, -20.0, 1.0, 33, 7), (129, 2, 60.0, 2.0, 40, 3),
    (5, 4, -300.0, 30.0, 20, 2), (70, 2, 0.0, 1.0, 256, 7), (30, 2, 0.0, 4000.0, 3, 7), (30, 2, 0.0, 300.0, 30, 4),
    (33, 5, 2.0, 0.5, 9, 7), (1, 1, 0.0, 1.0, 3, 1)])
def test_census_forms_bitexact(cuda, oracle, W, H, dmin, dstep, D, fs):
    torch = cuda
    from cnncrf import api
    rng = np.random.default_rng(W * 100 + fs)
    g1, g2 = (np.round(rng.random((H, W)) * 20).astype(np.float32) / 20 for _ in range(2))  # with ties
    vol = api.census_volume(*(torch.from_numpy(g).cuda() for g in (g1, g2)), fs, dmin, dstep, D, 0.7).cpu().numpy()
    assert np.array_equal(vol, oracle.census(g1, g2, fs, oracle.census_list(dmin, dstep, D), 0.7))
