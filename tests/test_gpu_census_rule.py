"""The rule between the census kernels: sparse lists and few labels of small windows stay with the general kernel, dense ones
take the bit strings, and on either side of the line the volume is the oracle's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs,step,D,bits", [
    (7, 1.0, 128, True), (7, 1.0, 3, True), (7, 1.0, 2, True), (7, 1.0, 1, False), (7, 1000.0, 3, False), (7, 1000.0, 2, False),
    (7, 100.0, 3, True), (7, 150.0, 3, False), (5, 1000.0, 3, False), (1, 1.0, 4, False), (1, 1.0, 12, True), (3, 300.0, 3, False),
    (13, 100.0, 5, True), (13, 300.0, 3, False), (16, 1.0, 2, True), (16, 300.0, 3, False)])
def test_census_rule(cuda, oracle, fs, step, D, bits):
    torch = cuda
    from cnncrf import _lib as L, api
    rng = np.random.default_rng(fs * 100 + D)
    g1, g2 = (np.round(rng.random((5, 70)) * 20).astype(np.float32) / 20 for _ in range(2))
    L.profile_reset()
    L.profile_enable(True)
    vol = api.census_volume(*(torch.from_numpy(g).cuda() for g in (g1, g2)), fs, 0.0, step, D, 0.7).cpu().numpy()
    L.profile_enable(False)
    launches = [L.profile_query(k)[0] for k in ("census_bits", "census")]
    L.profile_reset()
    assert launches == ([1, 0] if bits else [0, 1])
    assert np.array_equal(vol, oracle.census(g1, g2, fs, oracle.census_list(0.0, step, D), 0.7))


@pytest.mark.parametrize("fs,step,D", [(7, 1000.0, 3), (5, 1000.0, 2), (3, 1200.0, 3)])
def test_sparse_lists_cost_no_more(cuda, fs, step, D):
    """A sparse list of whole disparities takes no more than twice the time of one with fractions (the bit strings of all its
    columns took 4 to 9 times as long)."""
    torch = cuda
    from cnncrf import _lib as L, api
    g = [torch.rand((480, 720), device="cuda") for _ in range(2)]

    def time(dstep):
        api.census_volume(*g, fs, 0.0, dstep, D)
        L.profile_reset()
        L.profile_enable(True)
        for _ in range(5):
            api.census_volume(*g, fs, 0.0, dstep, D)
        L.profile_enable(False)
        ms = sum(L.profile_query(k)[1] for k in ("census_bits", "census"))
        L.profile_reset()
        return ms
    assert time(step) < 2.0 * time(step + 0.5)
