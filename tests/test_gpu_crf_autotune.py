"""The CRF autotuner times each way of running a pass once: where all tiles run it the same way (few chains), the default
stays, whatever the clock says, and the launches are those of one tile."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,D,h,v", [
    (40, 60, 32, 1, 1), (192, 256, 75, 1, 1),  # two warps per chain in both passes
    (1300, 20, 64, None, 1), (20, 1300, 128, 1, None)])  # in one of them
def test_equal_launches_are_timed_once(cuda, H, W, D, h, v):
    torch = cuda
    from cnncrf import _lib as L, tuning
    from cnncrf.api import crf_autotune
    d = [torch.rand(s, device="cuda") for s in ((H, W, D), (H, W), (H, W))]
    tuning.clear()
    try:
        for _ in range(4):
            L.profile_reset()
            L.profile_enable(True)
            crf_autotune(*d, L1=0.5, L2=1.5, delta=3, total_it=4, shape=1)
            L.profile_enable(False)
            tile, found, mh, mv = tuning.get_tile(W, H, D, 1, 3)
            assert found and mh > 0 and mv > 0
            for form, kernel, keys in ((h, "crf_h", ("ring_h", "chains_per_cta_h")), (v, "crf_v", ("ring_v", "chains_per_cta_v"))):
                launches = L.profile_query(kernel)[0]
                if form:
                    assert launches == 3 and all(tile[k] == tuning.DEFAULT[k] for k in keys)
                else:
                    assert launches % 3 == 0 and 3 * 3 <= launches <= 3 * 6
    finally:
        L.profile_enable(False)
        L.profile_reset()
        tuning.clear()
