"""The normalisation of tall images, whose row sums take several rows per CTA: bit for bit against the oracle through the net
on both sides of that limit, and a time that grows with the height and not with its square."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(ic, W, H):
    from cnncrf.api import StereoNet
    net = StereoNet(1, 1, ic, H + 2, W + 2, topology=1, unary=1, feat_channels=8)
    net.init_net(0.0, 1.0, 1.0)
    return net


@pytest.mark.parametrize("ic,H", [(3, 1518), (3, 1519), (5, 1521), (3, 3043), (1, 3038), (1, 3039), (1, 3100)])
def test_tall_images(cuda, oracle, ic, H):
    torch = cuda
    W = 5
    cfg = oracle.make_cfg(num_layers=1, topology=1, in_channels=ic, unary=1, disp_max=1.0, feat_channels=8, with_pairwise=False)
    net = _net(ic, W, H)
    params = oracle.xavier_params(cfg, seed=2)
    for i, a in enumerate(params):
        net.set_param(i, a)
    rng = np.random.default_rng(H)
    ims = [rng.random((H + 2, W + 2, 4)).astype(np.float32) for _ in range(2)]
    vol = net.predict(*(torch.from_numpy(x).cuda() for x in ims))
    assert np.array_equal(vol.cpu().numpy(), oracle.predict(cfg, params, *ims, oracle.disparity_list(0.0, 1.0, 1.0))[0])


def test_time_grows_with_the_height(cuda):
    torch = cuda
    from cnncrf import _lib as L

    def time(H):
        net = _net(3, 14, H)
        net.init_xavier(0)
        ims = [torch.rand((H + 2, 16, 4), device="cuda") for _ in range(2)]
        net.predict(*ims)
        L.profile_reset()
        L.profile_enable(True)
        for _ in range(5):
            net.predict(*ims)
        L.profile_enable(False)
        ms = sum(L.profile_query(k)[1] for k in ("rowsums", "norm_write"))
        L.profile_reset()
        return ms
    assert time(16000) < 6.0 * time(4000)  # a CTA per two rows: 11 times
