"""The FP32 convolutions' kernels and the rule between them, bit for bit
against the oracle through the whole net: channel counts on both sides of each
kernel's range (32, 64, 100, 104 channels; inputs in multiples of 16, 20 or
neither), first layers of every input kind, pixel counts around the 128-pixel
tiles (a one-pixel output, ragged ends, tiles across row ends)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # topology, input channels, feature channels, pairwise channels, W, H
    (1, 3, 100, 64, 1, 1), (0, 3, 100, 64, 127, 1), (1, 3, 100, 64, 128, 1), (1, 3, 100, 64, 43, 3), (0, 1, 100, 64, 129, 2),
    (1, 5, 100, 64, 31, 9), (1, 3, 33, 31, 21, 11), (1, 3, 32, 32, 21, 11), (1, 3, 34, 33, 21, 11), (1, 3, 48, 40, 37, 7),
    (1, 3, 64, 80, 37, 7), (0, 1, 65, 64, 37, 7), (1, 3, 80, 66, 50, 5), (1, 5, 96, 100, 50, 5), (1, 3, 104, 103, 50, 5),
    (1, 3, 105, 104, 50, 5), (1, 3, 112, 112, 18, 5), (0, 3, 128, 128, 18, 5), (1, 3, 20, 16, 90, 4), (1, 3, 60, 52, 90, 4),
]


@pytest.mark.parametrize("topology,ic,feat,pw,W,H", CASES)
def test_net_bitexact_over_kernels(cuda, oracle, topology, ic, feat, pw, W, H):
    torch = cuda
    from cnncrf.api import StereoNet
    D = 6
    cfg = oracle.make_cfg(num_layers=3, topology=topology, in_channels=ic, feat_channels=feat, pw_channels=pw, unary=1,
                          disp_max=float(D - 1))
    p = oracle.padding(cfg)
    rng = np.random.default_rng(feat * 1000 + pw)
    lp, rp = (rng.random((H + 2 * p, W + 2 * p, 4)).astype(np.float32) for _ in range(2))
    net = StereoNet(3, 1, ic, H + 2 * p, W + 2 * p, topology=topology, unary=1, feat_channels=feat, pw_channels=pw,
                    with_pairwise=True)
    net.init_net(0.0, float(D - 1), 1.0)
    params = oracle.xavier_params(cfg, seed=5)
    for i, a in enumerate(params):  # biases too
        params[i] = a if a.ndim == 4 else rng.uniform(-0.1, 0.1, a.shape).astype(np.float32)
        net.set_param(i, params[i])
    vol = net.predict(*(torch.from_numpy(x).cuda() for x in (lp, rp)))
    ovol, opw = oracle.predict(cfg, params, lp, rp, oracle.disparity_list(0.0, float(D - 1), 1.0))
    assert np.array_equal(vol.cpu().numpy(), ovol)
    assert np.array_equal(net.pairwise_out.cpu().numpy(), opw)


def test_epilogue_tanh_bitexact(cuda, oracle):
    """The epilogue's tanh of value pairs equals the oracle's, bit for bit: as
    the biases of layers with zero weights, in the first-layer kernel (one
    layer) and the wide one (two), values around every case of the function
    (2^-12, 9, the exponents' reductions, zeros, infinities, denormals)."""
    torch = cuda
    from cnncrf.api import StereoNet
    f = np.float32
    x = [0.0, -0.0, np.inf, -np.inf, 1e-45, -1e-40, 1e-30, 3e38, -3e38, 88.0, 20.0]
    for c in [2.0 ** -12, 9.0, 1.0, 8.9999] + [0.25 * np.log(2.0) * (2 * k + 1) for k in range(28)]:
        v = f(c)
        for _ in range(4):
            v = np.nextafter(v, f(0))
        for _ in range(9):
            x += [v, -v]
            v = np.nextafter(v, f(100))
    x = np.concatenate([np.array(x, f), np.random.default_rng(3).uniform(-10, 10, 3000).astype(f)])
    x = np.resize(x, (x.size + 99) // 100 * 100).reshape(-1, 100)
    ref = oracle.conv(x.reshape(1, -1, 1), np.ones((1, 1, 1, 1), f), None, act=1).reshape(x.shape)
    for layers in (1, 2):
        h = 3 if layers == 1 else 5
        net = StereoNet(layers, 1, 3, h, h, topology=1)
        net.init_net(0.0, 0.0, 1.0)
        for i in range(net.num_params()):
            net.set_param(i, np.zeros(net.param_shape(i), f))
        im = torch.rand((h, h, 4), device="cuda")
        for row, want in zip(x, ref):
            net.set_param(2 * layers - 1, row)
            net.predict(im, im)
            for side in (0, 1):
                got = net.features(side).cpu().numpy()[0, 0]
                assert np.array_equal(got.view(np.int32) & 0x7fffffff, want.view(np.int32) & 0x7fffffff)
                assert np.array_equal(got, want)
