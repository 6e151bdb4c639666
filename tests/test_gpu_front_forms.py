"""The normalisation of a pair's two images in common launches, bit for bit
against the oracle through the net: every input kind, images on 16 bytes and
on any float, row lengths and counts around the warps' and the CTAs', several
pairs per launch; and the FP32 net's two chains of layers on a stream of the
caller's, side by side and one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(oracle, ic, W, H, n=1, stream=None):
    from cnncrf.api import StereoNet
    cfg = oracle.make_cfg(num_layers=3, topology=1, in_channels=ic, unary=1, disp_max=3.0)
    p = oracle.padding(cfg)
    net = StereoNet(3, n, ic, H + 2 * p, W + 2 * p, topology=1, unary=1, with_pairwise=True, stream=stream)
    net.init_net(0.0, 3.0, 1.0)
    params = oracle.xavier_params(cfg, seed=9)
    for i, a in enumerate(params):
        net.set_param(i, a)
    return cfg, params, p, net


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("ic", [1, 3, 5])
@pytest.mark.parametrize("W,H", [(1, 1), (26, 2), (27, 3), (90, 1), (251, 14)])
def test_normalised_pairs(cuda, oracle, ic, W, H, aligned):
    torch = cuda
    cfg, params, p, net = _net(oracle, ic, W, H)
    rng = np.random.default_rng(W * 100 + ic)
    ims = [rng.random((H + 2 * p, W + 2 * p, 4)).astype(np.float32) for _ in range(2)]
    dev = []
    for im in ims:
        buf = torch.zeros(im.size + 4, device="cuda")
        v = buf[0 if aligned else 1:][:im.size].view(im.shape)
        v.copy_(torch.from_numpy(im))
        dev.append(v)
    vol = net.predict(*dev)
    ovol, opw = oracle.predict(cfg, params, ims[0], ims[1], oracle.disparity_list(0.0, 3.0, 1.0))
    assert np.array_equal(vol.cpu().numpy(), ovol)
    assert np.array_equal(net.pairwise_out.cpu().numpy(), opw)


def test_chains_on_a_callers_stream(cuda, oracle):
    torch = cuda
    from cnncrf import _lib as L
    W, H, n = 70, 20, 2
    st = torch.cuda.Stream()
    cfg, params, p, net = _net(oracle, 3, W, H, n=n, stream=st)
    rng = np.random.default_rng(4)
    ims = rng.random((6, 2, n, H + 2 * p, W + 2 * p, 4)).astype(np.float32)
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(st):
        for i, (l, r) in enumerate(ims):
            # new tensors each time, freed at once: their memory is reused by the next upload on this stream
            L.profile_enable(i == 3)
            got.append(net.predict(torch.from_numpy(l).cuda(), torch.from_numpy(r).cuda()).clone())
    L.profile_enable(False)
    st.synchronize()
    lst = oracle.disparity_list(0.0, 3.0, 1.0)
    for (l, r), v in zip(ims, got):
        for j in range(n):
            assert np.array_equal(v[j].cpu().numpy(), oracle.predict(cfg, params, l[j], r[j], lst)[0])
