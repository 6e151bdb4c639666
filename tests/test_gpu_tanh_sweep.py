"""The packed tanh of the FP32 convolutions' epilogue is the library's scalar tanh, bit for bit, on every float."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [k << 30 for k in range(4)])
def test_every_float(cuda, first):
    from cnncrf import _lib as L
    n = C.c_uint64(1)
    L.call("cnncrf_selftest_tanh", first, 1 << 30, C.byref(n), None)
    assert n.value == 0


def test_bad_ranges(cuda):
    from cnncrf import _lib as L
    n = C.c_uint64()
    for first, count in ((0, 0), (0, 3), (4, 1 << 32), (1 << 31, (1 << 31) + 2)):
        assert L.lib().cnncrf_selftest_tanh(first, count, C.byref(n), None) == L.EINVAL


def test_nan_stays_nan(cuda, oracle):
    """NaN through the epilogue, as the bias of a layer with zero weights: beside a number in its pair, on either side."""
    torch = cuda
    import numpy as np
    from cnncrf.api import StereoNet
    f = np.float32
    net = StereoNet(1, 1, 3, 3, 3, topology=1)
    net.init_net(0.0, 0.0, 1.0)
    net.set_param(0, np.zeros(net.param_shape(0), f))
    row = np.linspace(-3, 3, 100).astype(f)
    row[[0, 7, 20, 21, 99]] = np.nan
    net.set_param(1, row)
    im = torch.rand((3, 3, 4), device="cuda")
    net.predict(im, im)
    got = net.features(0).cpu().numpy()[0, 0]
    want = oracle.conv(row.reshape(1, -1, 1), np.ones((1, 1, 1, 1), f), None, act=1).reshape(-1)
    assert np.array_equal(np.isnan(got), np.isnan(row)) and np.array_equal(got, want, equal_nan=True)
