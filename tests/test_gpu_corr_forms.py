"""The FP32 integer correlation's kernels and the rule between them, bit for
bit against the oracle: channel counts in and off multiples of 4, row lengths
around the 64- and 128-pixel tiles, label counts around the 8-label groups and
both sides of 64 and 256, lists that repeat, skip or reverse taps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(torch, oracle, C, H, W, lst):
    from cnncrf.api import correlation_forward
    rng = np.random.default_rng(C * 1000 + W)
    fl, fr = (rng.standard_normal((C, H, W)).astype(np.float32) for _ in range(2))
    lst = np.asarray(lst, np.float32)
    out = correlation_forward(*(torch.from_numpy(f[None]).cuda() for f in (fl, fr)), lst).cpu().numpy()
    assert np.array_equal(out, oracle.correlation(fl.transpose(1, 2, 0), fr.transpose(1, 2, 0), lst))


@pytest.mark.parametrize("W", [1, 8, 63, 64, 65, 127, 128, 129, 200])
@pytest.mark.parametrize("C,D", [(4, 8), (100, 32), (20, 65)])
def test_row_lengths(cuda, oracle, C, D, W):
    check(cuda, oracle, C, 2, W, -np.arange(D))


@pytest.mark.parametrize("D", [1, 7, 9, 56, 63, 64, 65, 72, 127, 128, 130, 200, 256, 257])
@pytest.mark.parametrize("C", [8, 36, 7])
def test_label_counts(cuda, oracle, C, D):
    check(cuda, oracle, C, 2, 150, -np.arange(D))


@pytest.mark.parametrize("lst", [[0, 0, 0], [-1, 0, 1], [3, 2, 1, 0, -1], [-5, -8, -11, -14], [4, -60, 4, 0],
                                 list(range(-40, 41, 2)), [-300, -299], [0, -255], [0, -256], [0.25, 0.0, -0.25], [7, -3.75, 2.5]])
def test_lists(cuda, oracle, lst):
    check(cuda, oracle, 100, 3, 70, lst)
