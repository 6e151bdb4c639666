"""The CRF chain passes' forms (one or two warps per chain, two or three block
buffers, whole 16-byte vectors or ragged ones) at the sizes where they can go
wrong, against the oracle bit for bit: chain lengths around the 8-node blocks
and the 32-node sums, label counts around the lanes' 1, 2, 4, 6 and 8 labels
and off the 4-label chunks, chain counts on both sides of the paired form's
limit, and the offsets that the truncation makes redundant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(torch, oracle, H, W, D, L1, L2, delta, shape, iters=2, seed=0):
    from cnncrf.api import crf_solve
    rng = np.random.default_rng(seed + 1000 * H + 10 * W + D)
    cost = rng.random((H, W, D)).astype(np.float32)
    wx = (rng.random((H, W)) * 0.5).astype(np.float32)
    wy = (rng.random((H, W)) * 0.5).astype(np.float32)
    wx[rng.random((H, W)) < 0.1] = 0.0
    olab, olb, _, _ = oracle.crf(cost, wx, wy, L1, L2, delta, iters, shape=shape)
    d = [torch.from_numpy(x).cuda() for x in (cost, wx, wy)]
    lab, lb = crf_solve(*d, L1=L1, L2=L2, delta=delta, total_it=iters, shape=shape)
    assert np.array_equal(lab.cpu().numpy(), olab) and lb == olb


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 65])
@pytest.mark.parametrize("D", [24, 75, 128])
def test_chain_lengths(cuda, oracle, n, D):
    check(cuda, oracle, n, 11, D, 0.5, 1.5, 3, 1)
    check(cuda, oracle, 11, n, D, 0.4, 1.3, 2, 0)


@pytest.mark.parametrize("D", [1, 2, 3, 4, 28, 31, 33, 36, 63, 64, 65, 68, 125, 126, 127, 129, 132, 191, 193, 196, 253, 255, 256])
@pytest.mark.parametrize("delta", [1, 4])
def test_label_counts(cuda, oracle, D, delta):
    check(cuda, oracle, 13, 19, D, 0.3, 2.0, delta, 1)


# 1216 chains are the paired form's limit (less for 256 labels, by its shared memory)
@pytest.mark.parametrize("H,W,D", [(3, 1216, 32), (3, 1217, 32), (1217, 3, 40), (1216, 5, 64), (4, 1300, 61), (9, 700, 256),
                                   (700, 9, 256), (3, 2500, 128)])
def test_chain_counts(cuda, oracle, H, W, D):
    check(cuda, oracle, H, W, D, 0.5, 1.5, 3, 1)


@pytest.mark.parametrize("L1,L2,delta,shape", [(0.5, 1.5, 3, 1), (0.5, 1.5, 4, 1), (2.0, 1.0, 4, 1), (3.0, 2.0, 3, 0), (0.5, 1.51, 3, 1)])
@pytest.mark.parametrize("D", [30, 96])
def test_redundant_offsets(cuda, oracle, L1, L2, delta, shape, D):
    """rho at the far offsets reaches L2 (or just does not): the kernels leave them out (or not)."""
    check(cuda, oracle, 17, 21, D, L1, L2, delta, shape, iters=3)


# the solver's phi at a pitch of whole chunks (or not: few labels, images a few pixels wide), read back as C1
@pytest.mark.parametrize("D", [1, 2, 3, 5, 30, 63, 75, 97, 190, 255])
@pytest.mark.parametrize("H,W", [(1, 9), (9, 2), (17, 40), (3, 1300)])
def test_c1_of_any_pitch(cuda, oracle, H, W, D):
    torch = cuda
    from cnncrf.api import SlackProp
    rng = np.random.default_rng(H * 1000 + D)
    cost = rng.random((H, W, D)).astype(np.float32)
    wx, wy = ((rng.random((H, W)) * 0.5).astype(np.float32) for _ in range(2))
    olab, olb, _, oc1 = oracle.crf(cost, wx, wy, 0.5, 1.5, 3, 3, shape=1, want_c1=True)
    d = [torch.from_numpy(x).cuda() for x in (cost, wx, wy)]
    labels = torch.zeros((H, W), device="cuda", dtype=torch.int32)
    sp = SlackProp()
    sp.init(d[0], labels)
    for k, v in (("L1", 0.5), ("L2", 1.5), ("delta", 3), ("total_it", 3), ("shape", 1)):
        sp.ops[k] = v
    sp.update_W(d[1], d[2])
    for _ in range(2):  # the second solve starts on what the first left behind
        sp.execute()
        assert np.array_equal(labels.cpu().numpy(), olab) and sp.LB() == olb
        assert np.array_equal(sp.get_C1().cpu().numpy(), oc1)
