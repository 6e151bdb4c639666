"""Host threads side by side, a handle or a workspace each: calls of different sizes launch the same kernels with different
amounts of shared memory, whose limit the threads share per kernel and device."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def together(works, rounds):
    """Each work repeated by a thread of its own, all at once; the first error or wrong result of any."""
    import torch
    bad, start = [], threading.Barrier(len(works))

    def loop(work):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(60)
                for _ in range(rounds):
                    if bad:
                        return
                    work()
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    ts = [threading.Thread(target=loop, args=(w,)) for w in works]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not bad, bad[0]


def test_crf_block_buffers(cuda, oracle):
    """The same label count with three block buffers (few chains) and with two (more chains, paired or single)."""
    torch = cuda
    from cnncrf.api import crf_solve
    works = []
    for H, W in ((8, 300), (1200, 6), (1217, 7)):
        rng = np.random.default_rng(H)
        cost, wx, wy = rng.random((H, W, 128)).astype(np.float32), *((rng.random((H, W)) * 0.5).astype(np.float32) for _ in "xy")
        olab, olb, _, _ = oracle.crf(cost, wx, wy, 0.5, 1.5, 3, 2, shape=1)
        d = [torch.from_numpy(x).cuda() for x in (cost, wx, wy)]

        def work(d=d, olab=olab, olb=olb):
            lab, lb = crf_solve(*d, L1=0.5, L2=1.5, delta=3, total_it=2, shape=1, stream=torch.cuda.current_stream())
            assert np.array_equal(lab.cpu().numpy(), olab) and lb == olb
        works.append(work)
    torch.cuda.synchronize()
    together(works, 150)


def test_correlation_and_census_sizes(cuda, oracle):
    """Correlations of different widths and channel counts (integer and fractional lists), census volumes of different ranges."""
    torch = cuda
    from cnncrf import api
    works = []
    for C, D, step in ((64, 40, 1.0), (100, 20, 1.0), (64, 100, 1.0), (128, 90, 1.0), (64, 30, 0.5), (100, 12, 0.5)):
        rng = np.random.default_rng(C + D)
        fl, fr = (torch.from_numpy(rng.random((1, C, 10, 140)).astype(np.float32)).cuda() for _ in range(2))
        disp = -np.arange(D, dtype=np.float32) * np.float32(step)
        want = api.correlation_forward(fl, fr, disp)

        def work(a=(fl, fr, disp), want=want):
            assert torch.equal(api.correlation_forward(*a, stream=torch.cuda.current_stream()), want)
        works.append(work)
    for D, fs in ((60, 7), (20, 7)):
        rng = np.random.default_rng(D)
        l, r = (torch.from_numpy(rng.random((20, 90)).astype(np.float32)).cuda() for _ in range(2))
        want = api.census_volume(l, r, fs, 0.0, 1.0, D)

        def work(a=(l, r, fs, 0.0, 1.0, D), want=want):
            assert torch.equal(api.census_volume(*a, stream=torch.cuda.current_stream()), want)
        works.append(work)
    torch.cuda.synchronize()
    together(works, 800)
