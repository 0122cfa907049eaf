"""Device memory kept between set-ups: results do not depend on what a reused block held before, threads with
their own handles do not disturb each other, and the memory goes back to the device with the last Fmm
handle."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _step(fmm, seed, n):
    import exafmm.laplace as lap
    rng = np.random.default_rng(seed)
    x, q = rng.random((n, 3)), rng.uniform(-1, 1, n)
    t = lap.setup(lap.init_sources(x, q), lap.init_targets(x), fmm)
    return lap.evaluate(t, fmm)


def _fmm():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import exafmm.laplace as lap
    return lap.LaplaceFmm(4, 40)


def test_reused_blocks_and_return():
    sizes = [(1, 20000), (2, 3000), (3, 50000), (1, 20000)]
    want = {}
    for seed, n in sizes:
        fmm = _fmm()  # a handle of its own: nothing is kept from one to the next
        _step(fmm, *sizes[0])  # the scale-invariant operators are those of the first tree's radius, as below
        want[seed] = _step(fmm, seed, n)
        del fmm
    gc.collect()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    fmm = _fmm()
    for _ in range(3):
        for seed, n in sizes:
            assert np.array_equal(_step(fmm, seed, n), want[seed])
    del fmm
    gc.collect()
    # within the 2 MiB pages of the device allocator
    assert torch.cuda.mem_get_info()[0] >= free0 - (8 << 20)


def test_threads():
    want = {s: _step(_fmm(), s, 8000 + 1000 * s) for s in range(4)}
    bad = []

    def work(s):
        try:
            fmm = _fmm()
            for _ in range(5):
                if not np.array_equal(_step(fmm, s, 8000 + 1000 * s), want[s]):
                    bad.append(s)
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
