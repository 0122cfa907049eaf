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


def _other(kernel, precision, p):
    import exafmm.helmholtz as hel
    import exafmm.laplace as lap
    import exafmm.modified_helmholtz as yuk
    m = {"laplace": lap, "modified_helmholtz": yuk, "helmholtz": hel}[kernel]
    make = {"laplace": lambda: lap.LaplaceFmm(p, 40, precision=precision),
            "modified_helmholtz": lambda: yuk.ModifiedHelmholtzFmm(p, 40, 4.0, precision=precision),
            "helmholtz": lambda: hel.HelmholtzFmm(p, 40, 4.0 + 1.0j, precision=precision)}[kernel]
    return m, make


def _solve(kernel, precision, p, seed, n):
    m, make = _other(kernel, precision, p)
    fmm = make()
    rng = np.random.default_rng(seed)
    g = rng.standard_normal((n, 3))
    x = g / np.linalg.norm(g, axis=1)[:, None] * (0.05 + rng.random(n) ** 3)[:, None]
    q = rng.uniform(-1, 1, n) + (1j * rng.uniform(-1, 1, n) if kernel == "helmholtz" else 0)
    tree = m.setup(m.init_sources(x, q), m.init_targets(x), fmm)
    return m.evaluate(tree, fmm)


# p = 11: the real kernels' transforms run through cuFFT, with grids of their own
PATHS = [("laplace", "mixed", 6), ("modified_helmholtz", "mixed", 5), ("modified_helmholtz", "fp64", 4),
         ("helmholtz", "mixed", 5), ("helmholtz", "fp64", 4), ("laplace", "mixed", 11)]


def test_blocks_of_one_path_serve_another():
    """Every path of the evaluate on blocks that held another's tables, counters and spectra."""
    sizes = [(1, 12000), (2, 3000), (3, 20000)]
    want = {}
    for path in PATHS:
        for s in sizes:
            want[path, s] = _solve(*path, *s)  # nothing is kept: the handle is freed after each
            gc.collect()
    keep = _fmm()
    for r in range(2):
        for s in sizes:
            for path in PATHS[::-1] if r else PATHS:
                got = _solve(*path, *s)
                # close pairs of the mixed Laplace path meet in FP64 atomic sums
                assert np.linalg.norm(got - want[path, s]) <= 1e-13 * np.linalg.norm(want[path, s]), (path, s)
    del keep


def test_batch_on_blocks_of_other_systems():
    from exafmm.batch import BatchedFmm, batched_workload
    import exafmm.laplace as lap
    systems = batched_workload(nsys=6, nmin=2000, nmax=9000, seed=3)
    for precision, tol in (("fp64", 0.0), ("mixed", 1e-13)):
        def batch():
            return BatchedFmm(systems, lambda: lap.LaplaceFmm(4, 64, precision=precision))
        b = batch()
        want = [o.clone() for o in b.evaluate_batch(2)]
        torch.cuda.synchronize()
        del b
        gc.collect()
        keep = _fmm()
        for path in PATHS[:3]:
            _solve(*path, 5, 15000)
        b = batch()
        got = b.evaluate_batch(2)
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert float((g - w).norm()) <= tol * float(w.norm())
        del b, keep
        gc.collect()


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


def _tree(fmm, seed, n):
    import exafmm.laplace as lap
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen)
    q = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    return lap.setup(lap.init_sources(x, q), lap.init_targets(x), fmm)


def test_freeing_a_tree_leaves_another_threads_capture_alone():
    """CUDA breaks a capture when any thread waits for the whole device: a release waits for the tree's own work."""
    import exafmm.laplace as lap
    fmm = _fmm()
    held = [_tree(fmm, 1, 20000)]
    want = torch.empty(20000, 4, dtype=torch.float64, device="cuda")
    lap.evaluate(held[0], fmm, out=want)
    torch.cuda.synchronize()
    a = torch.zeros(1000, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        a.add_(1)
        t = threading.Thread(target=held.clear)
        t.start()
        t.join()
        a.add_(1)
    g.replay()
    out = torch.empty_like(want)
    lap.evaluate(_tree(fmm, 1, 20000), fmm, out=out)
    torch.cuda.synchronize()
    assert bool((a == 2).all()) and torch.equal(out, want)


def test_blocks_of_a_tree_freed_with_work_in_flight():
    """A tree evaluated on one stream and freed at once, the next one set up on another stream in its memory."""
    import exafmm.laplace as lap
    fmm = _fmm()
    seeds, n = range(6), 60000
    want = []
    for s in seeds:
        o = torch.empty(n, 4, dtype=torch.float64, device="cuda")
        lap.evaluate(_tree(fmm, s, n), fmm, out=o)
        torch.cuda.synchronize()
        want.append(o)
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    for s in seeds:
        with torch.cuda.stream(streams[s % 2]):
            outs.append(torch.empty(n, 4, dtype=torch.float64, device="cuda"))
            tree = _tree(fmm, s, n)
            for _ in range(3):
                lap.evaluate(tree, fmm, out=outs[-1])
            del tree
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert torch.equal(o, w)
