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


def _setup_on(stream, fmm, x, q):
    """laplace.setup with its work on a stream."""
    import ctypes
    from exafmm import _core, _lib
    L, st, h = _lib.lib(), ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    p = ctypes.c_void_p(x.data_ptr())
    _lib.check(L.xfmm_build_tree(fmm._h, p, len(x), p, len(x), -1, 1, st, ctypes.byref(h)))
    tree = _core.Tree(h, fmm, len(x), len(x))
    for f in (L.xfmm_build_list, L.xfmm_m2l_setup, L.xfmm_precompute):
        _lib.check(f(fmm._h, h, st))
    _lib.check(L.xfmm_set_charges(fmm._h, h, ctypes.c_void_p(q.data_ptr()), 1, st))
    return tree


def _evaluate_on(stream, fmm, tree, out):
    import ctypes
    from exafmm import _lib
    _lib.check(_lib.lib().xfmm_evaluate(fmm._h, tree._h, ctypes.c_void_p(out.data_ptr()), 1,
                                        ctypes.c_void_p(stream.cuda_stream)))


def _inputs(seeds, n):
    gen = torch.Generator(device="cuda").manual_seed(7)
    xs = [torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen) for _ in seeds]
    qs = [torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5 for _ in seeds]
    outs = [torch.zeros(n, 4, dtype=torch.float64, device="cuda") for _ in seeds]
    torch.cuda.synchronize()
    return xs, qs, outs


def test_blocks_of_a_tree_freed_with_work_in_flight():
    """A tree evaluated on one stream and freed at once, the next one set up on another stream in its memory."""
    fmm, n, k = _fmm(), 60000, 6
    xs, qs, outs = _inputs(range(k), n)
    streams = [torch.cuda.Stream() for _ in range(2)]
    want = []
    for i in range(k):
        o = torch.zeros_like(outs[i])
        tree = _setup_on(streams[0], fmm, xs[i], qs[i])
        torch.cuda.synchronize()
        _evaluate_on(streams[0], fmm, tree, o)
        torch.cuda.synchronize()
        want.append(o)
        del tree
    for i in range(k):
        tree = _setup_on(streams[i % 2], fmm, xs[i], qs[i])
        for _ in range(4):
            _evaluate_on(streams[i % 2], fmm, tree, outs[i])
        del tree
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert torch.equal(o, w)


def test_memory_of_a_captured_tree_is_reused_only_after_its_replays():
    """A graph of evaluates launched several times, its tree freed at once, the next one set up in its memory."""
    fmm, n = _fmm(), 60000
    (x, x2), (q, q2), (out, other) = _inputs(range(2), n)
    s, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    want = torch.zeros_like(out)
    tree = _setup_on(s, fmm, x, q)
    _evaluate_on(s, fmm, tree, want)
    torch.cuda.synchronize()
    for r in range(3):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(4):
                _evaluate_on(s, fmm, tree, out)
        out.zero_()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with torch.cuda.stream(s2):
            for _ in range(5):
                g.replay()
        del tree  # with launches in flight
        tree = _setup_on(s, fmm, x2, q2)
        _evaluate_on(s, fmm, tree, other)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        assert r == 0 or torch.cuda.mem_get_info()[0] >= free - (8 << 20)  # the tree's blocks are used again
        del tree, g
        tree = _setup_on(s, fmm, x, q)
        _evaluate_on(s, fmm, tree, out)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
