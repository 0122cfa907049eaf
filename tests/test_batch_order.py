"""A batch of mixed Laplace systems that share one operator set rebases every system's rows onto system 0's
arrays.  Whichever system comes first, some rebased offsets are negative in one of the two orders (the other
system's arrays lie below system 0's): both orders must give each system its own result."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _batch_eval(fmm, trees, outs):
    from exafmm import _lib
    L, k = _lib.lib(), len(trees)
    arr = lambda v: (ctypes.c_void_p * k)(*v)  # noqa: E731
    h = ctypes.c_void_p()
    _lib.check(L.xfmm_batch_create(arr([fmm._h.value] * k), arr([t._h.value for t in trees]), k, None, ctypes.byref(h)))
    try:
        _lib.check(L.xfmm_batch_evaluate(h, None, arr([o.data_ptr() for o in outs]), 1, None))
        torch.cuda.synchronize()
    finally:
        _lib.check(L.xfmm_batch_free(h))


def test_result_does_not_depend_on_which_system_is_first():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import exafmm.laplace as lap
    rng = np.random.default_rng(11)
    fmm = lap.LaplaceFmm(6, 64, precision="mixed")
    trees, want = [], []
    for n in (4000, 9001):
        x, q = torch.tensor(rng.random((n, 3))).cuda(), torch.tensor(rng.uniform(-1, 1, n)).cuda()
        t = lap.setup(lap.init_sources(x, q), lap.init_targets(x), fmm)
        o = torch.empty(n, 4, dtype=torch.float64, device="cuda")
        lap.evaluate(t, fmm, out=o)
        trees.append(t)
        want.append(o.clone())
    for order in ((0, 1), (1, 0)):
        outs = [torch.zeros_like(want[i]) for i in order]
        _batch_eval(fmm, [trees[i] for i in order], outs)
        for i, o in zip(order, outs):
            # one evaluate against another: FP32 rounding of the mixed path, its bound against the reference
            assert float((o - want[i]).norm() / want[i].norm()) < 5e-6, order
