"""The Laplace far field takes an equivalent surface line by line (4 p - 4 lines of p points, 2 (p - 2) of
p - 2): every order from the smallest surface (p = 2, no interior lines) to the largest, on an adaptive tree
with W-list (M2P) interactions, against FP64 direct sums.

Tolerance: the kernel-independent FMM's truncation error at order p, which falls by about three quarters of
a digit per order from a few tenths at p = 2 (a wrong or missing surface point leaves errors of the
order of the far field itself, above 1e-2); mixed precision: its bound 5e-6 where larger.  At p = 2 and 3 the
truncation error would hide a missing point: there the numpy FMM of the same order is the reference, within
the bounds of the FP64 and mixed paths against a reference FMM (1e-9, 5e-6)."""
import numpy as np
import pytest

from oracle import fmm_np, orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 3, 5, 7, 11, 13, 16])
def test_orders(p):
    import exafmm.laplace as lap
    rng = np.random.default_rng(p)
    n = 6000
    g = rng.standard_normal((n, 3))
    x = g / np.linalg.norm(g, axis=1)[:, None] * (0.02 + rng.random(n) ** 4)[:, None]
    q = rng.uniform(-1, 1, n)
    direct = orc.direct("laplace", x, q, x)
    bound = max(3e-1 * 10.0 ** (-0.75 * (p - 2)), 3e-9)
    for precision, floor in (("fp64", 0.0), ("mixed", 5e-6)):
        fmm = lap.LaplaceFmm(p, 60 if p < 7 else 200, precision=precision)
        tree = lap.setup(lap.init_sources(x, q), lap.init_targets(x), fmm)
        assert p > 5 or tree.info()["nm2p"] > 0
        pe, ge = orc.rel_l2(lap.evaluate(tree, fmm), direct)
        assert pe < max(bound, floor) and ge < 10 * max(bound, floor), (precision, pe, ge)


@pytest.mark.parametrize("p", [2, 3, 4])
def test_small_orders_against_the_same_fmm(p):
    import exafmm.laplace as lap
    rng = np.random.default_rng(p)
    n = 3000
    g = rng.standard_normal((n, 3))
    x = g / np.linalg.norm(g, axis=1)[:, None] * (0.02 + rng.random(n) ** 4)[:, None]
    q = rng.uniform(-1, 1, n)
    ref = fmm_np.NpFmm("laplace", p, 60).setup(x, q, x).evaluate()
    for precision, tol in (("fp64", 1e-9), ("mixed", 5e-6)):
        fmm = lap.LaplaceFmm(p, 60, precision=precision)
        tree = lap.setup(lap.init_sources(x, q), lap.init_targets(x), fmm)
        assert tree.info()["nm2p"] > 0
        pe, ge = orc.rel_l2(lap.evaluate(tree, fmm), ref)
        assert pe < tol and ge < tol, (precision, pe, ge)
