"""Below 9,472 target leaves several warps share a leaf (near field, far field) or a surface (P2M, P2L); from there on
one warp takes it.  Each kernel and precision on one system just below and one just above that count, with
leaves from one body to several blocks of 32 targets, against direct sums on a sample.

Tolerance: the FMM's truncation error at p = 6, as in the batched tests (1e-4 in potential, 1e-3 in gradient); a
leaf's near field or a surface left out leaves errors of the order of the result.  And mixed against FP64 on the
same tree: the mixed path's bound, 5e-6."""
import functools

import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu
LIMIT = 148 * 64


def _modules():
    import exafmm.helmholtz as hel
    import exafmm.laplace as lap
    import exafmm.modified_helmholtz as yuk
    return {"laplace": (lap, lambda prec: lap.LaplaceFmm(6, 6, precision=prec)),
            "modified_helmholtz": (yuk, lambda prec: yuk.ModifiedHelmholtzFmm(6, 6, 2.0, precision=prec)),
            "helmholtz": (hel, lambda prec: hel.HelmholtzFmm(6, 6, 2.0 + 0.5j, precision=prec))}


def _points(n):
    return np.random.default_rng(0).random((n, 3))


def _leaves(x, y):
    m, fmm = _modules()["laplace"]
    tree = m.setup(m.init_sources(x, np.zeros(len(x))), m.init_targets(y), fmm("fp64"))
    d = tree.dump()
    return int((d["ni"][d["leafs"], 4] > 0).sum())


@functools.lru_cache(None)
def _sizes():
    """The numbers of bodies that give the most target leaves below the limit and the fewest from it on (in steps)."""
    lo, hi = 10000, 80000
    x = _points(hi)
    assert _leaves(x[:lo], x[:lo]) < LIMIT <= _leaves(x[:hi], x[:hi])
    while hi - lo > 64:
        mid = (lo + hi) // 2
        if _leaves(x[:mid], x[:mid]) < LIMIT:
            lo = mid
        else:
            hi = mid
    return lo, hi


@pytest.mark.parametrize("above", [False, True])
@pytest.mark.parametrize("kernel", ["laplace", "modified_helmholtz", "helmholtz"])
def test_below_and_above(kernel, above):
    n = _sizes()[above]
    rng = np.random.default_rng(1)
    x = _points(80000)[:n]
    q = rng.uniform(-1, 1, n) + (1j * rng.uniform(-1, 1, n) if kernel == "helmholtz" else 0)
    m, make = _modules()[kernel]
    wavek = {"laplace": 0.0, "modified_helmholtz": 2.0, "helmholtz": 2.0 + 0.5j}[kernel]
    outs = {}
    for prec in ("fp64", "mixed"):
        fmm = make(prec)
        tree = m.setup(m.init_sources(x, q), m.init_targets(x), fmm)
        d = tree.dump()
        assert (int((d["ni"][d["leafs"], 4] > 0).sum()) >= LIMIT) == above
        outs[prec] = m.evaluate(tree, fmm)
    s = rng.choice(n, 500, replace=False)
    direct = orc.direct(kernel, x, q, x[s], wavek) if kernel != "laplace" else orc.direct(kernel, x, q, x[s])
    pe, ge = orc.rel_l2(outs["fp64"][s], direct)
    assert pe < 1e-4 and ge < 1e-3, (pe, ge)
    pm, gm = orc.rel_l2(outs["mixed"], outs["fp64"])
    assert pm < 5e-6 and gm < 5e-6, (pm, gm)


@pytest.mark.parametrize("kernel", ["laplace", "modified_helmholtz", "helmholtz"])
def test_large_leaves_of_large_systems(kernel):
    """Above the limit, leaves of up to 200 targets: several blocks of 32, several targets per lane (uniform tree)."""
    rng = np.random.default_rng(2)
    n, size = 30000, 1.0 / 32
    x = _points(n)
    cells = np.floor(x[:40] / size) * size  # one cell each
    y = np.concatenate([x] + [c + size * (0.1 + 0.8 * rng.random((k, 3))) for c, k in zip(cells, range(35, 200, 4))])
    q = rng.uniform(-1, 1, n) + (1j * rng.uniform(-1, 1, n) if kernel == "helmholtz" else 0)
    m, make = _modules()[kernel]
    wavek = {"laplace": 0.0, "modified_helmholtz": 2.0, "helmholtz": 2.0 + 0.5j}[kernel]
    outs = {}
    for prec in ("fp64", "mixed"):
        fmm = make(prec)
        tree = m.setup(m.init_sources(x, q), m.init_targets(y), fmm, nonadaptive_depth=5)
        t = tree.dump()
        nt = t["ni"][t["leafs"], 4]
        assert (nt > 0).sum() >= LIMIT and nt.max() > 128
        outs[prec] = m.evaluate(tree, fmm)
    s = n + rng.choice(len(y) - n, 500, replace=False)
    direct = orc.direct(kernel, x, q, y[s], wavek) if kernel != "laplace" else orc.direct(kernel, x, q, y[s])
    pe, ge = orc.rel_l2(outs["fp64"][s], direct)
    assert pe < 1e-4 and ge < 1e-3, (pe, ge)
    pm, gm = orc.rel_l2(outs["mixed"], outs["fp64"])
    assert pm < 5e-6 and gm < 5e-6, (pm, gm)
