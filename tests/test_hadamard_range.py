"""The mixed M2L Hadamard keeps its accuracy for sources far weaker than others beside them: a tile takes sources of
very different size in several passes, and with the screened kernels children and the operator's factors have
exponents by windows of 2^-28.

A screened kernel shows a weak source: the strong one's field is gone where the weak one's targets are (k per box
as large as the order's FP32 check potentials allow).  Each set of targets is compared with
the FP64 path at the same order, by its own norm.  Tolerance: the mixed path's bound, 5e-6 (a source that is
lost, or held to a few bits, leaves 1e-4 to 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 5e-6


def _modules():
    import exafmm.helmholtz as hel
    import exafmm.modified_helmholtz as yuk
    import exafmm.laplace as lap
    return {"laplace": (lap, lambda p, ncrit, _, precision: lap.LaplaceFmm(p, ncrit, precision=precision)),
            "modified_helmholtz": (yuk, yuk.ModifiedHelmholtzFmm), "helmholtz": (hel, hel.HelmholtzFmm)}


def _both(kernel, wavek, p, ncrit, x, q, y, depth=None):
    m, cls = _modules()[kernel]
    out = []
    for precision in ("mixed", "fp64"):
        fmm = cls(p, ncrit, wavek, precision=precision)
        tree = m.setup(m.init_sources(x, q), m.init_targets(y), fmm, nonadaptive_depth=depth)
        out.append(m.evaluate(tree, fmm))
    return out


def _check(mixed, full, parts, columns=((slice(0, 1), "potential"), (slice(1, 4), "gradient"))):
    for name, rows in parts.items():
        for c, what in columns:
            d = full[rows][:, c]
            err = np.linalg.norm(mixed[rows][:, c] - d) / np.linalg.norm(d)
            assert err < TOL, (name, what, err)


def _ball(rng, n, centre, radius):
    g = rng.standard_normal((n, 3))
    return np.asarray(centre) + radius * g / np.linalg.norm(g, axis=1)[:, None] * rng.random((n, 1)) ** (1 / 3)


# p = 11: the transforms run through cuFFT for the real kernels
@pytest.mark.parametrize("kernel,wavek,p", [("modified_helmholtz", 40.0, 6), ("modified_helmholtz", 40.0, 11),
                                            ("helmholtz", 3.0 + 40.0j, 6)])
@pytest.mark.parametrize("weak", [1e-6, 1e-9])
def test_weak_ball_beyond_the_screening_length(kernel, wavek, p, weak):
    rng = np.random.default_rng(p)
    n = 3000
    x = np.concatenate([_ball(rng, n, (0, 0, 0), 0.05), _ball(rng, n, (1, 0.1, 0), 0.05)])
    q = rng.uniform(-1, 1, 2 * n) + (1j * rng.uniform(-1, 1, 2 * n) if kernel == "helmholtz" else 0)
    q[n:] *= weak
    mixed, full = _both(kernel, wavek, p, 32, x, q, x)
    _check(mixed, full, {"strong": slice(0, n), "weak": slice(n, 2 * n)})


def test_laplace_gradient_of_a_distant_weak_ball():
    """The gradient falls off faster than the potential: a weak ball far away is ruled by its own charges."""
    rng = np.random.default_rng(5)
    n = 3000
    x = np.concatenate([_ball(rng, n, (0, 0, 0), 0.05), _ball(rng, n, (1000, 100, 0), 0.05)])
    q = rng.uniform(-1, 1, 2 * n)
    q[n:] *= 1e-7
    mixed, full = _both("laplace", None, 6, 32, x, q, x)
    _check(mixed, full, {"strong": slice(0, n), "weak": slice(n, 2 * n)}, [(slice(1, 4), "gradient")])


def _boxes(rng, n, cells):
    """n points well inside each of the unit cells of a 4 x 4 x 4 box (its corners are added: they fix the root box)."""
    pts = [np.asarray(c) + 0.2 + 0.6 * rng.random((n, 3)) for c in cells]
    return np.concatenate(pts + [np.zeros((1, 3)), np.full((1, 3), 4.0)])


@pytest.mark.parametrize("k,p", [(15.0, 6), (25.0, 4)])
def test_weak_child_beside_a_strong_one(k, p):
    """Two siblings, one 1.5e-5 or 7e-10 of the other, and targets that only the weak one's field reaches."""
    rng = np.random.default_rng(1)
    n = 400
    x = _boxes(rng, n, [(0, 0, 0), (1, 0, 0)])
    q = np.concatenate([rng.uniform(0.5, 1, n), 50 * np.exp(-k) * rng.uniform(0.5, 1, n), np.zeros(2)])
    y = _boxes(rng, n, [(3, 0, 0)])
    mixed, full = _both("modified_helmholtz", k, p, 64, x, q, y, depth=2)
    _check(mixed, full, {"targets": slice(0, n)})


def test_far_child_beside_a_near_one():
    """One source cell, and target cells whose operator entries differ by the screening (1e-9 in a block)."""
    rng = np.random.default_rng(2)
    n = 400
    x = _boxes(rng, n, [(0, 0, 0)])
    q = np.concatenate([rng.uniform(0.5, 1, n), np.zeros(2)])
    y = _boxes(rng, n, [(2, 0, 0), (3, 1, 1), (3, 3, 3)])
    mixed, full = _both("modified_helmholtz", 8.0, 8, 64, x, q, y, depth=2)
    _check(mixed, full, {"near": slice(0, n), "far": slice(n, 2 * n), "farthest": slice(2 * n, 3 * n)})


@pytest.mark.parametrize("tcgen05", ["0", "1"])
def test_weak_half_of_a_full_volume(tcgen05, monkeypatch):
    """Full tiles of several groups, and the dense targets of the tcgen05 form."""
    monkeypatch.setenv("XFMM_HADAMARD_TCGEN05", tcgen05)
    rng = np.random.default_rng(3)
    n = 40000
    x = rng.random((n, 3))
    q = rng.uniform(-1, 1, n) * np.where(x[:, 0] < 0.25, 1.0, 1e-9)
    mixed, full = _both("modified_helmholtz", 80.0, 5, 20, x, q, x)
    _check(mixed, full, {"strong": x[:, 0] < 0.25, "weak": x[:, 0] > 0.75})


def test_several_tiles_per_cta():
    """Tiles of several passes and an operator of two windows, one after another in a CTA: the bits of one tile each."""
    import exafmm.modified_helmholtz as yuk
    rng = np.random.default_rng(4)
    n = 60000
    x = rng.random((n, 3))
    q = rng.uniform(-1, 1, n) * np.where(x[:, 0] < 0.25, 1.0, 1e-9)
    fmm = yuk.ModifiedHelmholtzFmm(4, 12, 80.0, precision="mixed")
    tree = yuk.setup(yuk.init_sources(x, q), yuk.init_targets(x), fmm)
    ref = yuk.evaluate(tree, fmm)
    for tiles in (3, 64):
        tree.set_tuning("sparse_hadamard_tiles_per_cta", tiles)
        assert np.array_equal(yuk.evaluate(tree, fmm), ref)


def test_batch_with_weak_sources():
    """The batch's one-launch Hadamard takes a tile's passes too: the weak balls' gradients are as near to FP64 as
    those of single evaluates (which FP32 stages of both bound), within a factor of two for another rounding."""
    torch = pytest.importorskip("torch")
    import exafmm.laplace as lap
    from exafmm.batch import BatchedFmm
    rng = np.random.default_rng(6)
    n, systems = 2000, []
    for k in range(3):
        x = np.concatenate([_ball(rng, n, (0, 0, 0), 0.05), _ball(rng, n, (1000, 100 * k, 0), 0.05)])
        q = rng.uniform(-1, 1, 2 * n)
        q[n:] *= 1e-7
        systems.append((x, q))
    full = BatchedFmm(systems, lambda: lap.LaplaceFmm(6, 32, precision="fp64"))
    want = [o.clone().cpu().numpy() for o in full.evaluate_each()]
    b = BatchedFmm(systems, lambda: lap.LaplaceFmm(6, 32, precision="mixed"))
    one = [o.clone().cpu().numpy() for o in b.evaluate_each()]
    all_ = [o.clone().cpu().numpy() for o in b.evaluate_batch(2)]

    def err(a, w, rows):
        return np.linalg.norm(a[rows, 1:] - w[rows, 1:]) / np.linalg.norm(w[rows, 1:])
    for a, o, w in zip(all_, one, want):
        for rows in (slice(0, n), slice(n, 2 * n)):
            assert err(a, w, rows) <= 2 * err(o, w, rows)
        assert err(o, w, slice(n, 2 * n)) < 1e-3  # weak sources dropped: 1e-2
    torch.cuda.synchronize()
