"""Work shared between warps and CTAs keeps its order of summation: repeated FP64 evaluates (split-K
translations whose parts meet in a scratch, leaves shared by several warps) are bit-identical, and a batch,
whose persistent near field has one warp per leaf take a leaf's parts one after another, gives the bits of
the single evaluates, for every kernel and for leaves from one target to several blocks of 32.  Repeated mixed
evaluates give the same bits too (Laplace: on points without close pairs, whose corrections meet in atomic sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _fmm(kernel, precision="fp64"):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import exafmm.helmholtz as hel
    import exafmm.laplace as lap
    import exafmm.modified_helmholtz as yuk
    return {"laplace": lambda: lap.LaplaceFmm(4, 100, precision=precision),
            "modified_helmholtz": lambda: yuk.ModifiedHelmholtzFmm(4, 100, 3.0, precision=precision),
            "helmholtz": lambda: hel.HelmholtzFmm(4, 100, 3.0 + 0.5j, precision=precision)}[kernel]


def _system(kernel, n, seed):
    rng = np.random.default_rng(seed)
    g = rng.standard_normal((n, 3))
    x = g / np.linalg.norm(g, axis=1)[:, None] * (0.01 + rng.random(n) ** 3)[:, None]
    q = rng.uniform(-1, 1, n)
    return x, q + 1j * rng.uniform(-1, 1, n) if kernel == "helmholtz" else q


@pytest.mark.parametrize("kernel", ["laplace", "modified_helmholtz", "helmholtz"])
def test_batch_and_repeats_give_the_same_bits(kernel):
    from exafmm.batch import BatchedFmm
    b = BatchedFmm([_system(kernel, n, n) for n in (300, 2500, 6000)], _fmm(kernel))
    first = [o.clone() for o in b.evaluate_each()]
    again = [o.clone() for o in b.evaluate_each()]
    batch = [o.clone() for o in b.evaluate_batch(2)]
    torch.cuda.synchronize()
    for f, a, c in zip(first, again, batch):
        assert torch.equal(f, a) and torch.equal(f, c)


@pytest.mark.parametrize("kernel", ["laplace", "modified_helmholtz", "helmholtz"])
def test_repeated_mixed_evaluates_give_the_same_bits(kernel):
    import exafmm.helmholtz as hel
    import exafmm.laplace as lap
    import exafmm.modified_helmholtz as yuk
    m = {"laplace": lap, "modified_helmholtz": yuk, "helmholtz": hel}[kernel]
    fmm = _fmm(kernel, "mixed")()
    rng = np.random.default_rng(1)
    g = np.stack(np.meshgrid(*[np.arange(22.0)] * 3), axis=-1).reshape(-1, 3)
    x = g + 0.4 * rng.random(g.shape)  # neighbours at least 0.6 apart
    q = rng.uniform(-1, 1, len(x)) + (1j * rng.uniform(-1, 1, len(x)) if kernel == "helmholtz" else 0)
    tree = m.setup(m.init_sources(x, q), m.init_targets(x), fmm)
    first = m.evaluate(tree, fmm)
    for _ in range(3):
        assert np.array_equal(m.evaluate(tree, fmm), first)
