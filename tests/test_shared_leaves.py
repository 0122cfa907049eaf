"""Work shared between warps and CTAs keeps its order of summation: repeated FP64 evaluates (split-K
translations whose parts meet in a scratch, leaves shared by several warps) are bit-identical, and a batch,
whose persistent near field has one warp per leaf take a leaf's parts one after another, gives the bits of
the single evaluates, for every kernel and for leaves from one target to several blocks of 32."""
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
