"""A tree evaluated with one set of operators, then with another in the same memory: nothing of the first set is used
for the second, in the default form of the mixed M2L Hadamard and in the opt-in tcgen05 form, which keeps its
operator blocks in a layout of its own.  Reference: the second operators on a tree of their own, the same
arithmetic (1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tcgen05", ["0", "1"])
def test_second_operators_on_the_same_tree(tcgen05, monkeypatch):
    import exafmm.modified_helmholtz as yuk
    from exafmm import _lib
    monkeypatch.setenv("XFMM_HADAMARD_TCGEN05", tcgen05)
    rng = np.random.default_rng(1)
    n = 40000
    x, q = rng.random((n, 3)), rng.uniform(-1, 1, n)

    def fmm(wavek):
        return yuk.ModifiedHelmholtzFmm(4, 20, wavek, precision="mixed")

    keep = fmm(1.0)  # while a handle lives, released blocks are kept, and serve the second operators
    tree = yuk.setup(yuk.init_sources(x, q), yuk.init_targets(x), fmm(2.0))
    yuk.evaluate(tree, tree.fmm)
    tree.fmm = None  # the first operators' memory is free
    tree.fmm = fmm(4.0)
    _lib.check(_lib.lib().xfmm_precompute(tree.fmm._h, tree._h, None))
    out = yuk.evaluate(tree, tree.fmm)
    own = yuk.setup(yuk.init_sources(x, q), yuk.init_targets(x), fmm(4.0))
    ref = yuk.evaluate(own, own.fmm)
    del keep
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)
