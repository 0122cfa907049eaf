"""The FP64 M2L Hadamard forms a complex product from three real ones; the tile edges (targets around a
CTA's 256, a warp's 32, a tile's 8) on the real and complex kernels against direct sums.

Tolerance: the FMM's truncation error at p = 8 (5e-7 on these sets; potentials and gradients of the real
kernel 1e-6 and 1e-5, the complex kernel at k = 2 the same)."""
import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["laplace", "helmholtz"])
@pytest.mark.parametrize("n,ncrit", [(500, 32), (2200, 30), (9000, 30), (11000, 30), (30000, 100)])
def test_direct(kernel, n, ncrit):
    import exafmm.helmholtz as hel
    import exafmm.laplace as lap
    rng = np.random.default_rng(n)
    x, q = rng.random((n, 3)), rng.uniform(-1, 1, n)
    m, wk = (lap, 0.0) if kernel == "laplace" else (hel, 2.0)
    if kernel == "helmholtz":
        q = q + 1j * rng.uniform(-1, 1, n)
    fmm = lap.LaplaceFmm(8, ncrit) if kernel == "laplace" else hel.HelmholtzFmm(8, ncrit, wk + 0j)
    t = m.setup(m.init_sources(x, q), m.init_targets(x), fmm)
    out = m.evaluate(t, fmm)
    s = rng.choice(n, min(n, 500), replace=False)
    d = orc.direct(kernel, x, q, x[s], wk) if kernel == "helmholtz" else orc.direct(kernel, x, q, x[s])
    pe, ge = orc.rel_l2(out[s], d)
    assert pe < 1e-6 and ge < 1e-5, (pe, ge)
