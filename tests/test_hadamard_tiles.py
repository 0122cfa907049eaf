"""The mixed path's M2L Hadamard (k_hadamard_h: tiles of up to 512 targets with their sources in shared
memory, FP16 head/tail operands on the exponents of their sources) against the FP64 path on the same
tree: tile sizes from a few targets (positions split over the warps) to several full tiles, trees whose
tiles close early, and charges whose scale or range stresses the exponents.

Tolerance: the mixed path's bound against FP64 results at low orders, 5e-6 relative L2; scaling all
charges by a power of two scales every step exactly, up to the order of the FP64 atomic sums of the close
pairs (1e-14)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 5e-6


def _points(kind, n, rng):
    if kind == "cube":
        return rng.random((n, 3))
    g = rng.standard_normal((n, 3))
    g /= np.linalg.norm(g, axis=1)[:, None]
    return g if kind == "sphere" else g * (0.02 + rng.random(n) ** 4)[:, None]


def _solve(x, q, p, ncrit, precision, kernel="laplace"):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import exafmm.laplace as lap
    import exafmm.modified_helmholtz as yuk
    m = lap if kernel == "laplace" else yuk
    fmm = m.LaplaceFmm(p, ncrit, precision=precision) if kernel == "laplace" else \
        m.ModifiedHelmholtzFmm(p, ncrit, 5.0, precision=precision)
    t = m.setup(m.init_sources(x, q), m.init_targets(x), fmm)
    return m.evaluate(t, fmm)


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kind,n,p,ncrit,kernel", [
    ("cube", 600, 4, 32, "laplace"),            # a handful of targets: one group, positions over 8 warps
    ("cube", 9000, 4, 16, "laplace"),           # 73 targets: two groups
    ("cube", 30000, 3, 20, "laplace"),          # a full tile and a remainder
    ("cube", 120000, 2, 16, "laplace"),         # full volumes: 512 targets and about 1000 sources per tile
    ("sphere", 60000, 4, 20, "laplace"),        # surface: half-occupied positions
    ("cluster", 60000, 4, 20, "laplace"),       # deep adaptive tree
    ("cluster", 30000, 4, 20, "modified_helmholtz"),  # one group per level
])
def test_mixed_matches_fp64(kind, n, p, ncrit, kernel):
    rng = np.random.default_rng(n + p)
    x, q = _points(kind, n, rng), rng.uniform(-1, 1, n)
    ref = _solve(x, q, p, ncrit, "fp64", kernel)
    out = _solve(x, q, p, ncrit, "mixed", kernel)
    assert _rel(out[:, 0], ref[:, 0]) < TOL and _rel(out[:, 1:], ref[:, 1:]) < TOL


@pytest.mark.parametrize("exponent", [-60, 60])
def test_power_of_two_charges_scale_exactly(exponent):
    rng = np.random.default_rng(3)
    x, q = rng.random((20000, 3)), rng.uniform(-1, 1, 20000)
    a = _solve(x, q, 4, 32, "mixed")
    b = _solve(x, q * 2.0 ** exponent, 4, 32, "mixed") * 2.0 ** -exponent
    assert _rel(b, a) < 1e-14


def test_charges_of_very_different_size():
    """Charges 10^6 smaller in one half: both halves keep the mixed path's accuracy, in a field that the large
    charges rule in both (test_hadamard_range.py looks at weak charges alone)."""
    rng = np.random.default_rng(4)
    x, q = rng.random((40000, 3)), rng.uniform(-1, 1, 40000)
    q[x[:, 0] < 0.5] *= 1e-6
    ref, out = _solve(x, q, 4, 32, "fp64"), _solve(x, q, 4, 32, "mixed")
    for half in (x[:, 0] < 0.5, x[:, 0] >= 0.5):
        assert _rel(out[half], ref[half]) < TOL
