"""Block capacities of the device memory pool (no GPU needed): blocks that can be kept are rounded up to a few sizes,
blocks too large to be kept (over 512 MiB) are allocated at their own size."""
import ctypes

import pytest


def _capacity(n):
    from exafmm import _lib
    fn = getattr(_lib.lib(), "_ZN4xfmm13pool_capacityEm")  # xfmm::pool_capacity(size_t)
    fn.restype, fn.argtypes = ctypes.c_size_t, [ctypes.c_size_t]
    return fn(n)


@pytest.mark.parametrize("n", [1, 511, 512, 513, 8191, 8193, 100001, (1 << 20) + 1, (300 << 20) + 7, 500 << 20])
def test_kept_sizes_are_rounded_by_at_most_an_eighth(n):
    c = _capacity(n)
    assert n <= c <= max(512, n + n // 8 + 512) and c % 512 == 0
    assert _capacity(c) == c


@pytest.mark.parametrize("n", [(512 << 20) + 1, (513 << 20), 5 * (1 << 30) + 3, 70 * (1 << 30) + 12345])
def test_blocks_that_are_never_kept_have_their_own_size(n):
    assert _capacity(n) == n
