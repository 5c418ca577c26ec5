"""SortUsingThrust where a sort gets two CTAs per SM: the number of keys from which it does,
several tiles per CTA, ragged ends, one to four passes, and keys in order, in reverse and equal."""
import numpy as np
import pytest

from test_gpu_sort import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2_499_999, 2_500_000, 2_500_001, 3_178_892, 6_000_007])
@pytest.mark.parametrize("bits", [7, 17, 30])
def test_random(n, bits):
    _check(np.random.default_rng(n + bits).integers(-2 ** (bits - 1), 2 ** (bits - 1), n, dtype=np.int64).astype(np.int32))


def test_ordered_and_equal_keys():
    n = 2_600_003
    k = (np.arange(n) // 10).astype(np.int32)
    _check(k)
    _check(k[::-1].copy())
    _check(np.full(n, 5, np.int32))
    _check((k + np.random.default_rng(0).integers(-3, 4, n)).astype(np.int32))
