"""SortUsingThrust where a sort gets two CTAs per SM: the number of keys from which it does,
several tiles per CTA, ragged ends, one to four passes, and keys in order, in reverse and equal."""
import numpy as np
import pytest

from simulation_project_gb300.lib import DeviceArray, call
from simulation_project_gb300.types import MpsError
from test_gpu_barrier_timeouts import no_polls
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


def test_a_sort_that_gives_up():
    """Reported, and the next one is right."""
    keys = np.random.default_rng(1).integers(0, 2 ** 24, 2_600_003).astype(np.int32)
    dk, dv = DeviceArray.from_host(keys), DeviceArray.from_host(np.arange(len(keys), dtype=np.int32))
    with no_polls(), pytest.raises(MpsError):
        call("SortUsingThrust", len(keys), dk.ptr, dv.ptr)
    _check(keys)
