"""SortUsingThrust's cooperative radix sort (k_sort) at the sizes and key ranges where it can
go wrong: one CTA and the first size with several, CTAs with ragged parts, more keys than a
tile per CTA holds, every number of passes (an odd one ends in the scratch arrays), digits
of 1 to 9 bits, the extremes of int, and sorts from several host threads."""
import threading

import numpy as np
import pytest

from simulation_project_gb300.lib import DeviceArray, call

pytestmark = pytest.mark.gpu


def _check(keys):
    vals = np.random.default_rng(1).integers(-2 ** 31, 2 ** 31, len(keys), dtype=np.int64).astype(np.int32)
    dk, dv = DeviceArray.from_host(keys), DeviceArray.from_host(vals)
    call("SortUsingThrust", len(keys), dk.ptr, dv.ptr)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.download(), keys[order])
    assert np.array_equal(dv.download(), vals[order])


@pytest.mark.parametrize("n", [2, 31, 511, 513, 4095, 4096, 4097, 5000, 155648, 155649, 882080, 933888, 933889, 2000003])
def test_sizes(n):
    _check(np.random.default_rng(n).integers(0, 85184, n, dtype=np.int64).astype(np.int32))


@pytest.mark.parametrize("bits", [1, 2, 8, 9, 10, 17, 18, 19, 26, 27, 28, 32])
@pytest.mark.parametrize("n", [3000, 70001])
def test_key_ranges(n, bits):
    keys = np.random.default_rng(bits).integers(0, 2 ** bits, n, dtype=np.int64) - 2 ** (bits - 1)
    keys[:2] = -2 ** (bits - 1), 2 ** (bits - 1) - 1
    _check(keys.astype(np.int32))


@pytest.mark.parametrize("n", [4096, 200000])
def test_sorted_reversed_and_equal_keys(n):
    k = np.arange(n, dtype=np.int32)
    _check(k)
    _check(k[::-1].copy())
    _check(np.full(n, -7, np.int32))
    _check(np.repeat(np.array([5, 3], np.int32), n // 2))


def test_host_threads_take_turns():
    errors = []

    def work(seed):
        try:
            for k in range(5):
                _check(np.random.default_rng(10 * seed + k).integers(-1000, 90000, 30000 + 7001 * seed,
                                                                     dtype=np.int64).astype(np.int32))
        except Exception as e:   # noqa: BLE001 (reported by the test's own thread)
            errors.append(e)
    ts = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
