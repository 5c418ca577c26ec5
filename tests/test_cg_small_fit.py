"""Where the inner CG in one launch applies (host code, no GPU): the SMs' shared memory, the
slices per CTA, the preconditioner's sizes, and rows whose columns need no more than 16 bits."""
import pytest

from simulation_project_gb300.solver import _lib


def fit(rows, longest=256, sms=152, levels=0, aggregates=0):
    return _lib().mps_debug_cg_small_slices(rows, longest, sms, levels, aggregates)


def most(**kw):
    return max([n for n in range(32, 40000, 32) if fit(n, **kw)], default=0)


@pytest.mark.parametrize("kw,rows", [(dict(longest=240), 29184), (dict(longest=241), 24320), (dict(longest=256), 24320),
                                     (dict(longest=384), 19456), (dict(levels=1, aggregates=128), 24320),
                                     (dict(levels=2, aggregates=176), 24320), (dict(levels=2, aggregates=368), 19456),
                                     (dict(levels=2, aggregates=369), 14592)])
def test_largest_system(kw, rows):
    assert most(**kw) == rows


@pytest.mark.parametrize("rows,slices", [(0, 0), (1, 1), (32 * 152, 1), (32 * 152 + 1, 2), (24320, 5), (24321, 0)])
def test_slices(rows, slices):
    assert fit(rows) == slices


def test_columns_of_16_bits():
    """On more SMs the rows would fit beyond the reach of 16-bit columns: not used there."""
    assert fit(32768, longest=128, sms=300) > 0
    assert fit(32769, longest=128, sms=300) == 0


@pytest.mark.parametrize("levels,aggregates", [(3, 200), (2, 1025), (1, 1025)])
def test_preconditioners_that_do_not_fit(levels, aggregates):
    assert fit(2000, levels=levels, aggregates=aggregates) == 0
