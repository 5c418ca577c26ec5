"""The stop path of the training kernel: waits that run out (a limit of no polls) are
reported, by the call or, if it did not wait for its loss, by the next one; the parameters
stay as they are; and with the default limit again the same network trains as a new one."""
import os
import sys

import numpy as np
import pytest

from simulation_project_gb300 import lib
from simulation_project_gb300.learned import Mlp
from simulation_project_gb300.lib import DeviceArray
from simulation_project_gb300.types import MpsError

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [100, 20_000])
def test_training_waits_that_run_out(rows):
    rng = np.random.default_rng(rows)
    X, T = rng.normal(0, 1, (rows, 12)).astype(np.float32), rng.normal(0, 1, (rows, 2)).astype(np.float32)
    dX, dT, g = DeviceArray.from_host(X), DeviceArray.from_host(T), DeviceArray((mo.NPARAMS,), np.float32)
    m, fresh = Mlp(max_batch=rows, seed=3), Mlp(max_batch=rows, seed=3)
    before = m.params()
    try:
        Mlp.debug_wait_spins(0)
        with pytest.raises(MpsError):
            m.loss_grad(dX.ptr, dT.ptr, rows, g.ptr)
        with pytest.raises(MpsError):
            m.train_step(dX.ptr, dT.ptr, rows, 1e-3, want_loss=True)
        m.train_step(dX.ptr, dT.ptr, rows, 1e-3)
        lib.call("mps_device_sync")
        with pytest.raises(MpsError):
            m.train_step(dX.ptr, dT.ptr, rows, 1e-3)
        assert Mlp.tc_timeouts() != 0
    finally:
        Mlp.debug_wait_spins(-1)
    assert np.array_equal(m.params(), before)
    loss = m.loss_grad(dX.ptr, dT.ptr, rows, g.ptr)
    ref_loss, ref_g = mo.loss_grad(before.astype(np.float64), X, T)
    assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
    assert np.linalg.norm(g.download() - ref_g) <= 3e-2 * np.linalg.norm(ref_g)
    for net in (m, fresh):
        net.train_step(dX.ptr, dT.ptr, rows, 1e-3, want_loss=True)
    # Adam's first steps are about lr in size whatever the gradient's; sums in another order
    # can turn the sign of a vanishing one
    d = np.abs(m.params() - fresh.params())
    assert d.max() <= 2.1e-3 and d.mean() <= 2e-5
    m.close()
    fresh.close()
