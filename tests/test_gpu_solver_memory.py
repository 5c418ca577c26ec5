"""Device memory that a solver holds: the rows of the FP64 list pass belong to that precision."""
import ctypes as C

import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import call
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu

ROOM, ENTRIES = 200_000, 384   # particles that the solvers have room for; entries of a row
ROWS = 12 * ENTRIES * ROOM     # bytes of the rows: int column and double weight


def _free():
    call("mps_device_sync")
    free, total = C.c_size_t(), C.c_size_t()
    assert C.CDLL("libcuda.so.1").cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    return free.value


def test_fp64_rows_come_with_the_precision():
    sc = scenes.dam_break(l0=0.02)
    call("mps_set_device", 0)
    Solver(sc).close()   # the context and the kernels
    at = [_free()]
    a = Solver(sc, precision="fp32_ir", max_particles=ROOM, max_neighbours=ENTRIES, preconditioner=0)
    at.append(_free())
    a.set_precision("fp64")
    at.append(_free())
    a.set_precision("fp32_ir")
    a.set_precision("fp64")   # held by now
    at.append(_free())
    b = Solver(sc, precision="fp64", max_particles=ROOM, max_neighbours=ENTRIES, preconditioner=0)
    at.append(_free())
    fp32, switch, again, fp64 = (x - y for x, y in zip(at, at[1:]))
    page = 16 << 20   # what the allocator may round up
    assert abs(switch - ROWS) <= page and abs(again) <= page and abs(fp64 - fp32 - ROWS) <= page
    for i in range(2):
        assert a.step(i)["cg_relres"] <= 1e-8 and b.step(i)["cg_relres"] <= 1e-8
    sa, sb = a.state(), b.state()
    for k in ("id", "pos", "vel", "press"):
        assert np.array_equal(sa[k], sb[k]), k
    a.close()
    b.close()
