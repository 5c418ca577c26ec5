"""Grid barriers whose wait runs out (a limit of no polls): the call reports it, nothing is
read or written out of range, and with the default limit again the same solver gives what a
new one does."""
import ctypes as C

import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import call
from simulation_project_gb300.solver import Solver, _lib
from simulation_project_gb300.types import MpsError

pytestmark = pytest.mark.gpu
STAGE_TIMEOUT = 32
OPT = {"cg_max_iter": 200, "compressibility": 1e-6}   # a few iterations per pass


class no_polls:
    def __enter__(self):
        call("mps_debug_barrier_polls", 0)

    def __exit__(self, *_):
        call("mps_debug_barrier_polls", -1)


def _block(shape, l0=0.004):
    p = scenes.default_param(l0, 1e-4)
    p.FreeSurfaceThreshold = 0.3
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3) * l0
    g = g + np.random.default_rng(0).uniform(-0.02 * l0, 0.02 * l0, g.shape)
    return scenes._finish("block", p, g, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)], [],
                          0, l0)


def _reset(s):
    """The scene's particles again, as at creation."""
    a = [np.ascontiguousarray(x, t) for x, t in ((s.scene.pos, np.float64), (s.scene.vel, np.float64),
                                                 (s.scene.press, np.float64), (s.scene.visc, np.float64),
                                                 (s.scene.ptype, np.int32))]
    assert _lib().mps_solver_set_particles(s.h, s.scene.n, *[x.ctypes.data for x in a]) == 0


def _three_steps(s):
    st = [s.step(i) for i in range(3)]
    assert all(q["error_flags"] == 0 for q in st)
    return [q["cg_iterations"] for q in st], s.state()


# up to 4,096 particles, whose sort has no barrier: the small system's CG (1,716 rows, 54 CTAs)
# and, in a profiling solver, the coarse V-cycle (a strip of 128 cells and more: two levels)
@pytest.mark.parametrize("shape,profile", [((13, 12, 11), 0), ((2, 4, 512), 1)], ids=["small_cg", "coarse_cycle"])
def test_solve_after_a_barrier_ran_out(shape, profile):
    sc = _block(shape)
    fresh = Solver(sc, precision="fp32_ir", profile=profile, **OPT)
    want = _three_steps(fresh)
    fresh.close()
    s = Solver(sc, precision="fp32_ir", profile=profile, **OPT)
    for _ in range(3):
        with no_polls():
            try:
                st = s.step(0)
                assert st["error_flags"] & STAGE_TIMEOUT and st["mg_levels"] >= 2
            except MpsError:
                assert not profile
            else:
                assert profile
        _reset(s)
    its, state = _three_steps(s)
    s.close()
    assert its == want[0]
    for k in ("pos", "vel", "press"):
        assert np.array_equal(state[k], want[1][k]), k
