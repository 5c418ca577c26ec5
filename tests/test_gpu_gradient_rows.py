"""Gradient rows of the FP32 list pass (k_list) where they fill up and run over: each holds
the first 64 neighbours within the gradient radius in candidate order, whichever of the
slice's two warps listed them, as the walk without lists (rows_sell = 1) writes them."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu
NEIGHBOUR_CAP = 2   # MPS_ERR_NEIGHBOUR_CAP


def _clumps(sizes, l0=0.01):
    """Clumps 20 l0 apart, the particles of each within 1.8 l0 of one another."""
    rng = np.random.default_rng(sum(sizes))
    pos = []
    for k, m in enumerate(sizes):
        d = rng.normal(size=(m, 3))
        r = 0.9 * l0 * rng.uniform(0.0, 1.0, (m, 1)) ** (1.0 / 3.0)
        pos.append(d / np.linalg.norm(d, axis=1, keepdims=True) * r + [20 * l0 * k, 3.3 * l0, 0.7 * l0 * k])
    p = scenes.default_param(l0, 1e-4)
    sc = scenes._finish("clumps", p, np.concatenate(pos), np.zeros((0, 3, 3)), np.zeros(0, np.int32),
                        [scenes._tri_normal_params(dt=p.Dt)], [], 0, l0)
    sc.vel = rng.normal(0.0, 0.05, sc.pos.shape)
    return sc


def _step(sc, variant):
    s = Solver(sc, precision="fp32_ir", rows_sell=variant, cg_max_iter=200)
    st = s.step(0)
    a = s.state()
    s.close()
    return st["error_flags"], np.concatenate([a["pos"], a["vel"], a["press"][:, None]], 1)


@pytest.mark.parametrize("sizes", [(64, 65), (66,), (80, 66, 130), (200,), (100,) * 7], ids=str)
def test_full_gradient_rows(sizes):
    sc = _clumps(sizes)
    flags, want = _step(sc, 1)
    assert bool(flags & NEIGHBOUR_CAP) == (max(sizes) > 65)
    for _ in range(5):
        f, got = _step(sc, 0)
        assert f == flags and got.tobytes() == want.tobytes()
