"""Wall distance of the step where eight warps share 32 particles' triangle lists: lists of
fewer triangles than a round takes, just as many, more, and of several hundred, particle
counts around a CTA's 32, and particles without a list, against the FP64 pass (a lane per
particle) through the wall's part of the particle number density."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu
L0 = 0.01


def _scene(n, m, seed=0):
    """n particles above a floor of m x m squares of two triangles."""
    p = scenes.default_param(L0, 1e-4)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * L0
    pos = g + np.random.default_rng(seed).uniform(-0.2 * L0, 0.2 * L0, g.shape)
    e = np.linspace(-0.5 * L0, (side - 0.5) * L0, m + 1)
    tris = []
    for a in range(m):
        for b in range(m):
            c = [(e[a + i], e[b + j], -0.6 * L0) for i, j in ((0, 0), (1, 0), (1, 1), (0, 1))]
            tris += [(c[0], c[1], c[2]), (c[0], c[2], c[3])]
    return scenes._finish("floor", p, pos, np.asarray(tris), np.zeros(len(tris), np.int32), [scenes._tri_normal_params(dt=p.Dt)],
                          [], seed, L0)


@pytest.mark.parametrize("n,m", [(1, 1), (31, 2), (32, 4), (33, 4), (500, 5), (1700, 9), (1700, 24), (5000, 40)])
def test_wall_part_of_the_number_density(n, m):
    sc = _scene(n, m)
    pnd = []
    for precision in ("fp32_ir", "fp64"):
        s = Solver(sc, precision=precision)
        assert s.pressure()["error_flags"] == 0
        q = s.debug_ppe()
        pnd.append(q["pnd"][np.argsort(q["id"], kind="stable")])
        s.close()
    a, b = pnd
    near = sc.pos[:, 2] < 1.2 * L0
    assert near.any() and b[near].max() > 0.1
    # the distance is that of FP32 coordinates (a few roundings of the extent), the weight's
    # slope is at most 2.1 / 0.4^2 per l0, and the fluid part has its own 37 roundings
    extent = np.abs(sc.pos).max() + L0
    tol = 2.1 / 0.16 * 16 * 2.0 ** -24 * extent / L0 + 64 * 2.0 ** -24 * b.max() + 2e-5
    assert np.abs(a - b).max() <= tol


# 200 particles for every triangle, and fewer: a lane per particle, and eight warps for 32
@pytest.mark.parametrize("n,m", [(3599, 3), (3600, 3), (3601, 3), (4000, 1)])
def test_few_triangles(n, m):
    test_wall_part_of_the_number_density(n, m)
