"""Wall distance and drag of many particles with few triangles (a lane per particle for short
lists, the marked rest by warps), bit for bit against the oracle: the number of particles
from which that route is taken, last CTAs of a few particles, no triangle near, lists around
the length at which a particle is left to the warps, full cells, and particles that are gone,
without a cell or not numbers."""
import numpy as np
import pytest

import gpu_ref
import orc
from simulation_project_gb300 import scenes
from test_gpu_ref_walls import _gpu, _oracle, _same, _state

pytestmark = pytest.mark.gpu


def _spheres(count, radius, subdiv, spread, seed=0):
    rng = np.random.default_rng(seed)
    return np.concatenate([scenes.icosphere(rng.uniform(0.1, 0.1 + spread, 3), radius, subdiv) for _ in range(count)])


def _check(st):
    g = gpu_ref.GpuRef(st)
    g.topology(st.n)
    _gpu(st, g)
    g.stream.sync()
    _oracle(st)
    _same(st, g)
    return st


@pytest.mark.parametrize("n", [63999, 64000, 64001, 64127, 64800])
def test_takeover(n):
    st = _check(_state(scenes.box_triangles((-0.005,) * 3, (0.405, 0.405, 0.41)), n_side=41, n=n))
    assert (st.stl_id >= 0).any() and (st.stl_id < 0).any()


# lists of a few entries, around 32, of hundreds, and cells at their 100
@pytest.mark.parametrize("tris", [lambda: _spheres(1, 0.03, 0, 0.1), lambda: _spheres(4, 0.03, 1, 0.1),
                                  lambda: _spheres(7, 0.02, 1, 0.02), lambda: _spheres(2, 0.02, 2, 0.0)],
                         ids=["20", "320", "560_close", "640_full_cells"])
def test_list_lengths(tris):
    t = tris()
    st = _check(_state(t, n_side=41))
    held = st.cells["m_TriangleNum"]
    assert len(t) * 100 <= st.n and held.max() >= min(len(t), 4)
    assert (st.stl_id >= 0).any() and (st.stl_id < 0).any()


# 200 particles for every triangle, and one fewer: lists of up to 64 and of up to 32 entries
@pytest.mark.parametrize("n", [64000, 64199, 64257])
@pytest.mark.parametrize("more", [0, 1])
def test_the_longer_short_lists(n, more):
    t = np.concatenate([_spheres(4, 0.05, 1, 0.1), np.asarray(_spheres(1, 0.05, 0, 0.1))])[:n // 200 + more]
    st = _check(_state(t, n_side=41, n=n))
    assert (st.stl_id >= 0).any() and (st.stl_id < 0).any()


# from 600,000 particles on 50 for every triangle are enough, from 2,000,000 on for longer lists
@pytest.mark.parametrize("n,balls", [(599_999, 100), (600_000, 100), (600_033, 149), (600_033, 151), (2_000_021, 260)])
def test_many_particles(n, balls):
    st = _check(_state(_spheres(balls, 0.03, 1, 0.8), n_side=127 if n > 700_000 else 85, n=n))
    assert (st.stl_id >= 0).any() and (st.stl_id < 0).any()


def test_no_triangles_near():
    _check(_state(np.asarray(_spheres(2, 0.02, 0, 0.1)) + 0.8, n_side=41))


@pytest.mark.parametrize("far", [3e18, np.inf, np.nan])
def test_particles_without_a_cell(far):
    st = _state(_spheres(4, 0.03, 1, 0.1), n_side=41)
    rng = np.random.default_rng(1)
    away = rng.choice(st.n, 200, replace=False)
    st.out_pos[away[:100], 0] = far
    st.out_pos[away[100:], 2] = -far
    st.out_id[rng.choice(st.n, 3000, replace=False)] = -2   # gone: the drag passes them by
    _check(st)
