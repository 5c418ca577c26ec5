"""The reference-named pair operators in sparse fluid (rp_sparse, k_ref_walk), bit for bit
against the oracle: the size from which a call asks, the sizes at which another kernel would
take it, fluid on both sides of the line, a grid too thin for 27 different cells, particles
to be skipped or far outside, and a last CTA of one target."""
import numpy as np
import pytest

from test_gpu_ref_pairs import L0, ORC, SLICE_OPS, _block, _compare, _scene

pytestmark = pytest.mark.gpu


def _cloud(n, density, seed):
    side = (n / density) ** (1.0 / 3.0) * L0
    return np.random.default_rng(seed).uniform(0.0, side, (n, 3))


@pytest.mark.parametrize("density", [0.003, 0.03, 0.12, 0.25])
@pytest.mark.parametrize("n", [16383, 16384, 20001, 40001, 64003, 100097])
def test_clouds(n, density):
    _compare(_scene(_cloud(n, density, n), n))


@pytest.mark.parametrize("shape,spacing", [((150, 1, 150), 3.0), ((30, 30, 30), 3.0)], ids=["layer", "lattice"])
def test_lattices(shape, spacing):
    _compare(_scene(_block(shape, spacing, seed=1), 1))


@pytest.mark.parametrize("far", [3e18, 1e19, np.inf, np.nan])
def test_skipped_and_far_particles(far):
    sc = _scene(_cloud(41_000, 0.03, 2), 2)

    def setup(st):
        rng = np.random.default_rng(3)
        away = rng.choice(st.n, 40, replace=False)
        st.out_pos[away[:20], 0] = far
        st.out_pos[away[20:], 2] = -far
        st.out_id[away] = -1
        st.out_id[rng.choice(st.n, 4000, replace=False)] = -1
    _compare(sc, setup)


def test_all_particles_far_outside():
    """Nothing to sample: every position is a NaN."""
    sc = _scene(_cloud(20_000, 0.03, 4), 4)

    def setup(st):
        st.out_pos[:] = np.nan
        st.out_id[:] = -1
    _compare(sc, setup, ops=SLICE_OPS)


@pytest.mark.parametrize("n", [194_560, 291_853])
@pytest.mark.parametrize("density", [0.03, 0.8])
def test_turbulence_groups_in_turn(density, n):
    """Two and three groups per warp, the last CTA with fewer; the walk beside it."""
    _compare(_scene(_cloud(n, density, 6), 6), ops=[("CalcTurbulenceViscosity", ORC.calc_turbulence_viscosity)])


@pytest.mark.parametrize("n", [215_999, 216_000, 216_001])
def test_predictor_takeover(n):
    """Eight targets per warp, then a lane per target, in dense fluid."""
    _compare(_scene(_block((61, 60, 60), seed=5)[:n], 5), ops=[("CalcExplicitly", ORC.calc_explicitly)])
