"""The pair sums of the reference-named operators (k_ref_pairs, k_ref_lanes) where they can
go wrong, bit for bit against the oracle: numbers of targets around a warp's share, warps
whose targets lie in many cells, grids too thin to skip cells, particles to be skipped or
far outside, the sizes at which another kernel takes over, and arrays that 16-byte loads
cannot read."""
import ctypes as C

import numpy as np
import pytest

import orc
from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import DeviceArray, call

pytestmark = pytest.mark.gpu
ORC = orc.oracle()
L0 = 0.01


def _scene(pos, seed, zone=None):
    p = scenes.default_param(L0, 1e-4, explicit_pressure=True, sonic=10.0)
    p.ArtificialPressure, p.r_coeff = 1e-3, 1.0
    zone = zone or (None, None)
    sc = scenes._finish("points", p, np.asarray(pos, np.float64), np.zeros((0, 3, 3)), np.zeros(0, np.int32),
                        [scenes._tri_normal_params(dt=p.Dt)], [], seed, L0, *zone)
    rng = np.random.default_rng(seed)
    sc.vel = rng.normal(0, 0.05, sc.pos.shape)
    sc.press = np.abs(rng.normal(0, 50.0, sc.n))
    orc.thermal_scene(sc, seed)
    orc.turbulent_scene(sc, seed)
    sc.param.Dt = 1e-4
    return sc


def _block(shape, spacing=1.0, jitter=0.3, seed=0):
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3) * spacing * L0
    return g + np.random.default_rng(seed).uniform(-jitter * L0, jitter * L0, g.shape)


def _thin():
    pos = _block((9, 9, 9))
    lo, hi = pos.min(0) - 0.5 * L0, pos.max(0) + 0.5 * L0
    return pos, (lo, hi)   # a zone without room around it: three cells along each axis, buffers aside


def _bound(g, st, pos_ptr=None):
    g.bind()
    if pos_ptr:
        call("InitializeDeviceConstInputParticles", g.p("id"), pos_ptr, *[g.p(k) for k in
             ["vel", "pressure", "density", "temperature", "kin_visc", "solid_rate", "type", "turb_visc", "strain"]])


def _bits(a):
    """Bytes of an array, every NaN the same one (the CPU's and the GPU's differ)."""
    return (np.where(np.isnan(a), np.float32(np.nan), a) if a.dtype.kind == "f" else a).tobytes()


def _compare(sc, setup=None, ops=None, misaligned=False):
    st = orc.RefState(sc)
    st.out_temperature[:st.n] = np.random.default_rng(3).uniform(295, 325, st.n).astype(np.float32)
    if setup:
        setup(st)
    import gpu_ref
    g = gpu_ref.GpuRef(st)
    shifted = DeviceArray((3 * st.n + 1,), np.float32) if misaligned else None
    _bound(g, st, shifted.ptr + 4 if misaligned else None)
    b = st.bindings()
    orc.ref_topology(ORC, st, b)
    ORC.calc_stl_distance(C.byref(b), st.n)
    g.topology(st.n)
    g.run("CalcSTLDistance", st.n)
    for name, f in ops or [("CalcTemperatureFactor", ORC.calc_temperature_factor),
                           ("CalcTurbulenceViscosity", ORC.calc_turbulence_viscosity),
                           ("CalcExplicitly", ORC.calc_explicitly),
                           ("CalcExplicitPressure", ORC.calc_explicit_pressure),
                           ("CalcExplicitPressureGradient", ORC.calc_explicit_pressure_gradient)]:
        f(C.byref(b), st.n)
        g.run(name, st.n)
        got = g.download()
        for k in ("turb_visc", "strain", "out_temperature", "out_kin_visc", "pressure", "out_pressure", "out_density",
                  "out_pos", "out_vel", "out_id"):
            assert _bits(getattr(st, k)) == _bits(got[k]), (name, k)
    return st


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 33, 500])
def test_few_targets(n):
    _compare(_scene(_block((8, 8, 8), seed=n)[:n], n))


@pytest.mark.parametrize("shape,spacing", [((14, 13, 12), 3.0), ((25, 1, 25), 1.0), ((28, 28, 27), 1.0),
                                           ((32, 30, 29), 1.7), ((5, 5, 5), 0.2)],
                         ids=["sparse", "layer", "eight_per_warp", "eight_per_warp_sparse", "crowded_cell"])
def test_shapes(shape, spacing):
    _compare(_scene(_block(shape, spacing, seed=1), 1))


def test_thin_grid():
    pos, zone = _thin()
    _compare(_scene(pos, 2, zone))


@pytest.mark.parametrize("far", [1e17, 3e18, 1e19, 3e38, np.inf, np.nan])
def test_skipped_and_far_particles(far):
    sc = _scene(_block((12, 11, 10), seed=4), 4)

    def setup(st):
        rng = np.random.default_rng(5)
        away = rng.choice(st.n, 6, replace=False)
        st.out_pos[away[:3], 0] = far
        st.out_pos[away[3:], 2] = -far
        st.out_id[away] = -1   # they are outside the zone: the operators mark them so anyway
        st.out_id[rng.choice(st.n, 40, replace=False)] = -1
    _compare(sc, setup)


@pytest.mark.parametrize("misaligned", [False, True])
def test_predictor_with_a_lane_per_target(misaligned):
    _compare(_scene(_block((67, 67, 67), seed=6), 6), ops=[("CalcExplicitly", ORC.calc_explicitly)], misaligned=misaligned)


def test_turbulence_with_four_targets_per_warp():
    _compare(_scene(_block((47, 47, 46), seed=7), 7),
             ops=[("CalcTurbulenceViscosity", ORC.calc_turbulence_viscosity)])


SLICE_OPS = [("CalcTemperatureFactor", ORC.calc_temperature_factor), ("CalcExplicitPressure", ORC.calc_explicit_pressure),
             ("CalcExplicitPressureGradient", ORC.calc_explicit_pressure_gradient)]


@pytest.mark.parametrize("shape,spacing,n", [((35, 35, 33), 1.0, 40001), ((36, 34, 33), 1.7, None), ((200, 1, 201), 1.0, None),
                                             ((36, 34, 33), 0.6, 40030)], ids=["ragged", "sparse", "layer", "crowded"])
def test_slices_of_32_targets(shape, spacing, n):
    """k_ref_slices: a last slice of one target, slices over many cells, lists emptied within a
    round, cells of a few and of 300 particles."""
    _compare(_scene(_block(shape, spacing, seed=8)[:n], 8), ops=SLICE_OPS)


@pytest.mark.parametrize("far", [3e18, 1e19, np.inf, np.nan])
def test_slices_with_skipped_and_far_particles(far):
    sc = _scene(_block((36, 35, 32), seed=9), 9)

    def setup(st):
        rng = np.random.default_rng(10)
        away = rng.choice(st.n, 40, replace=False)
        st.out_pos[away[:20], 0] = far
        st.out_pos[away[20:], 2] = -far
        st.out_id[away] = -1
        st.out_id[rng.choice(st.n, 400, replace=False)] = -1
    _compare(sc, setup, ops=SLICE_OPS)
