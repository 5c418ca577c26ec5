"""Grid barriers whose wait runs out (a limit of no polls): the call reports it, nothing is
read or written out of range, and with the default limit again the same solver gives what a
new one does."""
import ctypes as C

import numpy as np
import pytest

import gpu_ref
import orc
from simulation_project_gb300 import lib, scenes
from simulation_project_gb300.lib import DeviceArray, call
from simulation_project_gb300.solver import Solver, _lib
from simulation_project_gb300.types import CTriangleParameters, MpsError

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
    if s.scene.t:
        v = np.ascontiguousarray(s.scene.tri_vertices.reshape(-1, 9))
        tp = (CTriangleParameters * len(s.scene.tri_params))(*s.scene.tri_params)
        assert _lib().mps_solver_set_triangles(s.h, s.scene.t, v.ctypes.data, s.scene.tri_model.ctypes.data,
                                               len(s.scene.tri_params), C.addressof(tp)) == 0


def _three_steps(s):
    st = [s.step(i) for i in range(3)]
    assert all(q["error_flags"] == 0 for q in st)
    return [q["cg_iterations"] for q in st], s.state()


def _same(a, b):
    assert a[0] == b[0]
    for k in ("pos", "vel", "press"):
        assert np.array_equal(a[1][k], b[1][k]), k


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
    got = _three_steps(s)
    s.close()
    _same(got, want)


@pytest.mark.parametrize("precision", ["fp32_ir", "fp64"])
@pytest.mark.parametrize("scene", [lambda: _block((24, 24, 23)), lambda: scenes.dam_break(l0=0.01),
                                   lambda: scenes.rotating_bucket(l0=0.008, n_drag=4)],
                         ids=["no_walls", "resting_walls", "moving_walls"])
def test_step_after_a_sort_gave_up(scene, precision):
    """The sorts of the particles and of the wall bins (over 4,096 keys each): the step fails
    with an error, and so does the next as long as the limit holds."""
    sc = scene()
    fresh = Solver(sc, precision=precision)
    if sc.t:
        assert sum(map(len, fresh.debug_wall_bins().values())) > 4096
    want = _three_steps(fresh)
    fresh.close()
    s = Solver(sc, precision=precision)
    for first in (True, False):   # as a solver's first step, and after good ones
        with no_polls():
            for _ in range(2):
                with pytest.raises(MpsError):
                    s.step(0)
            with pytest.raises(MpsError):
                s.pressure()
        _reset(s)
        if first:
            _three_steps(s)
    got = _three_steps(s)
    s.close()
    _same(got, want)


def test_wall_bins_alone_after_a_sort_gave_up():
    sc = scenes.dam_break(l0=0.01)
    s, fresh = Solver(sc, precision="fp32_ir"), Solver(sc, precision="fp32_ir")
    with no_polls(), pytest.raises(MpsError):
        s.debug_wall_bins()
    assert s.debug_wall_bins() == fresh.debug_wall_bins()


def test_sorts_that_give_up():
    """SortUsingThrust and its variant without allocation report it and work again afterwards."""
    keys = np.random.default_rng(0).integers(-10 ** 6, 10 ** 6, 50_000).astype(np.int32)
    order = np.argsort(keys, kind="stable")
    lib.load().SortUsingThrustNoAlloc.argtypes = [C.c_int, C.c_void_p, C.c_void_p]
    for name in ("SortUsingThrust", "SortUsingThrustNoAlloc"):
        dk, dv = DeviceArray.from_host(keys), DeviceArray.from_host(np.arange(len(keys), dtype=np.int32))
        with no_polls(), pytest.raises(MpsError):
            call(name, len(keys), dk.ptr, dv.ptr)
        dk.upload(keys)
        dv.upload(np.arange(len(keys), dtype=np.int32))
        call(name, len(keys), dk.ptr, dv.ptr)
        assert np.array_equal(dk.download(), keys[order]) and np.array_equal(dv.download(), order)


def test_triangle_cells_whose_sort_gave_up():
    """The cells hold no triangle then (not stale or half sorted ones); the wall launchers
    report it until the next RegisterTriangleTopology has, and the one after works."""
    st = orc.RefState(scenes.rotating_bucket(l0=0.008, n_drag=4))
    g = gpu_ref.GpuRef(st)
    g.topology(st.n)
    s = g.stream.ref()
    g.walls()
    want = g.download()["cells"]
    assert want["m_TriangleNum"].sum() > 4096
    with no_polls():
        g.walls()
        got = g.download()["cells"]
        assert not got["m_TriangleNum"].any()
        for name in ("CalcSTLDistance", "CalcDragEffect"):
            with pytest.raises(MpsError):
                call(name, s, st.n)
    keys = DeviceArray.from_host(np.array([3, 1, 2], np.int32))
    call("SortUsingThrust", 3, keys.ptr, DeviceArray.from_host(np.zeros(3, np.int32)).ptr)   # its own sort was fine
    with pytest.raises(MpsError):
        g.walls()
    g.walls()
    got = g.download()["cells"]
    assert np.array_equal(got["m_TriangleNum"], want["m_TriangleNum"])
    for name in ("CalcSTLDistance", "CalcDragEffect"):
        g.run(name, st.n)
