"""Triangle cells, wall distance and drag of the reference-named launchers where their
kernels can go wrong, bit for bit against the oracle: few large triangles (32 lanes walk
one) and many small ones (8 lanes), cells at their capacity, cells filled in two calls,
numbers of particles around a warp's share, and calls on several streams at once."""
import ctypes as C

import numpy as np
import pytest

import orc
from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import call

pytestmark = pytest.mark.gpu
ORC = orc.oracle()


def _state(tris, n_side=9, seed=0, n=None):
    sc = scenes.random_block(n_side, seed=seed, with_box=False)
    pos = sc.pos if n is None else sc.pos[:n]
    out = scenes._finish("walls", sc.param, pos, np.asarray(tris), np.zeros(len(tris), np.int32),
                         [scenes._tri_normal_params(dt=sc.param.Dt, is_drag=True)], [], seed, 0.01)
    out.vel = np.random.default_rng(seed).normal(0, 0.2, out.pos.shape)
    d = scenes.DragParameter()
    d.DragToken, d.InputVelocityToken1 = b"E", b"V"
    d.CoefficientofInflueneRegion, d.VelocityIndex, d.VelocityExponential = 1.0, 1e-4, 1.0
    d.VelocityDragPermiabilityConstant = 1.0
    out.drag = [d]
    return orc.RefState(out)


def _spheres(count, radius, subdiv, seed=0):
    rng = np.random.default_rng(seed)
    return np.concatenate([scenes.icosphere(rng.uniform(0.0, 0.09, 3), radius, subdiv) for _ in range(count)])


def _oracle(st, register=1):
    b = st.bindings()
    orc.ref_topology(ORC, st, b)
    ORC.reset_triangle_topology(st.cells_n, orc.ptr(st.cells))
    for k in range(register):
        # the second call registers the last half of the triangles again
        first = 0 if k == 0 else st.t // 2
        ORC.register_triangle_topology(C.byref(b), orc.ptr(st.triangles[first:]), st.t - first, orc.ptr(st.cells),
                                       st.cells_n)
    ORC.calc_stl_distance(C.byref(b), st.n)
    ORC.calc_drag_effect(C.byref(b), st.n)


def _gpu(st, g, register=1):
    s = g.stream.ref()
    g.bind()
    call("ResetTriangleTopology", s, st.cells_n, g.p("cells"))
    for k in range(register):
        first = 0 if k == 0 else st.t // 2
        call("RegisterTriangleTopology", s, g.p("triangles") + first * st.triangles.itemsize, st.t - first, g.p("cells"),
             st.cells_n)
    call("CalcSTLDistance", s, st.n)
    call("CalcDragEffect", s, st.n)


def _same(st, g):
    got = g.download()
    for k in ("cells", "stl_distance", "stl_id", "drag_acc", "out_type", "magnifier_count"):
        assert getattr(st, k).tobytes() == got[k].tobytes(), k


CASES = {
    "box": lambda: scenes.box_triangles((-0.005, -0.005, -0.005), (0.095, 0.095, 0.1)),
    "huge": lambda: scenes.box_triangles((-3.0, -2.0, -4.0), (3.0, 2.5, 4.0)),
    "spheres": lambda: _spheres(6, 0.03, 1),
    "many_small": lambda: _spheres(30, 0.02, 2),          # 9,600 triangles
    "full_cells": lambda: _spheres(12, 0.02, 2, seed=1),  # more than 100 in a cell
}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("register", [1, 2])
def test_walls(case, register):
    import gpu_ref
    st = _state(CASES[case]())
    g = gpu_ref.GpuRef(st)
    g.topology(st.n)
    _gpu(st, g, register)
    g.stream.sync()
    got = g.download()
    if register == 1:
        _oracle(st)
        _same(st, g)
    else:
        # ids of the second call are counted from its own first triangle
        _oracle(st, register)
        assert st.cells.tobytes() == got["cells"].tobytes()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 127, 129])
def test_few_particles(n):
    import gpu_ref
    st = _state(_spheres(4, 0.03, 1), n=n)
    g = gpu_ref.GpuRef(st)
    g.topology(st.n)
    _gpu(st, g)
    g.stream.sync()
    _oracle(st)
    _same(st, g)


def test_several_streams():
    """Three sets, each with a stream of its own, their calls in turn and no waits between:
    the library's scratch serves one after the other."""
    import gpu_ref
    sets = [_state(_spheres(6 + 9 * k, 0.02, 2, seed=k), seed=k) for k in range(3)]
    gs = [gpu_ref.GpuRef(st) for st in sets]
    for st, g in zip(sets, gs):
        g.bind()
        g.topology(st.n)
        _oracle(st)
    for _ in range(20):
        for st, g in zip(sets, gs):
            _gpu(st, g)
    for st, g in zip(sets, gs):
        g.stream.sync()
        _same(st, g)
