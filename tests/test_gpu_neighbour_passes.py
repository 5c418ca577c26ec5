"""The FP32 neighbour passes (k_list, k_predict: a lane per target, candidates shared by the
slice's 32 targets) at the places where they can go wrong: fewer particles than a slice, a
ragged last slice, slices of many short pieces, runs too long for the 16-bit list entries,
rows longer than the list, cells smaller than the radius, and the size at which a warp
takes a whole slice of the predictor."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver
from simulation_project_gb300.types import grid_box

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _scene(pos, l0=0.01, coef=None, cells=None, seed=0, threshold=0.97, visc=1e-6):
    """Particles without walls; coef: Laplacian radius in l0, cells: cell size in l0."""
    p = scenes.default_param(l0, 1e-4)
    p.FreeSurfaceThreshold = threshold
    if coef:
        p.LaplacianInfluenceRadiusCoefficient = coef
    sc = scenes._finish("points", p, pos, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)],
                        [], seed, l0)
    if cells:
        radius = p.LaplacianInfluenceRadiusCoefficient
        p.LaplacianInfluenceRadiusCoefficient = cells
        z = sc.box.m_ComputeZone
        sc.box = grid_box([z.m_MinBound.x, z.m_MinBound.y, z.m_MinBound.z],
                          [z.m_MaxBound.x, z.m_MaxBound.y, z.m_MaxBound.z], p)
        p.LaplacianInfluenceRadiusCoefficient = radius
    sc.vel = np.random.default_rng(seed + 1).normal(0.0, 0.05, sc.pos.shape)
    sc.visc = np.full(sc.n, visc)
    return sc


def _block(side, l0=0.01, jitter=0.3, seed=0):
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * l0
    return g + np.random.default_rng(seed).uniform(-jitter * l0, jitter * l0, g.shape)


def _spray(n=1500, l0=0.01, seed=3):
    return np.random.default_rng(seed).uniform(0.0, 0.4, (n, 3)) * [1.0, 1.0, 0.2]


SCENES = {
    "27_targets": lambda: _scene(_block(3)),
    "ragged": lambda: _scene(_block(11)),
    "many_pieces": lambda: _scene(_spray()),
    "long_runs": lambda: _scene(_block(22), coef=2.1, cells=16.0),
    "small_cells": lambda: _scene(_block(11), cells=2.2),
}


def _pairs(sc, radius):
    """[n, n] distances (FP64, of the FP32 positions) and who can be whose neighbour: the 27
    cells around a particle's own."""
    x = sc.pos.astype(np.float32).astype(np.float64)
    b = sc.box
    lo = np.array([b.m_BufferedZone.m_MinBound.x, b.m_BufferedZone.m_MinBound.y, b.m_BufferedZone.m_MinBound.z])
    cell = np.trunc((sc.pos - lo) / b.m_CellSize).astype(int)
    for i in range(sc.n):
        r = np.sqrt(((x - x[i]) ** 2).sum(1))
        near = (np.abs(cell - cell[i]).max(1) <= 1) & (np.arange(sc.n) != i)
        yield i, r, near & (r < radius)


@pytest.mark.parametrize("name", list(SCENES))
def test_rows(name):
    """Neighbour sets, sums of weights and PND against numpy, and the walk without lists
    (rows_sell = 1) against the lists bit for bit."""
    sc = SCENES[name]()
    l0 = sc.param.InitialParticleDistance
    re, reg = l0 * sc.param.LaplacianInfluenceRadiusCoefficient, l0 * sc.param.GradientInfluenceRadiusCoefficient
    got = []
    for variant in (0, 1):
        s = Solver(sc, precision="fp32_ir", rows_sell=variant, compressibility=0.0)
        st = s.pressure()
        assert st["error_flags"] == 0
        q = s.debug_ppe()
        o = np.argsort(q["id"], kind="stable")
        got.append({k: v[o] for k, v in q.items()} | {"press": s.state()["press"], "its": st["cg_iterations"]})
        s.close()
    a, b = got
    for k in ("pnd", "diag", "rhs", "nbr_count", "nbr_idsum", "press", "its"):
        assert np.array_equal(a[k], b[k]), k
    p = sc.param
    coef = 2.0 * p.Dimension / (sc.lam * sc.n0_lap)
    for i, r, acc in _pairs(sc, re):
        # a pair within round-off of the radius may fall on either side
        sure = acc & (r < re * (1 - 1e-5))
        if sure.sum() == acc.sum():
            assert a["nbr_count"][i] == acc.sum()
            assert a["nbr_idsum"][i] == np.flatnonzero(acc).sum()
        rr = np.maximum(r[acc], 1e-3 * re)
        w = re / rr - 1.0
        rg = r[acc & (r < reg)]
        wg = reg / np.maximum(rg, 1e-3 * reg) - 1.0
        # a weight: 5 roundings' worth of re / r; a sum: at most 32 additions in FP32 each; a
        # pair on either side of the radius weighs less than 1e-5
        tol = 5 * U * (re / rr).sum() + 32 * U * w.sum() + 1e-5
        if a["diag"][i] != 1.0:
            assert abs(a["diag"][i] / coef - w.sum()) <= tol
        assert abs(a["pnd"][i] - wg.sum()) <= 5 * U * (reg / np.maximum(rg, 1e-3 * reg)).sum() + 32 * U * wg.sum() + 1e-5


@pytest.mark.parametrize("sides", [(10, 17)], ids=["row_grows"])
def test_rows_longer_than_the_list(sides):
    """The list has room for an eighth more entries than the longest row of the last step; the
    same solver on particles twice as dense, against a fresh one."""
    sc = _scene(_block(12, jitter=0.05))
    s = Solver(sc, precision="fp32_ir")
    first = s.pressure()["max_row"]
    dense = _scene(_block(12, jitter=0.05) * 0.9)
    dense.box = sc.box
    f = Solver(dense, precision="fp32_ir")
    pos, vel, press, visc = (np.ascontiguousarray(v, np.float64) for v in (dense.pos, dense.vel, dense.press, dense.visc))
    from simulation_project_gb300.solver import _check, _lib, _p
    _check(_lib().mps_solver_set_particles(s.h, dense.n, _p(pos), _p(vel), _p(press), _p(visc),
                                           _p(np.ascontiguousarray(dense.ptype, np.int32))), "set")
    a, b = s.pressure(), f.pressure()
    assert first > 0 and a["max_row"] == b["max_row"] > first + first // 8 + 15
    assert a["error_flags"] == 0 and b["error_flags"] == 0
    x, y = s.debug_ppe(), f.debug_ppe()
    for k in ("pnd", "diag", "nbr_count", "nbr_idsum", "sol"):
        assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("pos", [_block(3), _block(11), _spray(), _block(29), _block(30)],
                         ids=["27", "ragged", "spray", "24389", "27000"])
def test_predictor(pos):
    """One step without pressure (no particle passes the free-surface threshold): the FP32
    passes against the FP64 ones."""
    visc = 1e-2
    sc = _scene(pos, threshold=1e3, visc=visc)
    out = []
    for precision in ("fp32_ir", "fp64"):
        s = Solver(sc, precision=precision, pressure_mode=1)
        assert s.step(0)["error_flags"] == 0
        out.append(s.state())
        s.close()
    a, b = out
    assert np.array_equal(a["id"], b["id"])
    dv = np.abs(a["vel"] - b["vel"]).max(1)
    assert np.abs(b["vel"] - sc.vel).max() > 1e-4   # the viscous term is there to be seen
    l0, dt = sc.param.InitialParticleDistance, sc.param.Dt
    re = l0 * sc.param.LaplacianInfluenceRadiusCoefficient
    coef = 2.0 * sc.param.Dimension / (sc.lam * sc.n0_lap) * visc * dt
    rng = np.random.default_rng(5)
    for i in rng.choice(sc.n, min(sc.n, 300), replace=False):
        d = sc.pos - sc.pos[i]
        r = np.sqrt((d ** 2).sum(1))
        acc = (r < re * 1.00001) & (np.arange(sc.n) != i)
        rr = np.maximum(r[acc], 1e-3 * re)
        du = np.abs(sc.vel[acc] - sc.vel[i]).max(1)
        # FP32 positions (2 roundings of the coordinates) and 5 of the weight, FP32 velocities
        # and the sums' at most 32 additions
        dr = 2 * np.sqrt(3.0) * U * np.abs(sc.pos).max()
        w = np.maximum(re / rr - 1.0, 0.0)
        err = (du * (re / rr) * (dr / rr + 5 * U)).sum() + (32 * U * du * w).sum() + 2 * U * np.abs(sc.vel).max() * w.sum()
        assert dv[i] <= coef * err + 1e-7 * coef
