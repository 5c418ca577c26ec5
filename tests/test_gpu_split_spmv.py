"""The inner SpMV whose warps share a slice (k_spmv_ring_split) and the grid reductions of
the CG kernels at sizes where they can go wrong: fewer rows than a slice, ragged last
slices, more slices than resident CTAs take at once, slices with 32-bit columns, and the
size at which whole slices take over.  The refinement only ends at 1e-8 of the FP32-weight
operator's residual, recomputed here in FP64; a wrong product of the FP16 operator (which is
within 2^-11 of it) stalls it or multiplies its passes."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def _block(shape, seed=0, l0=0.004):
    p = scenes.default_param(l0, 1e-4)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3) * l0
    g = g + np.random.default_rng(seed).uniform(-0.02 * l0, 0.02 * l0, g.shape)
    return scenes._finish("block", p, g, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)], [],
                          seed, l0)


@pytest.mark.parametrize("njp", [False, True], ids=["jacobi", "multilevel"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (7, 7, 7), (11, 9, 10), (32, 31, 33), (50, 51, 49), (9, 150, 150)],
                         ids=["27_rows", "125_rows", "ragged", "33k", "125k", "wide_columns"])
def test_pressure_solve(shape, njp):
    sc = _block(shape)
    s = Solver(sc, precision="fp32_ir")
    r = s.pressure(njp=njp)
    assert r["error_flags"] == 0 and r["inner16"] == 1
    assert r["cg_relres"] <= 1e-8 and r["interior"] > 0
    if shape[1] == 150:
        assert r["nnz_wide"] > 0
    _, rel = s.debug_residual(0)
    assert rel <= 1e-8 * (1 + 1e-3)
    passes = Solver(sc, precision="fp32_ir", inner_weights=32).pressure(njp=njp)["ir_passes"]
    assert r["ir_passes"] <= passes + 2
    s.close()


def test_whole_slices_take_over():
    """411,774 particles: k_spmv_stream; one layer less, k_spmv_ring_split."""
    its = []
    for nx in (74, 71):
        s = Solver(_block((nx, 74, 75)), precision="fp32_ir")
        r = s.pressure()
        assert r["error_flags"] == 0 and r["cg_relres"] <= 1e-8
        its.append(r["cg_iterations"])
        s.close()
    assert abs(its[0] - its[1]) <= 3


def test_compaction_at_the_zone_bounds():
    """k_zone_flags compares doubles as ordered integers: the bounds themselves, both zeros
    against a zero bound, the nearest doubles outside, subnormals and infinities, and which
    particles stay when some leave and when none do."""
    p = scenes.default_param(0.01, 1e-4)
    hi = float(np.float32(0.3))
    box = scenes.grid_box(np.zeros(3), np.full(3, 0.3), p)
    mid = np.random.default_rng(0).uniform(0.1, 0.2, (300, 3))
    edge = [0.0, -0.0, hi, np.nextafter(hi, 1), np.nextafter(0.0, -1), 5e-324, -1e-300, np.inf, -np.inf, np.nextafter(hi, 0)]
    stays = [v for v in edge if not (v < 0.0 or v > hi)]
    for values in (edge, stays):
        pos = mid.copy()
        for k, v in enumerate(values):
            pos[7 * k, k % 3] = v
        want = np.flatnonzero(~((pos < 0.0) | (pos > hi)).any(1))
        sc = scenes._finish("zone", p, mid, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)],
                            [], 0, 0.01, np.zeros(3), np.full(3, 0.3))
        assert sc.box.m_ComputeZone.m_MaxBound.x == np.float32(hi) and sc.box.cell_num == box.cell_num
        sc.pos = pos
        s = Solver(sc, precision="fp32_ir")
        assert s.pressure()["particles"] == len(want)
        assert np.array_equal(np.sort(s.state()["id"]), want)
        s.close()


@pytest.mark.parametrize("n_side", [3, 27, 28, 58, 59])
def test_correction_shares(n_side):
    """k_correct_warp with 4, 16 and 32 particles per warp gives every particle its own
    update: the velocities of a step against the FP64 solver's, to the FP32 operators'
    accuracy over one step."""
    out = []
    for precision in ("fp32_ir", "fp64"):
        s = Solver(_block((n_side,) * 3), precision=precision)
        assert s.step(0)["error_flags"] == 0
        out.append(s.state()["vel"])
        s.close()
    scale = np.abs(out[1]).max()
    assert np.abs(out[0] - out[1]).max() <= 2e-3 * scale
