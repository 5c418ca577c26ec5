"""Which kernel the inner CG of a small system runs on, and that kernel at the sizes it then
has: k_cg_small with one to six slices per CTA and at the size at which the chain takes over,
each against the chain (a profiling solver), and the chain's k_spmv_ring_split on fewer rows
than a slice and on ragged last slices, which a default solver no longer gives it; and the
size at which a warp of the correction takes 32 particles."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver, _lib

pytestmark = pytest.mark.gpu


def _block(shape, coef=4.0, seed=0, l0=0.004):
    p = scenes.default_param(l0, 1e-4)
    p.LaplacianInfluenceRadiusCoefficient = coef
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3) * l0
    g = g + np.random.default_rng(seed).uniform(-0.02 * l0, 0.02 * l0, g.shape)
    return scenes._finish("block", p, g, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)], [],
                          seed, l0)


@pytest.mark.parametrize("shape,coef,njp,slices", [
    ((5, 5, 5), 4.0, False, 1), ((16, 17, 17), 4.0, True, 1), ((20, 21, 19), 4.0, False, 2), ((20, 21, 19), 4.0, True, 2),
    ((24, 24, 24), 4.0, True, 3), ((26, 26, 26), 4.0, True, 4), ((27, 27, 27), 4.0, False, 5), ((27, 27, 27), 4.0, True, 0),
    ((29, 29, 28), 4.0, False, 5), ((31, 31, 30), 3.7, False, 6), ((31, 31, 30), 4.0, False, 0)],
    ids=["one", "one_multilevel", "two", "two_multilevel", "three_multilevel", "four_multilevel", "five",
         "five_multilevel_chain", "five_full", "six", "six_long_rows_chain"])
def test_slices_per_cta(shape, coef, njp, slices):
    sc = _block(shape, coef)
    out = []
    for profile in (0, 1):
        s = Solver(sc, precision="fp32_ir", profile=profile)
        st = s.pressure(njp=njp)
        want = _lib().mps_debug_cg_small_slices(sc.n, st["max_row"], 152, st["mg_levels"], st["mg_level1"])
        assert s.debug_cg_small() == (0 if profile else slices) and want == slices
        assert st["error_flags"] == 0 and st["cg_relres"] <= 1e-8
        assert s.debug_residual(0)[1] <= 1e-8 * (1 + 1e-3)
        out.append((st["cg_iterations"], st["ir_passes"], s.state()["press"]))
        s.close()
    (ia, pa, a), (ib, pb, b) = out
    assert pa == pb and abs(ia - ib) <= pa
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


@pytest.mark.parametrize("njp", [False, True], ids=["jacobi", "multilevel"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (7, 7, 7), (11, 9, 10), (3, 3, 57)], ids=["27_rows", "125_rows", "ragged", "rod"])
def test_small_systems_on_the_chain(shape, njp):
    sc = _block(shape)
    passes = []
    for bits in (16, 32):
        s = Solver(sc, precision="fp32_ir", profile=1, inner_weights=bits)
        st = s.pressure(njp=njp)
        assert s.debug_cg_small() == 0 and st["inner16"] == (bits == 16)
        assert st["error_flags"] == 0 and st["cg_relres"] <= 1e-8
        assert s.debug_residual(0)[1] <= 1e-8 * (1 + 1e-3)
        passes.append(st["ir_passes"])
        s.close()
    assert passes[0] <= passes[1] + 2


@pytest.mark.parametrize("side", [43, 44])
def test_correction_shares(side):
    """16 and 32 particles per warp of the correction: the velocities of a step against the
    FP64 solver's, to the FP32 operators' accuracy over one step."""
    out = []
    for precision in ("fp32_ir", "fp64"):
        s = Solver(_block((side,) * 3), precision=precision)
        assert s.step(0)["error_flags"] == 0
        out.append(s.state()["vel"])
        s.close()
    assert np.abs(out[0] - out[1]).max() <= 2e-3 * np.abs(out[1]).max()
