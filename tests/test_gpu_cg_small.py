"""The inner CG of a pass in one launch (k_cg_small) against the chain of kernels (which a
profiling solver runs): fewer rows than a slice, slices over several coarse aggregates and
aggregates over several CTAs, one to five slices per CTA, the size at which the chain takes
over, flexible CG, and an iteration limit that ends it early."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def _block(shape, seed=0, l0=0.004, jitter=0.02):
    p = scenes.default_param(l0, 1e-4)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3) * l0
    g = g + np.random.default_rng(seed).uniform(-jitter * l0, jitter * l0, g.shape)
    return scenes._finish("block", p, g, np.zeros((0, 3, 3)), np.zeros(0, np.int32), [scenes._tri_normal_params(dt=p.Dt)], [],
                          seed, l0)


def _both(sc, njp, **kw):
    out = []
    for profile in (0, 1):
        s = Solver(sc, precision="fp32_ir", profile=profile, **kw)
        st = s.pressure(njp=njp)
        out.append((st, s.state()["press"], s.debug_residual(0)[1]))
        s.close()
    return out


@pytest.mark.parametrize("njp,flexible", [(False, 0), (True, 0), (True, 1)], ids=["jacobi", "multilevel", "flexible"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (7, 7, 7), (9, 40, 5), (13, 12, 11), (17, 17, 16), (24, 24, 23), (27, 27, 26),
                                   (27, 27, 27), (31, 31, 31)],
                         ids=["125", "343", "slab", "1716", "4624", "13248", "18954", "19683", "29791_chain"])
def test_against_the_kernel_chain(shape, njp, flexible):
    (a, pa, ra), (b, pb, rb) = _both(_block(shape), njp, flexible=flexible)
    assert a["error_flags"] == 0 and b["error_flags"] == 0 and a["inner16"] == 1
    assert a["interior"] == b["interior"] > 0 and a["mg_levels"] == b["mg_levels"]
    assert a["cg_relres"] <= 1e-8 and ra <= 1e-8 * (1 + 1e-3) and rb <= 1e-8 * (1 + 1e-3)
    # both solve the same system by the same recurrences; the sums' order may move a stop by one
    assert a["ir_passes"] == b["ir_passes"] and abs(a["cg_iterations"] - b["cg_iterations"]) <= a["ir_passes"]
    assert np.abs(pa - pb).max() <= 1e-5 * np.abs(pb).max()


@pytest.mark.parametrize("limit", [1, 2, 5])
def test_iteration_limit(limit):
    (a, pa, _), (b, pb, _) = _both(_block((13, 12, 11)), True, cg_max_iter=limit, ir_max_outer=2)
    assert a["error_flags"] == b["error_flags"] and a["cg_iterations"] == b["cg_iterations"] == 2 * limit
    assert np.abs(pa - pb).max() <= 1e-5 * np.abs(pb).max()


def test_solvers_in_threads():
    """Cooperative launches of several solvers at once: each finds its CTAs together or waits."""
    import threading
    shapes = [(24, 24, 23), (17, 17, 16), (24, 23, 22), (13, 12, 11)]
    out = [[None] * len(shapes) for _ in range(2)]

    def work(k, into):
        s = Solver(_block(shapes[k], seed=k), precision="fp32_ir")
        st = [s.step(i) for i in range(15)]
        into[k] = ([(q["error_flags"], q["cg_iterations"]) for q in st], s.state()["press"])
        s.close()
    for k in range(len(shapes)):
        work(k, out[0])
    threads = [threading.Thread(target=work, args=(k, out[1])) for k in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(*out):
        assert all(f == 0 for f, _ in a[0]) and a[0] == b[0]
        assert np.array_equal(a[1], b[1])
