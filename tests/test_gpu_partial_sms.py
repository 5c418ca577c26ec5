"""Calls on a part of the GPU's SMs (a green context of 16), where cooperative launches of one
or two CTAs per SM of the whole GPU are refused: the sorts take fewer CTAs, the solver its
kernel chain, with the results of the whole GPU."""
import ctypes as C
import threading

import numpy as np
import pytest

import gpu_ref
import orc
from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import DeviceArray, call
from simulation_project_gb300.solver import Solver

pytestmark = pytest.mark.gpu


class Green:
    """16 SMs: a stream of its own (`stream`, for ref()) and a context (`current`)."""

    def __init__(self):
        try:
            cu = C.CDLL("libcuda.so.1")
            fs = [getattr(cu, f) for f in ("cuDeviceGetDevResource", "cuDevSmResourceSplitByCount",
                                           "cuDevResourceGenerateDesc", "cuGreenCtxCreate", "cuGreenCtxStreamCreate",
                                           "cuCtxFromGreenCtx")]
        except (OSError, AttributeError) as e:
            pytest.skip(f"no green contexts: {e}")
        self.cu = cu
        whole, part, rest = (C.create_string_buffer(1024) for _ in range(3))
        groups, desc, ctx, self.stream, self.ctx = C.c_uint(1), C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p()
        for f, args in zip(fs, ((0, whole, 1), (part, C.byref(groups), whole, rest, 0, 16), (C.byref(desc), part, 1),
                                (C.byref(ctx), desc, 0, 1), (C.byref(self.stream), ctx, 1, 0), (C.byref(self.ctx), ctx))):
            rc = f(*args)
            if rc:
                pytest.skip(f"no green contexts: {f.__name__} returned {rc}")
        self.green = ctx

    def ref(self):
        return C.byref(self.stream)

    def current(self):
        assert self.cu.cuCtxSetCurrent(self.ctx) == 0

    def close(self):
        call("mps_device_sync")
        assert self.cu.cuStreamDestroy_v2(self.stream) == 0 and self.cu.cuGreenCtxDestroy(self.green) == 0


@pytest.fixture
def green():
    call("mps_set_device", 0)
    call("mps_device_sync")
    g = Green()
    yield g
    g.close()


def test_triangle_cells(green):
    st = orc.RefState(scenes.rotating_bucket(l0=0.002, n_drag=300))
    g = gpu_ref.GpuRef(st)
    g.walls()
    want = g.download()["cells"]
    assert want["m_TriangleNum"].sum() > 40000   # the sort asks for more CTAs than fit
    call("ResetTriangleTopology", green.ref(), st.cells_n, g.p("cells"))
    call("RegisterTriangleTopology", green.ref(), g.p("triangles"), st.t, g.p("cells"), st.cells_n)
    call("mps_device_sync")
    got = g.download()["cells"]
    assert np.array_equal(got["m_TriangleNum"], want["m_TriangleNum"])
    for c in np.flatnonzero(want["m_TriangleNum"]):
        k = want["m_TriangleNum"][c]
        assert np.array_equal(got["m_TriangleID"][c][:k], want["m_TriangleID"][c][:k])
    g.walls()   # and on an ordinary stream again


def _in_context(green, work):
    """work() in a thread whose current context is the green one."""
    out = []

    def run():
        green.current()
        try:
            out.append(work())
        except Exception as e:   # noqa: BLE001 (raised again by the test)
            out.append(e)
    t = threading.Thread(target=run)
    t.start()
    t.join()
    if isinstance(out[0], Exception):
        raise out[0]
    return out[0]


@pytest.mark.parametrize("n", [4096, 70_001, 3_000_001])
def test_sort(green, n):
    keys = np.random.default_rng(n).integers(-10 ** 6, 10 ** 6, n).astype(np.int32)

    def work():
        dk, dv = DeviceArray.from_host(keys), DeviceArray.from_host(np.arange(n, dtype=np.int32))
        call("SortUsingThrust", n, dk.ptr, dv.ptr)
        return dk.download(), dv.download()
    order = np.argsort(keys, kind="stable")
    k, v = _in_context(green, work)
    assert np.array_equal(k, keys[order]) and np.array_equal(v, order)


@pytest.mark.parametrize("l0", [0.02, 0.01], ids=["2k", "16k"])
def test_solver(green, l0):
    """The multilevel solve: one coarse level and, of the larger scene, two."""
    sc = scenes.dam_break(l0=l0)

    def work():
        s = Solver(sc, precision="fp32_ir")
        st = [s.step(i) for i in range(3)]
        out = [q["error_flags"] for q in st], [q["cg_relres"] for q in st], s.state()
        s.close()
        return out
    a, b = work(), _in_context(green, work)
    for flags, res, _ in (a, b):
        assert flags == [0, 0, 0] and max(res) <= 1e-8
    assert np.abs(a[2]["press"] - b[2]["press"]).max() <= 1e-4 * np.abs(a[2]["press"]).max()
    assert np.array_equal(a[2]["id"], b[2]["id"])
