"""The launchers' library-owned scratch: calls of different kinds do not wait for each other's
host waits."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

import gpu_ref
import orc
from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import DeviceArray, call

pytestmark = pytest.mark.gpu


def test_a_sort_beside_triangle_cells_that_wait():
    """RegisterTriangleTopology waits on the host for what its stream holds before it; another
    thread sorts meanwhile."""
    st = orc.RefState(scenes.rotating_bucket(l0=0.006, n_drag=16))
    g = gpu_ref.GpuRef(st)
    keys = np.random.default_rng(3).integers(0, 9000, 20_000).astype(np.int32)

    sets = [(DeviceArray.from_host(keys), DeviceArray.from_host(np.arange(len(keys), dtype=np.int32))) for _ in range(2)]

    def sort(k):
        call("SortUsingThrust", len(keys), sets[k][0].ptr, sets[k][1].ptr)
    sort(0)   # kernels loaded, scratch held
    g.walls()
    want = g.download()["cells"]
    call("ResetTriangleTopology", g.stream.ref(), st.cells_n, g.p("cells"))
    g.stream.sync()

    cu = C.CDLL("libcuda.so.1")
    release, held = threading.Event(), threading.Event()

    @C.CFUNCTYPE(None, C.c_void_p)
    def hold(_):   # the stream stands here until it is released, 10 s at most
        held.set()
        release.wait(10)
    assert cu.cuLaunchHostFunc(g.stream.handle, hold, None) == 0
    bins = threading.Thread(target=lambda: call("RegisterTriangleTopology", g.stream.ref(), g.p("triangles"), st.t,
                                                g.p("cells"), st.cells_n))
    other = threading.Thread(target=sort, args=(1,))
    try:
        assert held.wait(5)
        bins.start()
        time.sleep(0.3)   # it has queued its kernels and waits
        assert bins.is_alive()
        other.start()
        other.join(5)
        assert not other.is_alive() and bins.is_alive()
    finally:
        release.set()
        bins.join()
        other.join()
    call("mps_device_sync")
    order = np.argsort(keys, kind="stable")
    for dk, dv in sets:
        assert np.array_equal(dk.download(), keys[order]) and np.array_equal(dv.download(), order)
    got = g.download()["cells"]
    assert np.array_equal(got["m_TriangleNum"], want["m_TriangleNum"])
    for c in np.flatnonzero(want["m_TriangleNum"]):
        k = want["m_TriangleNum"][c]
        assert np.array_equal(got["m_TriangleID"][c][:k], want["m_TriangleID"][c][:k])
