"""RegisterTriangleTopology on a grid of 140 million cells: the cells of the far corner, which
a 32-bit count of a warp per cell does not reach, get their triangles."""
import numpy as np
import pytest

from simulation_project_gb300 import scenes
from simulation_project_gb300.lib import DeviceArray, Stream, call
from simulation_project_gb300.refpath import triangle_records
from simulation_project_gb300.types import CELL_DTYPE, grid_box

pytestmark = pytest.mark.gpu


def test_far_cells():
    torch = pytest.importorskip("torch")
    p = scenes.default_param(0.01, 1e-4)
    size = 0.04   # of a cell
    box = grid_box(np.zeros(3), np.full(3, 516 * size - 0.02), p)
    cells = box.cell_num
    assert 2 ** 32 // 32 < cells < 2 ** 31 // 12
    if torch.cuda.mem_get_info()[0] < 80e9:
        pytest.skip("needs 57 GB for the cells")
    lo = np.array([box.m_BufferedZone.m_MinBound.x, box.m_BufferedZone.m_MinBound.y, box.m_BufferedZone.m_MinBound.z])
    g = np.array([box.m_GridSize.x, box.m_GridSize.y, box.m_GridSize.z])
    assert np.prod(g.astype(np.int64)) == cells
    at = np.array([[0, 0, 0], g - 3, [g[0] - 3, 2, 5], g - 3])   # cells of small triangles, each inside its cell
    tri = lo + (at[:, None, :] + 0.5 + 0.1 * np.eye(3)[None]) * size
    rec = triangle_records(tri, 0)
    d = {k: DeviceArray.from_host(v) for k, v in (("tri", rec), ("one", np.zeros(64, np.int32)))}
    c = DeviceArray(cells, CELL_DTYPE)
    one = d["one"].ptr
    call("InitializeDeviceMemConst", p, 0, d["tri"].ptr, len(tri), one, 0, one, one, c.ptr, cells, one, one, one, box)
    s = Stream()
    call("ResetTriangleTopology", s.ref(), cells, c.ptr)
    call("RegisterTriangleTopology", s.ref(), d["tri"].ptr, len(tri), c.ptr, cells)
    s.sync()
    want = {}
    for t, (i, j, k) in enumerate(at):
        want.setdefault(int((i * g[1] + j) * g[2] + k), []).append(t)
    got = np.zeros(1, CELL_DTYPE)
    for key, ids in want.items():
        call("mps_memcpy_dtoh", got.ctypes.data, c.ptr + key * CELL_DTYPE.itemsize, CELL_DTYPE.itemsize)
        assert got["m_TriangleNum"][0] == len(ids) and got["m_TriangleID"][0][:len(ids)].tolist() == ids, key
    for key in (1, 2 ** 27, cells - 1):
        call("mps_memcpy_dtoh", got.ctypes.data, c.ptr + key * CELL_DTYPE.itemsize, CELL_DTYPE.itemsize)
        assert got["m_TriangleNum"][0] == 0, key
    c.free()
