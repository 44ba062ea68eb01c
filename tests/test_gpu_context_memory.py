"""What contexts keep of freed device memory: all of a device's together no more than one does."""
import ctypes

import pytest

from fluidloom_gb300 import Context
from fluidloom_gb300.amr import FlMesh

pytestmark = pytest.mark.gpu


def test_contexts_keep_one_bound_together():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    first = Context(0)
    before, total = torch.cuda.mem_get_info()
    bound, slack = total // 64, 256 << 20
    cells = bound // 2 // 22  # 22 bytes a cell: each context alone stays below the bound
    ctxs = [first] + [Context(0) for _ in range(3)]
    meshes = [FlMesh() for _ in ctxs]
    for c, m in zip(ctxs, meshes):
        c.call("fl_mesh_alloc", ctypes.c_size_t(cells), 0, ctypes.byref(m))
    assert before - torch.cuda.mem_get_info()[0] > bound  # they are there
    for c, m in zip(ctxs, meshes):
        c.call("fl_mesh_free", ctypes.byref(m))
    for c in ctxs:
        c.sync()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= bound + slack, (kept, bound)
    # the others' memory serves one that outlives them
    for c in ctxs[1:]:
        c.close()
    m = FlMesh()
    first.call("fl_mesh_alloc", ctypes.c_size_t(cells), 0, ctypes.byref(m))
    first.call("fl_mesh_free", ctypes.byref(m))
    first.sync()
    first.close()
