"""The key-order check where a warp's range of leaves starts and ends, and the shadow levels on columns
at odd addresses: two leaves swapped in a mesh in key order are put back by a regrid, and a balance on
columns off by one leaf marks what it marks on aligned ones."""
import ctypes
import functools

import numpy as np
import pytest

from tests import _oracle as O
from tests.test_gpu_amr import cfg, mesh, run_adapt

pytestmark = pytest.mark.gpu


@functools.lru_cache
def in_key_order(level):
    cols = O.uniform_mesh(level)
    p = np.argsort(O.cell_keys(cols["x"], cols["y"], cols["z"], cols["level"], None, 21, 21), kind="stable")
    return {k: np.ascontiguousarray(v[p]) for k, v in cols.items()}


@pytest.mark.parametrize("level,at", [(1, 0), (2, 30), (2, 31), (2, 62), (7, None), (7, 31), (7, 2 ** 21 - 2)] +
                         [(7, 32 * k - 1) for k in (2, 5, 6, 7, 8, 14, 4096, 65535)])
def test_swapped_leaves(ctx, level, at):
    want = in_key_order(level)
    cols = {k: v.copy() for k, v in want.items()}
    if at is not None:
        for v in cols.values():
            v[[at, at + 1]] = v[[at + 1, at]]
    rc, got, st, _ = run_adapt(ctx, cols, cfg(max_level=8, min_level=0, balance_mode=1))
    assert rc == 0
    for k in ("x", "y", "z", "level"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


@pytest.mark.parametrize("off", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("drop", [0, 1, 2, 3])
def test_shadow_columns(ctx, off, drop):
    cols = O.random_octree(7, ext=(1, 1, 1), rounds=4, max_level=5, frac=0.3)
    rng = np.random.default_rng(off)
    cols["flags"] = (rng.integers(0, 8, len(cols["x"])) == 0).astype(np.int32)
    cols["state"] = (rng.integers(0, 5, len(cols["x"])) == 0).astype(np.uint8)
    n = len(cols["x"]) - off - drop
    c = cfg(max_level=5, balance_mode=1)

    def marks(m, view):
        rc = ctx.lib.fl_balance_enforce(ctx.handle, ctypes.byref(view), ctypes.byref(c), None)
        assert rc in (0, -5)
        return m.download()["flags"]

    whole = mesh(ctx, cols)
    view = type(whole.m).from_buffer_copy(whole.m)
    for k, w in (("x", 4), ("y", 4), ("z", 4), ("level", 1), ("state", 1), ("flags", 4), ("material", 4)):
        setattr(view, k, getattr(whole.m, k) + off * w)
    view.num_cells = n
    got = marks(whole, view)[off:off + n]
    part = mesh(ctx, {k: np.ascontiguousarray(v[off:off + n]) for k, v in cols.items()})
    np.testing.assert_array_equal(got, marks(part, part.m))
    want, _ = O.balance({k: v[off:off + n] for k, v in cols.items()}, O.domain(max_level=5), 1, 5, 4096)
    np.testing.assert_array_equal(got, want)
