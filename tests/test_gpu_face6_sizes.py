"""FACE6 balance around the leaf count where a leaf's faces go from lanes to one thread, and with columns at
every alignment, against the oracle: meshes with jumps of two levels and more, gaps, solid leaves."""
import ctypes
import functools

import numpy as np
import pytest

from tests import _oracle as O
from tests.test_gpu_amr import cfg, mesh

pytestmark = pytest.mark.gpu

LINE = 1 << 17  # the most leaves whose faces are spread over lanes


@functools.lru_cache(maxsize=1)
def jumps():
    """48^3 leaves of level 6, some split once, some of those again, shuffled blocks in key order."""
    rng = np.random.default_rng(3)
    e = 48
    i = np.arange(e ** 3)
    p, lv = np.stack([i % e, i // e % e, i // e ** 2]), np.full(e ** 3, 6)
    c = np.arange(8)
    kids = np.stack([c & 1, c >> 1 & 1, c >> 2])
    for l in (6, 7):
        split = (lv == l) & (rng.random(len(lv)) < (0.03 if l == 6 else 0.1))
        fine = (2 * p[:, split][:, :, None] + kids[:, None, :]).reshape(3, -1)
        p, lv = np.concatenate([p[:, ~split], fine], axis=1), np.append(lv[~split], np.full(fine.shape[1], l + 1))
    key = O.cell_keys(*p.astype(np.int32), lv.astype(np.uint8), None, 21, 21)
    order = np.argsort(key, kind="stable")
    n = len(order)
    return {"x": p[0][order].astype(np.int32), "y": p[1][order].astype(np.int32), "z": p[2][order].astype(np.int32),
            "level": lv[order].astype(np.uint8), "state": (rng.random(n) < 0.05).astype(np.uint8),
            "flags": np.zeros(n, np.int32), "material": np.zeros(n, np.uint32)}


@pytest.mark.parametrize("n,off", [(1, 0), (5, 1), (4099, 2), (LINE - 1, 0), (LINE, 0), (LINE, 3), (LINE + 1, 0), (LINE + 1, 1),
                                   (LINE + 30, 2), (LINE + 1027, 0)])
def test_balance(ctx, n, off):
    cols = jumps()
    assert len(cols["x"]) >= n + off
    part = {k: np.ascontiguousarray(v[:n + off]) for k, v in cols.items()}
    whole = mesh(ctx, part)
    view = type(whole.m).from_buffer_copy(whole.m)
    for k, w in (("x", 4), ("y", 4), ("z", 4), ("level", 1), ("state", 1), ("flags", 4), ("material", 4)):
        setattr(view, k, getattr(whole.m, k) + off * w)
    view.num_cells = n
    c = cfg(max_level=9, balance_mode=0, iters=6)
    rc = ctx.lib.fl_balance_enforce(ctx.handle, ctypes.byref(view), ctypes.byref(c), None)
    assert rc in (0, -5)
    want, _ = O.balance({k: v[off:] for k, v in part.items()}, O.domain(max_level=9), 0, 9, 6)
    np.testing.assert_array_equal(whole.download()["flags"][off:], want)
