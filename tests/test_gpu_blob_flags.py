"""Blob flags: the cheap sum with its exact re-check against the exact kernel (which a blob of negative
amplitude selects) and the oracle, with thresholds that fall exactly on cells' values, wide and
narrow blobs, none at all, blobs outside the cube, ragged cell counts."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300.amr import Mesh
from tests import _oracle as O

pytestmark = pytest.mark.gpu


def flags(ctx, cols, blobs, lo, hi, ml):
    m = Mesh(ctx, cols)
    b = np.ascontiguousarray(blobs, np.float32).reshape(-1, 5)
    ctx.call("fl_flags_from_blobs", ctypes.byref(m.m), b.ctypes.data_as(ctypes.c_void_p), len(b), ctypes.c_float(lo),
             ctypes.c_float(hi), ml)
    return m.download()["flags"]


def cells(n, seed):
    rng = np.random.default_rng(seed)
    lv = rng.integers(2, 9, n)
    xyz = [(rng.random(n) * (1 << lv)).astype(np.int32) for _ in range(3)]
    return {"x": xyz[0], "y": xyz[1], "z": xyz[2], "level": lv.astype(np.uint8), "state": np.zeros(n, np.uint8),
            "flags": np.full(n, 7, np.int32), "material": np.zeros(n, np.uint32)}


FAR = np.float32([[900.0, 900.0, 900.0, 1.0, -1e-30]])  # adds nothing; its sign keeps the exact kernel


@pytest.mark.parametrize("n", [1, 255, 1025, 200003])
@pytest.mark.parametrize("k", [0, 1, 7, 64, 1024])
def test_near_sum_equals_exact(ctx, n, k):
    rng = np.random.default_rng(1000 * k + n)
    cols = cells(n, n)
    w = 10.0 ** rng.uniform(-2.5, 0.5, k)
    blobs = np.concatenate([rng.uniform(-0.3, 1.3, (k, 3)), (1 / (2 * w * w))[:, None], rng.uniform(0, 2, (k, 1))],
                           1).astype(np.float32)
    # values of some cells, in FP32 steps of a plain sum: thresholds on, just above and below them
    s = (0.5 ** cols["level"].astype(np.float32))
    p = np.stack([(cols[a] + np.float32(0.5)) * s for a in "xyz"], 1)
    pick = rng.integers(0, n, 2)
    v = [sum(float(b[4]) * np.exp(-float(((p[i] - b[:3]) ** 2).sum()) * float(b[3])) for b in blobs) for i in pick]
    lo, hi = np.float32(min(v)), np.float32(max(v))
    for a, b in ((lo, hi), (np.nextafter(lo, np.float32(9)), np.nextafter(hi, np.float32(-9))), (0.4, 0.7)):
        got = flags(ctx, cols, blobs, a, b, 7)
        np.testing.assert_array_equal(got, flags(ctx, cols, np.concatenate([blobs, FAR]), a, b, 7) if k < 1024 else
                                      O.blob_flags(cols, blobs, float(a), float(b), 7))
    np.testing.assert_array_equal(got, O.blob_flags(cols, blobs, 0.4, 0.7, 7))
