"""Trilinear ghosts at the edges of a warp's round: every way the columns share 32 lanes, ragged
query counts, corners outside the mesh, level-0 and negative queries, against the same FP32 sums in
numpy."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray
from fluidloom_gb300.amr import AdaptConfig, Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 3, 4, 5, 33, 1001])
@pytest.mark.parametrize("C", [1, 2, 5, 8, 10, 11, 16, 17, 31, 32])
def test_interp_column_widths(ctx, C, nq):
    rng = np.random.default_rng(100 * C + nq)
    e, lv = 6, 3
    i = rng.permutation(e ** 3).astype(np.int32)
    cols = {"x": i % e, "y": (i // e) % e, "z": i // (e * e), "level": np.full(e ** 3, lv, np.uint8)}
    m = Mesh(ctx, cols)
    f = rng.standard_normal((e ** 3, C)).astype(np.float32)
    q = rng.integers(-3, 2 * e + 3, (3, nq)).astype(np.int32)
    ql = rng.choice(np.array([0, lv, lv + 1, lv + 1, lv + 1], np.uint8), nq)
    df, dl, out = DeviceArray.from_host(ctx, f), DeviceArray.from_host(ctx, ql), DeviceArray(ctx, (nq, C), np.float32)
    dq = [DeviceArray.from_host(ctx, a) for a in q]
    ctx.call("fl_interp_trilinear", ctypes.byref(m.m), ctypes.byref(AdaptConfig.make(max_level=7)), df.ptr, C,
             *[a.ptr for a in dq], dl.ptr, ctypes.c_size_t(nq), out.ptr)
    row = np.full((e, e, e), -1)
    row[cols["z"], cols["y"], cols["x"]] = np.arange(e ** 3)
    want = np.zeros((nq, C), np.float32)
    half = np.trunc(q / 2).astype(np.int64)
    for n in range(nq):
        if ql[n] != lv + 1:
            continue
        for k in range(8):
            p = half[:, n] + [k & 1, (k >> 1) & 1, k >> 2]
            if (p < 0).any():
                continue
            p %= 1 << lv  # the key codec keeps an anchor's low 21 bits
            if (p < e).all():
                want[n] += np.float32(0.125) * f[row[p[2], p[1], p[0]]]
    np.testing.assert_array_equal(out.to_host(), want)
