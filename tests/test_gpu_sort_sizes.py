"""The radix sort at the edges of its tiles: both tile depths, whole and ragged
last tiles, the sizes where the depth changes, every shape, keys with many ties,
against numpy's stable sort."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray

pytestmark = pytest.mark.gpu

SMALL = 1 << 20  # the most keys a small-tile sort takes


@pytest.mark.parametrize("shape", [(8, 256), (8, 512), (9, 256), (9, 512)])
@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 2049, 151 * 1024 + 7, SMALL - 1, SMALL, SMALL + 1])
def test_sort_at_tile_edges(ctx, n, shape):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    keys[rng.random(n) < 0.5] &= np.uint64(0xFF000)  # ties and near-constant digits
    ids = np.arange(n, dtype=np.uint32)
    ctx.call("fl_sort_set_config", *shape)
    try:
        dk, di = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, ids)
        ctx.call("fl_sort_pairs_u64_u32", dk.ptr, di.ptr, ctypes.c_size_t(n), 0, 63)
        order = np.argsort(keys, kind="stable")
        np.testing.assert_array_equal(di.to_host(), order.astype(np.uint32))
        np.testing.assert_array_equal(dk.to_host(), keys[order])
    finally:
        ctx.call("fl_sort_set_config", 8, 256)
