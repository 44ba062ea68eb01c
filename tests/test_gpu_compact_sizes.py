"""Compaction and permutation at the edges: tile borders, everything dropped or kept, EMPTY keys
with a live state, and elements of every word width at aligned and unaligned addresses, against
numpy."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray

pytestmark = pytest.mark.gpu

EMPTY = np.uint64(0xFFFFFFFFFFFFFFFF)
INVALID = np.uint32(0xFFFFFFFF)


@pytest.mark.parametrize("keep", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("n", [1, 31, 511, 513, 4095, 4096, 4097, 3 * 4096 + 100, 70000])
def test_compact_at_tile_edges(ctx, n, keep):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    keys[rng.random(n) < 0.05] = EMPTY
    state = (rng.random(n) < keep).astype(np.uint32) * rng.integers(1, 9, n, dtype=np.uint32)
    dk, ds = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, state)
    perm, si = DeviceArray(ctx, (n,), np.uint32), DeviceArray(ctx, (n,), np.uint32)
    sk, m = DeviceArray(ctx, (n,), np.uint64), ctypes.c_size_t(7)
    ctx.call("fl_compact_and_permute", dk.ptr, ds.ptr, ctypes.c_size_t(n), perm.ptr, sk.ptr, si.ptr, ctypes.byref(m))
    live = np.nonzero((state != 0) & (keys != EMPTY))[0]
    order = live[np.argsort(keys[live], kind="stable")]
    want = np.full(n, INVALID, np.uint32)
    want[order] = np.arange(len(order), dtype=np.uint32)
    assert m.value == len(live)
    np.testing.assert_array_equal(perm.to_host(), want)
    np.testing.assert_array_equal(sk.to_host()[:len(live)], keys[order])
    np.testing.assert_array_equal(si.to_host()[:len(live)], order.astype(np.uint32))


@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("elem", [1, 2, 3, 4, 6, 7, 8, 12, 16, 20, 32, 76, 100])
def test_apply_permutation_word_widths(ctx, elem, offset):
    n = 1000
    rng = np.random.default_rng(elem)
    perm = rng.permutation(n).astype(np.uint32)
    perm[rng.random(n) < 0.2] = INVALID
    src = rng.integers(0, 256, n * elem + offset, dtype=np.uint8)
    ds, dp = DeviceArray.from_host(ctx, src), DeviceArray.from_host(ctx, perm)
    dd = DeviceArray(ctx, (n * elem + offset,), np.uint8).zero()
    at = ctypes.c_void_p(ds.ptr.value + offset), ctypes.c_void_p(dd.ptr.value + offset)
    ctx.call("fl_apply_permutation", *at, ctypes.c_size_t(elem), ctypes.c_size_t(n), dp.ptr)
    want = np.zeros((n, elem), np.uint8)
    ok = perm != INVALID
    want[perm[ok]] = src[offset:].reshape(n, elem)[ok]
    np.testing.assert_array_equal(dd.to_host()[offset:].reshape(n, elem), want)
