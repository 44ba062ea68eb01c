"""Large sorts that put low passes off: low digits set by the high ones, few digits that are not (every
pass runs after all), full ones, odd and even pass counts, bit ranges, every shape, against numpy's
stable sort."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray

pytestmark = pytest.mark.gpu

PLANNED = 2 << 20  # the fewest keys of a sort that may put passes off


@pytest.mark.parametrize("shape", [(8, 256), (8, 512), (9, 256), (9, 512)])
@pytest.mark.parametrize("what", ["set", "set, odd", "one late", "few", "ties", "full"])
@pytest.mark.parametrize("n,bits", [(PLANNED - 1, (0, 63)), (PLANNED, (0, 63)), (PLANNED + 3073, (0, 56)),
                                    (PLANNED + 3073, (5, 64))])
def test_sort_puts_passes_off(ctx, n, bits, what, shape):
    rng = np.random.default_rng(n)
    top = rng.integers(0, 1 << (31 if what != "ties" else 9), n, dtype=np.uint64)
    low = rng.integers(0, 1 << 33, 11, dtype=np.uint64)
    if what == "set, odd":  # one more full digit
        low = low & np.uint64(0xFFFFFF)
        keys = (top << np.uint64(33)) | (rng.integers(0, 1 << 9, n, dtype=np.uint64) << np.uint64(24)) | low[top % np.uint64(11)]
    elif what == "full":
        keys = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    elif what == "few":  # not set by the high digits
        keys = ((top & np.uint64(0xFFFFF)) << np.uint64(33)) | low[rng.integers(0, 11, n)]
    else:
        keys = (top << np.uint64(33)) | low[top % np.uint64(11)]
        if what == "one late":  # two neighbours in the sorted order that only a low digit parts
            keys[n // 3] = (top[7] << np.uint64(33)) | (low[top[7] % np.uint64(11)] ^ np.uint64(1))
            keys[7], keys[n // 3] = max(keys[7], keys[n // 3]), min(keys[7], keys[n // 3])
    ids = np.arange(n, dtype=np.uint32)
    part = (keys >> np.uint64(bits[0])) & np.uint64((1 << (bits[1] - bits[0])) - 1)
    order = np.argsort(part, kind="stable")
    ctx.call("fl_sort_set_config", *shape)
    try:
        dk, di = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, ids)
        ctx.call("fl_sort_pairs_u64_u32", dk.ptr, di.ptr, ctypes.c_size_t(n), *bits)
        np.testing.assert_array_equal(di.to_host(), order.astype(np.uint32))
        np.testing.assert_array_equal(dk.to_host(), keys[order])
    finally:
        ctx.call("fl_sort_set_config", 8, 256)


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("bits", [(0, 56), (5, 61), (8, 64)])
def test_bits_beside_the_sorted_ones(ctx, bits, swap):
    """Bits outside the range take no part: in the order that is checked either.  One pair differs only in
    the range's lowest bit, against the bits above the range (or below it)."""
    n, (lo, hi) = PLANNED + 5, bits
    rng = np.random.default_rng(lo)
    top = rng.permutation(n).astype(np.uint64) << np.uint64(1)
    part = top << np.uint64(hi - lo - 23)  # unique but for the pair; every low bit 0
    a, b = n // 3, 2 * n // 3
    part[b] = part[a]
    part[b if swap else a] |= np.uint64(1)
    keys = part << np.uint64(lo)
    if hi < 64:  # the keys as a whole are in order once the high digits are
        above = part > (part[a] | np.uint64(1))
        above[b] = True
        keys[above] |= np.uint64(1) << np.uint64(hi)
    if lo:
        keys |= rng.integers(0, 1 << lo, n, dtype=np.uint64)
    order = np.argsort(part, kind="stable")
    dk, di = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, np.arange(n, dtype=np.uint32))
    ctx.call("fl_sort_pairs_u64_u32", dk.ptr, di.ptr, ctypes.c_size_t(n), *bits)
    np.testing.assert_array_equal(di.to_host(), order.astype(np.uint32))
    np.testing.assert_array_equal(dk.to_host(), keys[order])
