"""Large sorts whose low digits take few values that the high digits do not decide: a small tag beside repeated
keys, pairs and longer runs of one high part, few and many, up to more than are sorted by themselves; the result
against numpy's stable sort, and the time against keys that fill their digits."""
import ctypes
import time

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray

pytestmark = pytest.mark.gpu

N = (2 << 20) + 4099


def spread(v):
    """Distinct 30-bit values of distinct ones below 2^30."""
    return (v * np.uint64(0x2545F491)) & np.uint64((1 << 30) - 1)


def make(n, what, run, rng):
    low = rng.integers(0, 1 << 33, 11, dtype=np.uint64)
    own = spread(rng.permutation(n).astype(np.uint64))
    if what == "tags":  # one digit: a tag beside keys that come up run times each
        return (spread(rng.integers(0, n // run, n, dtype=np.uint64)) << np.uint64(33)) | rng.integers(0, 4, n, dtype=np.uint64)
    top = own
    k = n // 10 if what == "many" else 3 * run
    if what == "all":
        top = spread(rng.permutation(n).astype(np.uint64) // np.uint64(run))
    else:  # k keys in runs of one high part, the others on their own, set by it
        top = own.copy()
        at = rng.choice(n, k, replace=False)
        top[at] = top[at[np.arange(k) // run * run]]
    keys = (top << np.uint64(33)) | low[top % np.uint64(11)]
    free = rng.random(n) < 0.5 if what == "all" else np.isin(np.arange(n), at if what != "set" else [])
    return np.where(free, (top << np.uint64(33)) | low[rng.integers(0, 11, n)], keys)


def check(ctx, keys, bits):
    n = len(keys)
    part = (keys >> np.uint64(bits[0])) & np.uint64((1 << (bits[1] - bits[0])) - 1)
    order = np.argsort(part, kind="stable")
    dk, di = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, np.arange(n, dtype=np.uint32))
    ctx.call("fl_sort_pairs_u64_u32", dk.ptr, di.ptr, ctypes.c_size_t(n), *bits)
    np.testing.assert_array_equal(di.to_host(), order.astype(np.uint32))
    np.testing.assert_array_equal(dk.to_host(), keys[order])


@pytest.mark.parametrize("shape", [(8, 256), (9, 512)])
@pytest.mark.parametrize("run", [2, 3, 31, 32, 33, 64, 65, 1000, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("what", ["tags", "all", "many", "few"])
def test_runs(ctx, what, run, shape):
    keys = make(N, what, run, np.random.default_rng(run))
    ctx.call("fl_sort_set_config", *shape)
    try:
        check(ctx, keys, (0, 63))
        if run in (33, 1025):
            check(ctx, keys, (3, 63))
            check(ctx, keys, (0, 64))
    finally:
        ctx.call("fl_sort_set_config", 8, 256)


@pytest.mark.parametrize("bits", [(0, 63), (0, 55), (3, 63)])
@pytest.mark.parametrize("run", [2, 1024, 1025, 1057, 4096, 100003])
def test_runs_the_sample_misses(ctx, run, bits):
    """Runs on none of the sampled places (their hash, and the keys drawn)."""
    w = np.arange(1, max(16 * int(N ** 0.5), N // 256) + 1, dtype=np.uint64)
    g = np.uint64(0x9e3779b97f4a7c15)
    h = w * g
    h = (h ^ (h >> np.uint64(32))) * g
    h = (h ^ (h >> np.uint64(29))) * g
    seen = [int(x) * N >> 64 for x in h]
    rng = np.random.default_rng(run)
    keys = make(N, "set", 2, rng)
    low = np.unique(keys & np.uint64((1 << 33) - 1))
    free = rng.permutation(np.setdiff1d(np.arange(N), seen))
    for k in range(2):
        at = free[k * run: (k + 1) * run]
        keys[at] = (keys[at[0]] >> np.uint64(33) << np.uint64(33)) | low[rng.integers(0, len(low), run)]
    check(ctx, keys, bits)


def test_runs_at_the_ends(ctx):
    """The first and the last keys in order are runs."""
    for run in (2, 33, 1024):
        keys = make(N, "set", run, np.random.default_rng(run))
        low = np.unique(keys & np.uint64((1 << 33) - 1))
        rng = np.random.default_rng(1)
        for top in (0, (1 << 30) - 1):
            at = rng.choice(N, run, replace=False)
            keys[at] = (np.uint64(top) << np.uint64(33)) | low[rng.integers(0, len(low), run)]
        check(ctx, keys, (0, 63))


@pytest.mark.parametrize("what,run", [("tags", 2), ("tags", 600), ("all", 2), ("all", 40), ("many", 2), ("few", 2), ("few", 300)])
def test_low_digits_undecided_cost_no_second_sort(ctx, what, run):
    """Not dearer than keys that fill their digits, but for a tenth."""
    n = 4 << 20
    rng = np.random.default_rng(5)
    t = []
    for keys in (rng.integers(0, 1 << 63, n, dtype=np.uint64), make(n, what, run, rng)):
        dk, di = DeviceArray.from_host(ctx, keys), DeviceArray.from_host(ctx, np.arange(n, dtype=np.uint32))
        ts = []
        for _ in range(15):
            ctx.call("fl_memcpy_h2d", dk.ptr, keys.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(8 * n))
            t0 = time.perf_counter()
            ctx.call("fl_sort_pairs_u64_u32", dk.ptr, di.ptr, ctypes.c_size_t(n), 0, 63)
            ctx.call("fl_ctx_synchronize")
            ts.append(time.perf_counter() - t0)
        t.append(float(np.median(ts)))
    assert t[1] < 1.1 * t[0], t
