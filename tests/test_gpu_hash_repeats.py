"""Hash build and query with and without repeated and EMPTY keys, at sizes around one round of the
grid, at high load, against sequential insertion (the last input of a key wins)."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray

pytestmark = pytest.mark.gpu

EMPTY = np.uint64(0xFFFFFFFFFFFFFFFF)


@pytest.mark.parametrize("repeat", [False, True])
@pytest.mark.parametrize("with_vals", [False, True])
@pytest.mark.parametrize("n", [1, 255, 257, 152 * 8 * 256 + 1, 3 * 152 * 8 * 256 + 77])
def test_build_and_query(ctx, n, with_vals, repeat):
    rng = np.random.default_rng(n)
    cap = 1 << max(10, int(np.ceil(np.log2(n / 0.7))))
    keys = np.unique(rng.integers(0, 1 << 62, n + n // 8, dtype=np.uint64))[:n]
    rng.shuffle(keys)
    if repeat:
        at = rng.integers(0, n, n // 3 + 1)
        keys[at] = keys[rng.integers(0, n, len(at))]
        keys[rng.integers(0, n, n // 50 + 1)] = EMPTY
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint32) if with_vals else np.arange(n, dtype=np.uint32)
    q = np.concatenate([keys, rng.integers(1 << 62, 1 << 63, n // 4 + 3, dtype=np.uint64), [EMPTY]])
    dk, dv, dq = (DeviceArray.from_host(ctx, a) for a in (keys, vals, q))
    tk, tv = DeviceArray(ctx, (cap,), np.uint64), DeviceArray(ctx, (cap,), np.uint32)
    out = DeviceArray(ctx, (len(q),), np.uint32)
    ctx.call("fl_hash_build", tk.ptr, tv.ptr, ctypes.c_uint64(cap), dk.ptr, dv.ptr if with_vals else None,
             ctypes.c_size_t(n))
    ctx.call("fl_hash_query", tk.ptr, tv.ptr, ctypes.c_uint64(cap), dq.ptr, out.ptr, ctypes.c_size_t(len(q)))
    order = np.argsort(keys, kind="stable")
    s = keys[order]
    pos = np.searchsorted(s, q, side="right") - 1
    hit = (pos >= 0) & (s[np.maximum(pos, 0)] == q) & (q != EMPTY)
    want = np.where(hit, vals[order[np.maximum(pos, 0)]], np.uint32(0xFFFFFFFF))
    np.testing.assert_array_equal(out.to_host(), want.astype(np.uint32))
    stored = tk.to_host()
    assert np.array_equal(np.sort(stored[stored != EMPTY]), np.unique(keys[keys != EMPTY]))
