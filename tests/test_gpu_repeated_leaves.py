"""Regrids of meshes that list leaves more than once: an octet merges once, however many copies of its
first sibling (more than the group arrays would hold if each led a group) or of another are listed, in
key order and shuffled, with fields, against the oracle; the other copies stay."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray
from tests import _oracle as O
from tests.test_gpu_amr import cfg, mesh, run_adapt

pytestmark = pytest.mark.gpu


def uniform(level, seed):
    e = 1 << level
    i = np.arange(e ** 3, dtype=np.int32)
    x, y, z = i % e, (i // e) % e, i // e ** 2
    rng = np.random.default_rng(seed)
    octet = x // 2 + (y // 2) * (e // 2) + (z // 2) * (e // 2) ** 2
    return {"x": x, "y": y, "z": z, "level": np.full(e ** 3, level, np.uint8), "state": np.zeros(e ** 3, np.uint8),
            "flags": np.append(-1, rng.choice([-1, -1, 0], e ** 3 // 8 - 1))[octet].astype(np.int32),
            "material": np.arange(e ** 3, dtype=np.uint32)}


def repeated(level, what, times, shuffled):
    cols = uniform(level, 3)
    rng = np.random.default_rng(times)
    first = ((cols["x"] | cols["y"] | cols["z"]) & 1) == 0
    pick = np.nonzero(first if what == "first" else (~first if what == "other" else first | ~first))[0]
    pick = pick[rng.integers(0, len(pick), max(1, len(pick) // 3))]
    p = np.append(np.arange(len(first)), np.repeat(pick, times))
    p = rng.permutation(p) if shuffled else p[np.argsort(O.cell_keys(*[cols[k][p] for k in ("x", "y", "z", "level")],
                                                                      None, 21, 21), kind="stable")]
    return {k: np.ascontiguousarray(v[p]) for k, v in cols.items()}


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("times", [1, 2, 40])
@pytest.mark.parametrize("what", ["first", "other", "any"])
@pytest.mark.parametrize("level", [1, 2, 4])
def test_adapt(ctx, level, what, times, shuffled, mode):
    cols = repeated(level, what, times, shuffled)
    n = len(cols["x"])
    f = np.random.default_rng(1).standard_normal((n, 3)).astype(np.float32)
    kw = dict(max_level=6, min_level=0, balance_mode=mode, max_balance_iterations=10, enforce_balance=1, averaging_rule=0)
    want, wst, wf = O.adapt(cols, kw, O.domain(max_level=6), f, 3)[:3]
    rc, got, st, gf = run_adapt(ctx, cols, cfg(max_level=6, min_level=0, balance_mode=mode), f, 3)
    assert rc in (0, -5)
    for k in ("x", "y", "z", "level", "state", "material", "flags"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    np.testing.assert_array_equal(gf, wf)
    assert st.num_groups == np.count_nonzero(want["level"] == level - 1)
    assert n - 8 * st.num_groups + st.num_groups == len(got["x"])


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("times", [1, 40])
def test_merge(ctx, times, shuffled):
    cols = repeated(2, "first", times, shuffled)
    m, out = mesh(ctx, cols), mesh(ctx, uniform(2, 0))
    n = len(cols["x"])
    group, count = DeviceArray(ctx, (n,), np.uint32), ctypes.c_size_t()
    ctx.call("fl_merge", ctypes.byref(m.m), ctypes.byref(cfg(max_level=6, min_level=0)), None, 0, ctypes.byref(out.m), None,
             group.ptr, ctypes.byref(count))
    g = group.to_host()
    merged = uniform(2, 3)["flags"].reshape(2, 2, 2, 2, 2, 2)[:, 0, :, 0, :, 0] == -1
    assert count.value == np.count_nonzero(merged)
    assert (np.bincount(g[g != 0xFFFFFFFF], minlength=count.value) == 8).all()
