"""Merge groups filed as they are found, and the face balance's table built from the cells: octets
drawn to merge, keep or split with stray cells among them, ragged counts, FACE6 and FULL26, in key
order and shuffled, with fields, against the oracle."""
import numpy as np
import pytest

from tests import _oracle as O
from tests.test_gpu_amr import cfg, run_adapt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("cut", [0, 3])
@pytest.mark.parametrize("level", [1, 2, 4])
def test_merge_groups(ctx, level, cut, shuffled, mode):
    e = 1 << level
    rng = np.random.default_rng(10 * level + cut)
    i = np.arange(e ** 3, dtype=np.int32)
    x, y, z = i % e, (i // e) % e, i // e ** 2
    octet = x // 2 + (y // 2) * (e // 2) + (z // 2) * (e // 2) ** 2
    fl = rng.choice([-1, -1, 0, 1], e ** 3 // 8)[octet]
    fl = np.where(rng.integers(0, 25, e ** 3) == 0, rng.integers(-1, 2, e ** 3), fl).astype(np.int32)
    cols = {"x": x, "y": y, "z": z, "level": np.full(e ** 3, level, np.uint8), "state": np.zeros(e ** 3, np.uint8),
            "flags": fl, "material": rng.integers(0, 9, e ** 3).astype(np.uint32)}
    p = rng.permutation(e ** 3)
    if not shuffled:
        p = np.argsort(O.cell_keys(x, y, z, cols["level"], None, 21, 21), kind="stable")
    p = p[:e ** 3 - cut]  # a mesh that does not fill its domain
    cols = {k: np.ascontiguousarray(v[p]) for k, v in cols.items()}
    f = rng.standard_normal((len(p), 3)).astype(np.float32)
    kw = dict(max_level=6, min_level=0, balance_mode=mode, max_balance_iterations=10, enforce_balance=1, averaging_rule=0)
    want, wst, wf = O.adapt(cols, kw, O.domain(max_level=6), f, 3)[:3]
    rc, got, st, gf = run_adapt(ctx, cols, cfg(max_level=6, min_level=0, balance_mode=mode), f, 3)
    assert rc in (0, -5)
    for k in ("x", "y", "z", "level", "state", "material", "flags"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    np.testing.assert_array_equal(gf, wf)
