"""A regrid's emission where groups of 32 cells change between plain and split ones: ragged counts,
all kept, all split, all merged, single cells in between, in key order and shuffled, with and without
fields and case ids, against the oracle."""
import numpy as np
import pytest

from tests import _oracle as O
from tests.test_gpu_amr import cfg, run_adapt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [0, 1, 5, 40])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("what", ["keep", "split all", "merge all", "one split", "one in forty", "mixed"])
def test_emit_groups(ctx, what, shuffled, C):
    cols = O.random_octree(5, ext=(2, 1, 1), rounds=3, max_level=5, frac=0.3, balanced=True)
    rng = np.random.default_rng(2)
    n = len(cols["x"])
    fl = np.zeros(n, np.int32)
    if what == "split all":
        fl[:] = 1
    elif what == "merge all":
        fl[:] = -1
    elif what == "one split":
        fl[n // 2] = 1
    elif what == "one in forty":
        fl[::40] = 1
        fl[7::40] = -1
    elif what == "mixed":
        fl = rng.integers(-1, 2, n).astype(np.int32)
    cols = dict(cols, flags=fl, material=rng.integers(0, 99, n).astype(np.uint32))
    if shuffled:
        p = rng.permutation(n)
        cols = {k: np.ascontiguousarray(v[p]) for k, v in cols.items()}
    fields = rng.standard_normal((n, C)).astype(np.float32) if C else None
    kw = dict(max_level=6, min_level=0, balance_mode=1, max_balance_iterations=10, enforce_balance=1, averaging_rule=0)
    want, wst, wf = O.adapt(cols, kw, O.domain(ext=(2, 1, 1), max_level=6), fields, C)[:3]
    rc, got, st, gf = run_adapt(ctx, cols, cfg(max_level=6, min_level=0, balance_mode=1, ext=(2, 1, 1)), fields, C)
    assert rc in (0, -5)
    for k in ("x", "y", "z", "level", "state", "material", "flags"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    if C:
        np.testing.assert_array_equal(gf, wf)
