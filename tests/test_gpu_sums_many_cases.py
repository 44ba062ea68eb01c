"""Conservation sums of pools of few and of many cases, of one chunk of bricks and of several, bit for bit: a case's
sums do not depend on the other cases of the pool."""
import numpy as np
import pytest

from fluidloom_gb300 import lbm
from fluidloom_gb300.lbm import Pool

pytestmark = pytest.mark.gpu

EXTS = [(1, 1, 1), (2, 1, 1), (3, 3, 3), (16, 8, 1), (5, 5, 6), (1, 2, 1), (9, 16, 2), (12, 8, 4), (16, 16, 2), (16, 11, 3)]


def sums(ctx, exts):
    cases = [lbm.periodic_box(8 * e[0], 8 * e[1], 8 * e[2], 0) for e in exts]
    pool = Pool(ctx, cases)
    b = pool.bricks()
    n = len(b["x"])
    # a field of the brick's place and its case's shape alone
    at = ((b["x"] * 31 + b["y"]) * 37 + b["z"]).astype(np.float64)[:, None] + np.arange(512) / 512
    f = np.stack([lbm.WQ[q] * (1 + 0.01 * np.sin(at * (q + 1))) for q in range(19)]).astype(np.float32)
    pool.upload(f.reshape(19, n, 512))
    got = pool.conservation()
    pool.close()
    return got


@pytest.mark.parametrize("copies", [1, 25, 26, 28])
def test_sums_of_many_cases(ctx, copies):
    want = np.concatenate([sums(ctx, [e]) for e in EXTS])
    np.testing.assert_array_equal(sums(ctx, EXTS * copies), np.tile(want, (copies, 1)))
