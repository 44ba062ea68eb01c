"""Captured steps across regrids that change how the steps are launched with the same classes of bricks on
every level (the general bricks' early launch, in pools of at most 32 bricks an SM): below that size,
above it and below again, with captured graphs against every launch in order on one stream."""
import numpy as np
import pytest

from fluidloom_gb300 import lbm
from fluidloom_gb300.lbm import Pool

pytestmark = pytest.mark.gpu


def refine(pool, ext):
    """The level-0 bricks of a box at the origin split, every other brick merged."""
    b = pool.bricks()
    inside = np.ones(len(b["x"]), bool)
    for k, e in zip("xyz", ext):
        inside &= (b[k] >> b["level"]) < e
    pool.regrid_flags(np.where(b["level"] == 0, inside, np.where(inside, 0, -1)).astype(np.int32))


@pytest.mark.parametrize("sums", [False, True])
def test_step_across_the_early_launch_limit(ctx, sums):
    boxes = [(5, 6, 3), (7, 5, 4), (5, 6, 3), (7, 5, 4)]
    sizes, out = [], []
    for streams, graphs in ((1, 0), (2, 1)):
        p = Pool(ctx, [lbm.cavity(128, 1, u_lid=0.05)])
        p.set_options(graphs=graphs, streams=streams)
        if sums:
            ctx.call("fl_pool_set_step_sums", p.h, 1)
        refine(p, boxes[0])
        rng = np.random.default_rng(4)
        n = p.info().num_bricks
        p.upload(lbm.equilibrium(1 + 0.01 * rng.random((n, 512)), 0.02 * rng.random((n, 512, 3))))
        got = []
        for box in boxes:
            refine(p, box)
            p.step(3)
            sizes.append(p.info().num_bricks)
            got.append(p.populations())
        out.append(got)
        p.close()
    assert sizes[:4] == [4096 + 7 * 90, 4096 + 7 * 140] * 2 and sizes[0] <= 32 * 152 < sizes[1]
    for a, b in zip(*out):
        np.testing.assert_array_equal(b, a)
