"""A pool's steps around the size where a level's interior and general bricks share a launch: the
dependency graph, with and without captured graphs, against every launch in order on one stream."""
import numpy as np
import pytest

from fluidloom_gb300 import lbm
from fluidloom_gb300.lbm import Pool

pytestmark = pytest.mark.gpu


def box(e, level):
    c = lbm.cavity(8 * max(e), level, u_lid=0.05)
    c.ext[:] = list(e)
    return c


@pytest.mark.parametrize("cases", [[box((2, 2, 2), 0)], [box((4, 4, 4), 1)], [box((8, 8, 9), 0)], [box((8, 8, 10), 0)],
                                   [box((8, 8, 8), 1), box((4, 4, 6), 2)], [box((9, 9, 9), 0), box((3, 3, 3), 2)]])
@pytest.mark.parametrize("steps", [1, 3])
def test_graph_equals_one_stream(ctx, cases, steps):
    out = []
    for streams, graphs in ((1, 0), (2, 0), (2, 1)):
        p = Pool(ctx, cases)
        p.set_options(graphs=graphs, streams=streams)
        b = p.bricks()
        fl = ((b["x"] + 2 * b["y"] + b["z"]) % 5 == 0).astype(np.int32)  # some bricks refined where the case allows
        p.regrid_flags(fl)
        rng = np.random.default_rng(4)
        n = p.info().num_bricks
        p.upload(lbm.equilibrium(1 + 0.01 * rng.random((n, 512)), 0.02 * rng.random((n, 512, 3))))
        p.step(steps)
        p.step(2)
        out.append(p.populations())
        p.close()
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])
