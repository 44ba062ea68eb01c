"""Neighbour rows of single-case meshes with gaps, through the octree whose missing nodes are made for the leaves
that want them, against the sorted locator (which serves the same mesh when it carries a case column): a node's
lowest corner left out, chains of them, few and most leaves left out, in key order and shuffled; and what such
meshes, and those that the octree can't serve, take beside the sorted locator alone."""
import ctypes
import time

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray
from fluidloom_gb300.amr import AdaptConfig, Mesh
from tests import _oracle as O
from tests.test_gpu_neighbours_octree import both, corner, take

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("keep", [0.02, 0.2, 0.5, 0.8, 0.98])
@pytest.mark.parametrize("shuffled", [False, True])
def test_random_gaps(ctx, keep, seed, shuffled):
    full = O.random_octree(60 + seed, ext=(2, 1, 2), rounds=4, max_level=6, frac=0.3, balanced=seed > 0)
    n = len(full["x"])
    rng = np.random.default_rng(seed)
    i = np.nonzero(rng.random(n) < keep)[0]
    both(ctx, take(full, rng.permutation(i) if shuffled else i), max_level=6, ext=(2, 1, 2), periodic=(seed & 1, 0, seed >> 1))


@pytest.mark.parametrize("level", [1, 2, 3, 4, 5])
def test_low_corners_left_out(ctx, level):
    full = O.random_octree(70, ext=(2, 2, 1), rounds=4, max_level=6, frac=0.4, balanced=False)
    low = ((full["x"] | full["y"] | full["z"]) & 1) == 0
    both(ctx, take(full, np.nonzero(~(low & (full["level"] >= level)))[0]), max_level=6, ext=(2, 2, 1))


@pytest.mark.parametrize("depth", [2, 3, 6, 8, 9, 13])
def test_deep_corner_left_out(ctx, depth):
    """The chain's lowest leaf, whose nodes are every other leaf's too; and the finest octet alone."""
    c = corner(depth)
    both(ctx, take(c, np.nonzero(~((c["level"] == depth) & ((c["x"] | c["y"] | c["z"]) == 0)))[0]), max_level=depth)
    both(ctx, take(c, np.nonzero(c["level"] == depth)[0]), max_level=depth)
    both(ctx, take(c, np.nonzero((c["level"] == depth) & (c["x"] == 1))[0]), max_level=depth)


@pytest.mark.parametrize("seed", range(3))
def test_gaps_and_overlaps(ctx, seed):
    """A child of a leaf, and a parent of leaves, next to gaps: the rows are the sorted locator's."""
    full = O.random_octree(80 + seed, ext=(1, 1, 1), rounds=4, max_level=5, frac=0.4, balanced=False)
    n = len(full["x"])
    rng = np.random.default_rng(seed)
    mesh = take(full, np.nonzero(rng.random(n) < 0.8)[0])
    i = rng.integers(0, len(mesh["x"]), 3)
    for up in (False, True):
        more = {k: (v[i] // 2 if up else v[i] * 2) if k in "xyz" else v[i] for k, v in mesh.items()}
        more["level"] = more["level"] - np.minimum(more["level"], 1) if up else more["level"] + np.uint8(1)
        both(ctx, {k: np.concatenate([v, more[k].astype(v.dtype)]) for k, v in mesh.items()}, max_level=6)


def refined_corner(level):
    """All leaves of one level, those of one octant split once."""
    e = 1 << level
    i = np.arange(e ** 3, dtype=np.int32)
    p = np.stack([i % e, i // e % e, i // e ** 2])
    inside = (p < e // 2).all(0)
    c = np.arange(8)
    fine = (2 * p[:, inside][:, :, None] + np.stack([c & 1, c >> 1 & 1, c >> 2])[:, None, :]).reshape(3, -1)
    x, y, z = np.concatenate([p[:, ~inside], fine], axis=1).astype(np.int32)
    n, coarse = len(x), int((~inside).sum())
    return {"x": x, "y": y, "z": z, "level": np.where(np.arange(n) < coarse, level, level + 1).astype(np.uint8),
            "state": np.zeros(n, np.uint8), "flags": np.zeros(n, np.int32), "material": np.zeros(n, np.uint32)}


@pytest.mark.parametrize("what", ["one gap", "gaps", "listed twice"])
def test_not_dearer_than_the_sorted_locator(ctx, what):
    full = refined_corner(7)
    n = len(full["x"])
    i = np.arange(n)
    deep = np.nonzero((full["level"] == 8) & (((full["x"] | full["y"] | full["z"]) & 1) == 0))[0]
    if what == "one gap":
        i = np.delete(i, deep[len(deep) // 2])
    elif what == "gaps":
        i = i[np.random.default_rng(1).random(n) < 0.98]
    else:
        i = np.append(i, deep[3])
    cols, t = take(full, i), []
    for with_case in (True, False):
        m = Mesh(ctx, dict(cols, case_id=np.zeros(len(i), np.uint16)) if with_case else cols)
        out = DeviceArray(ctx, (len(i) * 26,), np.uint32)
        cfg, ts = AdaptConfig.make(max_level=8), []
        for _ in range(15):
            ctx.call("fl_ctx_synchronize")
            t0 = time.perf_counter()
            ctx.call("fl_neighbour_rebuild", ctypes.byref(m.m), ctypes.byref(cfg), 1, out.ptr)
            ts.append(time.perf_counter() - t0)
        t.append(float(np.median(ts)))
    assert t[1] < (1.15 if what == "listed twice" else 1.05) * t[0], t  # listed twice: a wait more, then the locator
