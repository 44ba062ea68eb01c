"""Neighbour rows of single-case meshes, located through the leaves' octree, against the sorted
locator (which serves the same mesh when it carries a case column): meshes that fill their domain, in
key order and shuffled, unbalanced, deep at one corner, on one level, periodic, above the probes'
level limit -- and those that have no octree, with holes, overlaps, repeated or outside leaves, in a
domain far larger than the leaves."""
import ctypes

import numpy as np
import pytest

from fluidloom_gb300 import DeviceArray
from fluidloom_gb300.amr import AdaptConfig, Mesh
from tests import _oracle as O

pytestmark = pytest.mark.gpu


def rows(ctx, cols, sub, **kw):
    m = Mesh(ctx, cols)
    out = DeviceArray(ctx, (len(cols["x"]) * 26 * sub,), np.uint32)
    ctx.call("fl_neighbour_rebuild", ctypes.byref(m.m), ctypes.byref(AdaptConfig.make(**kw)), sub, out.ptr)
    return out.to_host()


def both(ctx, cols, **kw):
    # of a repeated leaf either copy may be named: the sorted locator's two passes race for it
    _, cell = np.unique(np.stack([cols[k].astype(np.int64) for k in ("x", "y", "z", "level")]), axis=1,
                        return_inverse=True)
    cell = np.append(cell.reshape(-1), -1)
    for sub in (1, 4):
        want = rows(ctx, dict(cols, case_id=np.zeros(len(cols["x"]), np.uint16)), sub, **kw)
        got = rows(ctx, cols, sub, **kw)
        if len(np.unique(cell)) == len(cell):
            np.testing.assert_array_equal(got, want)
        none = np.uint32(0xFFFFFFFF)
        np.testing.assert_array_equal(*[cell[np.where(r == none, len(cell) - 1, r)] for r in (got, want)])


def take(cols, i):
    return {k: np.ascontiguousarray(v[i]) for k, v in cols.items()}


def corner(depth):
    """One chain of splits at the lowest corner: leaves of every level from 1 to depth."""
    x, y, z, lv = [], [], [], []
    for l in range(1, depth + 1):
        for c in range(1 if l < depth else 0, 8):
            x.append(c & 1), y.append((c >> 1) & 1), z.append(c >> 2), lv.append(l)
    n = len(x)
    return {"x": np.array(x, np.int32), "y": np.array(y, np.int32), "z": np.array(z, np.int32),
            "level": np.array(lv, np.uint8), "state": np.zeros(n, np.uint8), "flags": np.zeros(n, np.int32),
            "material": np.zeros(n, np.uint32)}


@pytest.mark.parametrize("periodic", [(0, 0, 0), (1, 1, 1), (0, 1, 0)])
@pytest.mark.parametrize("ext", [(1, 1, 1), (2, 1, 3), (5, 2, 1)])
@pytest.mark.parametrize("balanced", [True, False])
def test_filled(ctx, ext, periodic, balanced):
    cols = O.random_octree(sum(ext) + balanced, ext=ext, rounds=4, max_level=6, frac=0.25, balanced=balanced)
    kw = dict(max_level=6, ext=ext, periodic=periodic)
    both(ctx, cols, **kw)
    both(ctx, take(cols, np.random.default_rng(1).permutation(len(cols["x"]))), **kw)
    both(ctx, cols, **dict(kw, max_level=4))  # leaves deeper than the limit are no one's neighbour


@pytest.mark.parametrize("depth", [1, 2, 5, 9, 13, 20])
def test_deep_corner(ctx, depth):
    both(ctx, corner(depth), max_level=depth)


@pytest.mark.parametrize("level", [0, 1, 3, 5])
def test_uniform(ctx, level):
    both(ctx, O.uniform_mesh(level, (1, 1, 1)), max_level=8, periodic=(1, 0, 1))
    both(ctx, O.uniform_mesh(level, (3, 2, 1)), max_level=8, ext=(3, 2, 1))


@pytest.mark.parametrize("seed", range(4))
def test_no_octree(ctx, seed):
    rng = np.random.default_rng(seed)
    full = O.random_octree(30 + seed, ext=(2, 2, 2), rounds=3, max_level=5, frac=0.3, balanced=False)
    n = len(full["x"])
    kw = dict(max_level=6, ext=(2, 2, 2), periodic=(seed & 1, 0, 0))
    both(ctx, take(full, rng.random(n) < 0.9), **kw)                                  # holes
    both(ctx, take(full, np.sort(np.append(np.arange(n), rng.integers(0, n, 5)))), **kw)  # repeated leaves
    i = rng.integers(0, n, 4)
    child = {k: np.concatenate([v, (v[i] * 2 if k in "xyz" else v[i] + (k == "level")).astype(v.dtype)])
             for k, v in full.items()}
    both(ctx, child, **kw)                                                            # children of leaves
    outside = {k: v.copy() for k, v in full.items()}
    outside["x"][rng.integers(0, n, 2)] += 1 << 7
    both(ctx, outside, **kw)
    both(ctx, take(full, np.arange(min(n, 20))), max_level=6, ext=(60, 50, 40), depth=21, anchor=15)
