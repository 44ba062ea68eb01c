"""Performance cases: the work a program on this framework has it do, through its public entry
points, from the smallest calls to the largest.

Kinds (a case is a dict of plain values, "kind" first):

  step     fl_pool_step on a refined pool of lattice-Boltzmann cases, then the populations as a
           field (the loop between two regrids); "monitor" reads the conservation sums each step
  regrid   one regrid of a pool by the application's own flags, after its vorticity indicator
  mesh     one regrid of a bare octree that follows moving features: flags, fl_adapt (2:1 balance,
           split, merge, rebuild in key order, fields carried along), neighbour table
  sort     Hilbert keys of cells and the key/id radix sort
  hash     hash table build and query
  ghost    halo gather and scatter, coarse-to-fine interpolation, restriction
  compact  compaction of live cells into key order and the permutation of a field

Meshes are made here on dense numpy grids (blobs over a threshold, closed to a 2:1 balance), so
their sizes follow from the case alone; flow fields, keys and field values come from the seed.
`exact` restates every computed number in 64 bits in plain torch.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from fluidloom_gb300 import Context
from fluidloom_gb300.amr import AdaptConfig, AdaptStats, Mesh
from fluidloom_gb300.lbm import CX, CY, CZ, INLET, MOVING, OUTLET, WALL, WQ, Pool, cavity, sphere_channel

Q = 19
DEV = "cuda"
OPP = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, Q)]


def listed():
    return [
        # the smallest simulation a user runs: a 32^3 cavity, twenty steps between two regrids
        {"name": "step_cavity", "kind": "step", "flow": "cavity", "n": 1, "edge": 32, "level": 2, "frac": 0.05,
         "shape": 1, "steps": 20, "monitor": False},
        # a batch of independent cavities of mixed sizes advanced in one pool
        {"name": "step_batch", "kind": "step", "flow": "cavity", "n": 24, "edge": 0, "level": 2, "frac": 0.07,
         "shape": 2, "steps": 4, "monitor": False},
        # the flow past a sphere at the headline configuration's size, wake refined to level 3
        {"name": "step_sphere", "kind": "step", "flow": "sphere", "n": 1, "edge": 64, "level": 3, "frac": 0.045,
         "shape": 3, "steps": 2, "monitor": False},
        # obstacles given as a voxel mask, mass and momentum read after every step
        {"name": "step_monitored", "kind": "step", "flow": "mask", "n": 1, "edge": 40, "level": 2, "frac": 0.12,
         "shape": 4, "steps": 6, "monitor": True},
        # a regrid of a mid-size sphere channel: indicator, balance, remap, tables rebuilt
        {"name": "pool_regrid", "kind": "regrid", "flow": "sphere", "n": 1, "edge": 48, "level": 3, "frac": 0.05,
         "shape": 5},
        # a large octree following moving blobs: faces, edges and corners balanced, neighbour rows
        {"name": "mesh_large", "kind": "mesh", "top": 10, "span": 4, "balance": 1, "blobs": 48, "shape": 6, "fields": 0},
        # a small octree with the default face balance and five field components carried along
        {"name": "mesh_small", "kind": "mesh", "top": 7, "span": 2, "balance": 0, "blobs": 12, "shape": 7, "fields": 5},
        # the cell order of a large mesh: keys of shuffled leaves, 63-bit sort
        {"name": "sort_large", "kind": "sort", "cells": 15074927, "bits": 21},
        # the cell order of a small one, keys at the mesh's own depth
        {"name": "sort_small", "kind": "sort", "cells": 40961, "bits": 10},
        # a cell table: build, then as many queries, a sixth of them absent
        {"name": "hash_table", "kind": "hash", "cells": 2500003},
        # a ghost exchange of 19 populations: listed cells out and back, fine ghosts interpolated
        {"name": "ghost_fill", "kind": "ghost", "cells": 262144, "comp": 19, "share": 0.3, "ordered": False},
        # cells dropped from a mesh, the rest back in key order with their fields
        {"name": "compact", "kind": "compact", "cells": 300007, "comp": 8, "keep": 0.8},
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["step", "step", "step", "regrid", "mesh", "mesh", "sort", "hash", "ghost", "compact"])
    shape = rng.randrange(1, 10000)
    if kind in ("step", "regrid"):
        flow = rng.choice(["cavity", "sphere", "mask"])
        c = {"kind": kind, "flow": flow, "n": 1, "level": rng.choice([1, 2, 3]), "frac": round(rng.uniform(0.02, 0.2), 3),
             "shape": shape}
        if flow == "cavity":
            c["n"] = logint(1, 32)
            c["edge"] = 0 if c["n"] > 4 else 8 * rng.randrange(2, 8)
        else:
            c["edge"] = 8 * rng.randrange(2, 7)
        if c["level"] == 3:
            c["frac"] = round(c["frac"] / 4, 4)
        if kind == "step":
            c["steps"] = rng.choice([1, 2, 3, 5])
            c["monitor"] = rng.random() < 0.3
        for _ in range(5):  # within the largest listed case
            if work(c)["bytes"] < 2.5e10:
                break
            c["n"], c["frac"] = max(1, c["n"] // 2), round(c["frac"] / 2, 4)
            if c["kind"] == "step":
                c["steps"] = max(1, c["steps"] // 2)
        return c
    if kind == "mesh":
        top = rng.choice([6, 7, 8, 9])
        return {"kind": kind, "top": top, "span": rng.choice([2, 3]) if top == 9 else rng.choice([1, 2, 3]), "balance": rng.choice([0, 1, 1]),
                "blobs": rng.randrange(4, 49), "shape": shape, "fields": rng.choice([0, 0, 1, 4, 19]) if top < 9 else 0}
    if kind == "sort":
        return {"kind": kind, "cells": logint(1000, 15000000), "bits": rng.choice([8, 10, 13, 17, 21])}
    if kind == "hash":
        return {"kind": kind, "cells": logint(1000, 15000000)}
    if kind == "ghost":
        return {"kind": kind, "cells": logint(2000, 1500000), "comp": rng.choice([1, 3, 4, 5, 19, 27]),
                "share": round(rng.uniform(0.05, 0.9), 3), "ordered": rng.random() < 0.5}
    return {"kind": kind, "cells": logint(1000, 6000000), "comp": rng.choice([1, 2, 3, 4, 8, 19]),
            "keep": round(rng.uniform(0.3, 1.0), 3)}


# ---------------------------------------------------------------- shared pieces
_state = {"ctx": None, "fields": 0}


def _ctx():
    if _state["ctx"] is None:
        _state["ctx"] = Context(0)
    return _state["ctx"]


class _Raw:
    def __init__(self, ptr, shape, kind, strides, owner):
        self.owner = owner  # what frees the memory stays alive as long as a tensor over it
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (int(ptr), False),
                                         "strides": strides, "version": 3}


def _wrap(owner, ptr, shape, kind, strides=None):
    """Device memory of the library as a torch tensor (no copy)."""
    return torch.as_tensor(_Raw(ptr, shape, kind, strides, owner), device=DEV)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _sz(n):
    return ctypes.c_size_t(n)


# ---------------------------------------------------------------- pools: meshes from the case alone
def _flow_cases(case):
    """Per pool case: flow kind and level-0 bricks per axis (x, y, z)."""
    rng = np.random.default_rng(case["shape"])
    out = []
    for _ in range(case["n"]):
        e = (case["edge"] or 8 * int(rng.choice([2, 3, 4, 5, 6, 8]))) // 8
        out.append({"cavity": (e, e, e), "sphere": (2 * e, e, e), "mask": (2 * e, e, e)}[case["flow"]])
    return out


def _lbm_cases(case, seed):
    """The cases as the program sets them up; velocities vary with the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for ext in _flow_cases(case):
        if case["flow"] == "cavity":
            c = cavity(8 * ext[0], case["level"], u_lid=float(rng.uniform(0.04, 0.06)), tau=float(rng.uniform(0.55, 0.7)))
        else:
            nx, ny, nz = (8 * e for e in ext)
            c = sphere_channel(nx, ny, nz, case["level"], radius=ny / 8.0, centre=(nx / 4.0, ny / 2.0, nz / 2.0),
                               u_in=float(rng.uniform(0.035, 0.045)), tau=0.56, band=3.0 * ny / 32.0)
            if case["flow"] == "mask":
                c.has_sphere = 0
                c.bc[:] = [INLET, OUTLET, WALL, MOVING, 0, 0]
                c.wall_u[:] = [0.02, 0.0, 0.0]
        out.append(c)
    return out


def _solid_voxels(case):
    """The voxel mask of a "mask" flow at level 1 (bool z, y, x): a few boxes and a cylinder."""
    (ex, ey, ez), = _flow_cases(case)
    nx, ny, nz = 16 * ex, 16 * ey, 16 * ez
    z, y, x = np.ogrid[:nz, :ny, :nx]
    m = (x - nx * 0.25) ** 2 + (y - ny * 0.5) ** 2 < (ny * 0.1) ** 2
    m = m & (z >= 0)
    m[nz // 4: nz // 2, : ny // 5, nx // 2: nx // 2 + nx // 12] = True
    m[:, -(ny // 6):, nx // 3: nx // 3 + nx // 10] = True
    return m


def _blob_field(n, rng, k):
    """Sum of k Gaussians at the centres of an (nz, ny, nx) grid of bricks (long axis: unit length)."""
    s = max(n)
    z, y, x = (((np.arange(m) + 0.5) / s).astype(np.float32) for m in n)
    v = np.zeros(n, np.float32)
    for _ in range(k):
        c = [rng.uniform(0, m / s) for m in n]
        w = rng.uniform(0.06, 0.2)
        v += (np.exp(-((z - c[0]) / w) ** 2)[:, None, None] * np.exp(-((y - c[1]) / w) ** 2)[None, :, None]
              * np.exp(-((x - c[2]) / w) ** 2)[None, None, :]).astype(np.float32)
    return v


def _grow(b, periodic):
    """b or any of its 26 neighbours."""
    for a in range(3):
        lo, hi = np.roll(b, 1, a), np.roll(b, -1, a)
        if not periodic[a]:
            idx = [slice(None)] * 3
            idx[a] = 0
            lo[tuple(idx)] = False
            idx[a] = -1
            hi[tuple(idx)] = False
        b = b | lo | hi
    return b


def _pair(b):
    return b.reshape(b.shape[0] // 2, 2, b.shape[1] // 2, 2, b.shape[2] // 2, 2).any((1, 3, 5))


def _twice(b):
    return b.repeat(2, 0).repeat(2, 1).repeat(2, 2)


def _near_solid(case, lc, ext, l):
    """Bricks of level l that the pool itself refines: at the sphere's surface, or at mask voxels."""
    n = tuple(e << l for e in ext[::-1])
    if case["flow"] == "sphere":
        f = np.float32
        inv = f(1.0 / (1 << l))
        lo2, hi2 = np.zeros(n, f), np.zeros(n, f)
        for a in range(3):
            i = np.arange(n[2 - a], dtype=f)
            lo, hi, cc = i * f(8) * inv, (i * f(8) + f(8)) * inv, f(lc.sphere_c[a])
            e = cc - np.clip(cc, lo, hi)
            fm = np.maximum(abs(cc - lo), abs(cc - hi))
            shp = [1, 1, 1]
            shp[2 - a] = -1
            lo2, hi2 = lo2 + (e * e).reshape(shp), hi2 + (fm * fm).reshape(shp)
        ro, ri = f(lc.sphere_r) + f(lc.band), max(f(lc.sphere_r) - f(lc.band), f(0))
        return (lo2 <= ro * ro) & (hi2 >= ri * ri)
    return np.zeros(n, bool)


@functools.lru_cache(maxsize=4)
def _splits_of(key, moved):
    case = dict(key)
    rng = np.random.default_rng(1000 + case["shape"])
    L, out = case["level"], []
    for ext, lc in zip(_flow_cases(case), _lbm_cases(case, 0)):
        per = [lc.bc[2 * (2 - a)] == 0 for a in range(3)]
        n = tuple(e << (L - 1) for e in ext[::-1])
        v = _blob_field(n, rng, 5)
        want = v > np.quantile(v, 1.0 - case["frac"])
        here = np.roll(want, moved, 2) if moved else want
        both = want | np.roll(want, 1, 2) if case["kind"] == "regrid" else want
        near = _near_solid(case, lc, ext, L - 1)
        split = [None] * L
        split[L - 1] = here | near
        s = both | near
        for l in range(L - 2, -1, -1):
            s = _pair(_grow(s, per)) | _near_solid(case, lc, ext, l)
            split[l] = s
        if L > 1:  # only bricks that exist can split
            split[L - 1] = split[L - 1] & _twice(split[L - 2])
        out.append(split)
    return out


def _splits(case, moved=0):
    """Per pool case: for each level the bricks (z, y, x) that are split, closed to a 2:1 balance.
    A "regrid" case has two such meshes, its finest bricks moved by one brick of the level above."""
    return _splits_of(tuple(sorted((k, v) for k, v in case.items() if k != "name")), moved)


def _brick_counts(case, moved=0):
    """Leaf bricks per level over all pool cases."""
    n = [0] * (case["level"] + 1)
    for ext, sp in zip(_flow_cases(case), _splits(case, moved)):
        have = ext[0] * ext[1] * ext[2]
        for l in range(case["level"]):
            k = int(sp[l].sum())
            n[l] += have - k
            have = 8 * k
        n[case["level"]] += have
    return n


def _leaf_flags(case, b, moved):
    """Per brick of the pool: 1 where the mesh is finer, -1 where it is coarser than here."""
    fl = np.zeros(len(b["x"]), np.int32)
    for i, sp in enumerate(_splits(case, moved)):
        for l in range(case["level"] + 1):
            k = np.nonzero((b["case_id"] == i) & (b["level"] == l))[0]
            if not len(k):
                continue
            x, y, z = b["x"][k], b["y"][k], b["z"][k]
            if l < case["level"]:
                fl[k[sp[l][z, y, x]]] = 1
            if l > 0:
                fl[k[~sp[l - 1][z >> 1, y >> 1, x >> 1]]] = -1
    return fl


def _view(ctx, s):
    """The pool's populations as a (19, bricks, 512) tensor (the field the library exports)."""
    h, ptr = ctypes.c_uint64(), ctypes.c_void_p()
    ctx.call("fl_pool_populations_field", s["pool"].h, s["field"], ctypes.byref(h))
    ctx.call("fl_soa_device_ptr", h, 0, ctypes.byref(ptr))
    cells, pitch, ver = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_uint64()
    ctx.call("fl_soa_info", h, ctypes.byref(cells), ctypes.byref(pitch), ctypes.byref(ver))
    key = (ptr.value, cells.value, pitch.value)
    if s.get("view_key") != key:
        n = cells.value // 512
        s["view"] = _wrap(s["pool"], ptr.value, (Q, n, 512), "<f4", (pitch.value, 2048, 4))
        s["view_key"] = key
    return s["view"]


def _make_pool(case, seed):
    ctx = _ctx()
    lcs = _lbm_cases(case, seed)
    pool = Pool(ctx, lcs)
    if case["flow"] == "mask":
        pool.set_solid_mask(0, 1, _solid_voxels(case))
    for _ in range(case["level"]):
        b = pool.bricks()
        fl = _leaf_flags(case, b, 0)
        if not (fl > 0).any():
            break
        pool.regrid_flags(np.maximum(fl, 0))
    b = pool.bricks()
    got = np.bincount(b["level"], minlength=case["level"] + 1).tolist()
    if got != _brick_counts(case):
        raise RuntimeError("bricks per level %s, want %s" % (got, _brick_counts(case)))
    _state["fields"] += 1
    s = {"pool": pool, "bricks": b, "lcs": lcs, "field": b"populations_%d" % _state["fields"]}
    f = _view(ctx, s)
    # a smooth flow with some disturbance, slightly off equilibrium
    g = _gen(seed)
    i = torch.arange(512, device=DEV)
    sc = torch.tensor(0.5 ** b["level"].astype(np.float64), dtype=torch.float32, device=DEV)[:, None]
    r = [(8 * torch.tensor(b[k], device=DEV)[:, None] + o + 0.5) * sc
         for k, o in (("x", i & 7), ("y", (i >> 3) & 7), ("z", i >> 6))]
    a = torch.rand((3, 6), generator=g, device=DEV)
    u = []
    for d in range(3):
        w = 0.05 + 0.15 * a[d, :3]
        ph = torch.sin(w[0] * r[0] + 6 * a[d, 3]) * torch.cos(w[1] * r[1] + 6 * a[d, 4]) * torch.cos(w[2] * r[2])
        u.append(0.015 * ph + 0.001 * (torch.rand(ph.shape, generator=g, device=DEV) - 0.5))
    if case["flow"] != "cavity":
        u[0] = u[0] + float(lcs[0].inlet_u[0])
    rho = 1.0 + 0.01 * torch.sin(0.11 * r[0] + 6 * a[0, 5]) * torch.cos(0.07 * r[1])
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    for q in range(Q):
        cu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
        e = 1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq
        f[q] = WQ[q] * (rho * e + 2e-4 * (torch.rand(rho.shape, generator=g, device=DEV) - 0.5))
    torch.cuda.synchronize()
    return s


def _prepare_step(case, seed):
    s = _make_pool(case, seed)
    if case["monitor"]:
        s["sums"] = torch.zeros((case["steps"], case["n"], 4), dtype=torch.float64, device=DEV)
    return s


def _run_step(case, s):
    pool = s["pool"]
    if not case["monitor"]:
        pool.step(case["steps"])
        return {"f": _view(pool.ctx, s)}
    for k in range(case["steps"]):
        pool.step(1)
        pool.ctx.call("fl_pool_conservation_async", pool.h, ctypes.c_void_p(s["sums"][k].data_ptr()))
    return {"f": _view(pool.ctx, s), "sums": s["sums"]}


def _prepare_regrid(case, seed):
    s = _make_pool(case, seed)
    pool = s["pool"]
    # the two meshes the pool moves between, and the application's flags for each move
    there = _leaf_flags(case, s["bricks"], 1)
    f0 = s["view"].clone()
    torch.cuda.synchronize()
    pool.regrid_flags(there)
    s["bricks1"] = pool.bricks()
    back = _leaf_flags(case, s["bricks1"], 0)
    pool.regrid_flags(back)
    b = pool.bricks()
    if any(not np.array_equal(b[k], s["bricks"][k]) for k in b):
        raise RuntimeError("the pool did not come back to its first mesh")
    _view(pool.ctx, s).copy_(f0)
    torch.cuda.synchronize()
    s["flags"], s["at"] = (there, back), 0
    return s


def _run_regrid(case, s):
    pool = s["pool"]
    flags, wmax = pool.flags()
    pool.regrid_flags(s["flags"][s["at"]])
    s["at"] ^= 1
    b = pool.bricks()
    return {"indicator": wmax, "flags": flags, "f": _view(pool.ctx, s), "x": b["x"], "y": b["y"], "z": b["z"],
            "level": b["level"]}


# ---------------------------------------------------------------- bare octrees
def _blob_tables(case, seed):
    """The features before and after a small move.  Centres lie on a 2^-14 grid well inside the unit
    cube and the seed shifts all of them by whole coarse cells, so every seed's mesh has as many leaves."""
    rng = np.random.default_rng(case["shape"])
    k, grid = case["blobs"], 1 << 14
    c = np.round(rng.uniform(0.3, 0.7, (k, 3)) * grid) / grid
    w = rng.uniform(0.02, 0.05, k) * min(1.5, (48 / k) ** (1 / 3))
    move = np.round(rng.uniform(-0.004, 0.004, (k, 3)) * grid) / grid
    cells = 1 << max(3, case["top"] - case["span"])
    far = np.random.default_rng(seed).integers(-(cells // 8), cells // 8 + 1, 3) / cells
    rest = [(1 / (2 * w * w))[:, None], np.ones((k, 1))]
    return [np.ascontiguousarray(np.concatenate([c + far + m] + rest, 1), np.float32) for m in (move, 0 * move)]


BLOB_LO, BLOB_HI = 0.4, 0.7


@functools.lru_cache(maxsize=8)
def _mesh_cells(key):
    """About how many leaves the case's mesh has (its blobs sampled on a 64^3 grid)."""
    case = dict(key)
    t = _blob_tables(case, 0)[1]
    x = (np.arange(64) + 0.5) / 64
    v = np.zeros((64, 64, 64))
    for cx, cy, cz, w, a in t:
        v += a * (np.exp(-w * (x - cz) ** 2)[:, None, None] * np.exp(-w * (x - cy) ** 2)[None, :, None]
                  * np.exp(-w * (x - cx) ** 2)[None, None, :])
    p = float((v > 0.5 * (BLOB_LO + BLOB_HI)).mean())
    return int(p * 8 ** case["top"] + (1 - p) * 8 ** (case["top"] - case["span"]))


def _cells_of(case):
    return _mesh_cells(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


COLS = (("x", "<i4"), ("y", "<i4"), ("z", "<i4"), ("level", "|u1"), ("state", "|u1"), ("flags", "<i4"),
        ("material", "<i4"))


def _column(mesh, name, kind, n):
    return _wrap(mesh, getattr(mesh.m, name), (n,), kind)


def _mesh_pass(ctx, s, case, table):
    """One regrid: flags by the blobs, adapt (carrying the fields), neighbour rows."""
    cfg = AdaptConfig.make(max_level=case["top"], min_level=case["top"] - case["span"], balance_mode=case["balance"],
                           depth=21, anchor=21, input_balanced=case["balance"] == 1 and s["balanced"])
    m = s["mesh"].m
    ctx.call("fl_flags_from_blobs", ctypes.byref(m), table.ctypes.data_as(ctypes.c_void_p), len(table),
             ctypes.c_float(BLOB_LO), ctypes.c_float(BLOB_HI), case["top"])
    st = AdaptStats()
    rc = ctx.lib.fl_adapt(ctx.handle, ctypes.byref(m), ctypes.byref(cfg), ctypes.byref(s["fields"]), case["fields"],
                          ctypes.byref(st))
    if rc not in (0, -5):  # -5: a face balance that stopped at its iteration limit, the mesh is usable
        raise RuntimeError("fl_adapt: %d" % rc)
    s["balanced"] = st.balance.converged == 1
    n = m.num_cells
    if n * 26 > s["nbr"].numel():
        s["nbr"] = torch.empty(n * 26 + n * 6, dtype=torch.int32, device=DEV)
    ctx.call("fl_neighbour_rebuild", ctypes.byref(m), ctypes.byref(cfg), 1, _p(s["nbr"]))
    return st, n


def _prepare_mesh(case, seed):
    ctx = _ctx()
    l0 = case["top"] - case["span"]
    e = 1 << l0
    n = e ** 3
    one = {"x": np.zeros(1, np.int32)}
    mesh = Mesh(ctx, one, capacity=max(n, int(1.2 * _cells_of(case))))
    i = torch.arange(n, device=DEV)
    cols = {"x": i % e, "y": (i // e) % e, "z": i // (e * e), "level": i * 0 + l0, "state": i * 0, "flags": i * 0,
            "material": torch.randint(0, 1 << 20, (n,), generator=_gen(seed), device=DEV)}
    for name, kind in COLS:
        _column(mesh, name, kind, n).copy_(cols[name])
    mesh.m.num_cells = n
    torch.cuda.synchronize()
    s = {"mesh": mesh, "fields": ctypes.c_void_p(0), "balanced": False, "at": 0,
         "nbr": torch.empty(0, dtype=torch.int32, device=DEV)}
    s["tables"] = _blob_tables(case, seed)
    plain = dict(case, fields=0)
    for _ in range(case["span"] + 1):  # into the moving state: features tracked, the rest coarse
        for t in s["tables"]:
            _mesh_pass(ctx, s, plain, t)
    if case["fields"]:
        _, n1 = _mesh_pass(ctx, s, plain, s["tables"][0])
        s["layout1"] = [_column(mesh, k, t, n1).clone() for k, t in COLS[:4]]
        torch.cuda.synchronize()
        _mesh_pass(ctx, s, plain, s["tables"][1])
        n = mesh.m.num_cells
        s["layout0"] = [_column(mesh, k, t, n).clone() for k, t in COLS[:4]]
        p = ctypes.c_void_p()
        ctx.call("fl_device_alloc", _sz(mesh.m.capacity * case["fields"] * 4), ctypes.byref(p))
        _wrap(mesh, p.value, (n, case["fields"]), "<f4").copy_(torch.randn((n, case["fields"]), generator=_gen(seed), device=DEV))
        s["fields"] = p
    torch.cuda.synchronize()
    return s


def _run_mesh(case, s):
    ctx = _ctx()
    st, n = _mesh_pass(ctx, s, case, s["tables"][s["at"]])
    s["at"] ^= 1
    m = s["mesh"].m
    out = {k: _column(s["mesh"], k, t, n) for k, t in COLS}
    out["nbr"] = s["nbr"][: n * 26]
    out["counts"] = np.array([st.num_split, st.num_groups, st.num_survivors, n, st.balance.iterations,
                              st.balance.total_violations_detected, st.balance.total_cells_marked_for_balance])
    if case["fields"]:
        out["fields"] = _wrap(s["mesh"], s["fields"].value, (n, case["fields"]), "<f4")
    return out


# ---------------------------------------------------------------- index primitives
def _cells(case, seed, bits):
    """Anchors of the leaves of a mesh in some order: clustered cells of a few levels."""
    n = case["cells"]
    g = _gen(seed)
    fine = min(bits, 10)
    c = torch.rand((24, 3), generator=g, device=DEV)
    k = torch.randint(0, 24, (n,), generator=g, device=DEV)
    r = (c[k] + 0.08 * torch.randn((n, 3), generator=g, device=DEV)) % 1.0
    lv = fine - torch.randint(0, 3, (n, 1), generator=g, device=DEV)
    a = (r * (1 << fine)).to(torch.int64).clamp_(0, (1 << fine) - 1)
    a = (a >> (fine - lv)) << (fine - lv)
    return [(a[:, d] << (bits - fine)).to(torch.int32).contiguous() for d in range(3)]


def _prepare_sort(case, seed):
    n = case["cells"]
    return {"xyz": _cells(case, seed, case["bits"]), "keys": torch.empty(n, dtype=torch.int64, device=DEV),
            "ids": torch.empty(n, dtype=torch.int32, device=DEV)}


def _run_sort(case, s):
    ctx, n = _ctx(), _sz(case["cells"])
    x, y, z = s["xyz"]
    ctx.call("fl_hilbert_encode", _p(x), _p(y), _p(z), case["bits"], _p(s["keys"]), _p(s["ids"]), n)
    ctx.call("fl_sort_pairs_u64_u32", _p(s["keys"]), _p(s["ids"]), n, 0, 3 * case["bits"])
    return {"keys": s["keys"], "ids": s["ids"]}


def _keys(n, g):
    """n distinct 63-bit keys in no order (an odd multiplier permutes the 63-bit integers)."""
    i = torch.randperm(n, generator=g, device=DEV) + torch.randint(0, 1 << 40, (1,), generator=g, device=DEV)
    return (i * 0x5851F42D4C957F2D) & 0x7FFFFFFFFFFFFFFF


def _prepare_hash(case, seed):
    n, g = case["cells"], _gen(seed)
    ctx = _ctx()
    cap = int(ctx.lib.fl_hash_compute_capacity(n))
    keys = _keys(n + n // 5, g)
    pick = torch.randint(0, n + n // 5, (n,), generator=g, device=DEV)  # a sixth of them not in the table
    return {"cap": cap, "keys": keys[:n].contiguous(), "queries": keys[pick].contiguous(),
            "vals": torch.randint(0, 1 << 31, (n,), generator=g, device=DEV).to(torch.int32),
            "tk": torch.empty(cap, dtype=torch.int64, device=DEV), "tv": torch.empty(cap, dtype=torch.int32, device=DEV),
            "out": torch.empty(n, dtype=torch.int32, device=DEV)}


def _run_hash(case, s):
    ctx, n, cap = _ctx(), _sz(case["cells"]), ctypes.c_uint64(s["cap"])
    ctx.call("fl_hash_build", _p(s["tk"]), _p(s["tv"]), cap, _p(s["keys"]), _p(s["vals"]), n)
    ctx.call("fl_hash_query", _p(s["tk"]), _p(s["tv"]), cap, _p(s["queries"]), _p(s["out"]), n)
    return {"found": s["out"]}


def _ghost_edge(case):
    return max(2, int(round(case["cells"] ** (1 / 3))))


def _prepare_ghost(case, seed):
    """A uniform mesh with a field of C components; a share of its cells listed as halo, fine ghost
    cells over its boundary, the sibling groups of a tenth of it."""
    ctx, g, C = _ctx(), _gen(seed), case["comp"]
    e = _ghost_edge(case)
    n = e ** 3
    lv = e.bit_length()  # the cells past the mesh's upper faces still have coordinates of their own
    mesh = Mesh(ctx, {"x": np.zeros(1, np.int32)}, capacity=n)
    i = torch.arange(n, device=DEV)
    cols = {"x": i % e, "y": (i // e) % e, "z": i // (e * e), "level": i * 0 + lv, "state": i * 0, "flags": i * 0,
            "material": i * 0}
    for name, kind in COLS:
        _column(mesh, name, kind, n).copy_(cols[name])
    mesh.m.num_cells = n
    h = max(1, int(case["share"] * n))
    idx = torch.randperm(n, generator=g, device=DEV)[:h]
    if case["ordered"]:
        idx = idx.sort()[0]
    nq = max(1, h // 4)
    fine = torch.randint(0, 2 * e, (3, nq), generator=g, device=DEV).to(torch.int32)
    groups = max(1, n // 80)
    first = torch.randperm(n // 8, generator=g, device=DEV)[:groups].sort()[0]
    members = first[:, None] * 8 + torch.arange(8, device=DEV)[None]
    s = {"mesh": mesh, "edge": e, "level": lv, "field": torch.randn((n, C), generator=g, device=DEV),
         "idx": idx.to(torch.int32).contiguous(), "back": torch.zeros((n, C), device=DEV),
         "pack": torch.empty((h, C), device=DEV), "fine": [fine[d].contiguous() for d in range(3)],
         "flevel": torch.full((nq,), lv + 1, dtype=torch.uint8, device=DEV), "ghost": torch.empty((nq, C), device=DEV),
         "members": members.to(torch.int32).contiguous(), "coarse": torch.empty((groups, C), device=DEV)}
    s["cfg"] = AdaptConfig.make(max_level=lv + 1, balance_mode=1, depth=21, anchor=21)
    torch.cuda.synchronize()
    return s


def _run_ghost(case, s):
    ctx, C = _ctx(), case["comp"]
    h = _sz(s["idx"].numel())
    ctx.call("fl_pack_halo", _p(s["field"]), C, _p(s["idx"]), h, _p(s["pack"]))
    ctx.call("fl_unpack_halo", _p(s["pack"]), C, _p(s["idx"]), h, _p(s["back"]))
    ctx.call("fl_interp_trilinear", ctypes.byref(s["mesh"].m), ctypes.byref(s["cfg"]), _p(s["field"]), C,
             *[_p(t) for t in s["fine"]], _p(s["flevel"]), _sz(s["flevel"].numel()), _p(s["ghost"]))
    ctx.call("fl_restrict_groups", _p(s["field"]), C, _p(s["members"]), _sz(s["members"].shape[0]), 0, _p(s["coarse"]))
    return {"pack": s["pack"], "back": s["back"], "ghost": s["ghost"], "coarse": s["coarse"]}


def _prepare_compact(case, seed):
    n, g, C = case["cells"], _gen(seed), case["comp"]
    keys = _keys(n, g)
    state = torch.zeros(n, dtype=torch.int32, device=DEV)
    state[torch.randperm(n, generator=g, device=DEV)[:max(1, int(case["keep"] * n))]] = 1
    return {"keys": keys, "state": state, "field": torch.randn((n, C), generator=g, device=DEV),
            "perm": torch.empty(n, dtype=torch.int32, device=DEV), "skeys": torch.zeros(n, dtype=torch.int64, device=DEV),
            "sids": torch.zeros(n, dtype=torch.int32, device=DEV), "dst": torch.zeros((n, C), device=DEV)}


def _run_compact(case, s):
    ctx, n, m = _ctx(), _sz(case["cells"]), ctypes.c_size_t()
    ctx.call("fl_compact_and_permute", _p(s["keys"]), _p(s["state"]), n, _p(s["perm"]), _p(s["skeys"]), _p(s["sids"]),
             ctypes.byref(m))
    ctx.call("fl_apply_permutation", _p(s["field"]), _p(s["dst"]), _sz(4 * case["comp"]), n, _p(s["perm"]))
    k = m.value
    return {"perm": s["perm"], "keys": s["skeys"][:k], "ids": s["sids"][:k], "field": s["dst"][:k]}


PREPARE = {"step": _prepare_step, "regrid": _prepare_regrid, "mesh": _prepare_mesh, "sort": _prepare_sort,
           "hash": _prepare_hash, "ghost": _prepare_ghost, "compact": _prepare_compact}
RUN = {"step": _run_step, "regrid": _run_regrid, "mesh": _run_mesh, "sort": _run_sort, "hash": _run_hash,
       "ghost": _run_ghost, "compact": _run_compact}


def prepare(case, seed):
    s = PREPARE[case["kind"]](case, seed)
    torch.cuda.synchronize()
    s["case"] = case
    return s


def run(state):
    return RUN[state["case"]["kind"]](state["case"], state)


def work(case):
    """Bytes and operations of one pass: each input read and each output written once; a fluid site
    update reads and writes 19 FP32 populations, a pass of the radix sort is not counted."""
    k = case["kind"]
    if k == "step":
        n = _brick_counts(case)
        lups = sum((b * 512) << l for l, b in enumerate(n)) * case["steps"]
        sums = sum(n) * 512 * 76 * case["steps"] if case["monitor"] else 0
        return {"bytes": 152 * lups + sums, "flops": 250 * lups}
    if k == "regrid":
        a, b = sum(_brick_counts(case)), sum(_brick_counts(case, 1))
        return {"bytes": 76 * 512 * (2 * a + b), "flops": 60 * 512 * a}
    if k == "mesh":
        n = _cells_of(case)  # flags 17 B, adapt 22 + 22 B and the fields twice, neighbour rows 13 + 104 B a leaf
        return {"bytes": n * (17 + 44 + 8 * case["fields"] + 117), "flops": 20 * case["blobs"] * n}
    n = case["cells"]
    if k == "sort":
        return {"bytes": 24 * n, "flops": 0}
    if k == "hash":
        return {"bytes": 12 * n + 12 * (1 << 20 if n < 629146 else 1 << math.ceil(math.log2(n / 0.6))) + 12 * n, "flops": 0}
    C = case["comp"]
    if k == "ghost":
        n = _ghost_edge(case) ** 3
        h, groups = max(1, int(case["share"] * n)), max(1, n // 80)
        nq = max(1, h // 4)
        return {"bytes": 4 * h * (2 + 4 * C) + 13 * n + nq * (13 + 36 * C) + groups * (32 + 36 * C),
                "flops": 16 * nq * C + 8 * groups * C}
    return {"bytes": 12 * n + 4 * n + case["keep"] * n * (12 + 8 * C), "flops": 0}


# ---------------------------------------------------------------- the same numbers in 64 bits
class _Octree:
    """Bricks of every case with dense lookup grids at the finest level."""

    def __init__(self, b, lcs, L, mask=None):
        self.L = L
        t = {k: torch.tensor(v.astype(np.int64), device=DEV) for k, v in b.items()}
        self.pos, self.level, self.cs = torch.stack([t["x"], t["y"], t["z"]]), t["level"], t["case_id"]
        self.n = len(self.level)
        self.ext = torch.tensor([list(c.ext) for c in lcs], device=DEV)
        self.bc = torch.tensor([list(c.bc) for c in lcs], device=DEV)
        size = (self.ext << L).prod(1)
        self.off = torch.cumsum(size, 0) - size
        self.grid = torch.zeros(int(size.sum()), dtype=torch.int64, device=DEV)
        for l in range(L + 1):
            k = torch.nonzero(self.level == l)[:, 0]
            d = L - l
            o = torch.arange(1 << (3 * d), device=DEV)
            m = (1 << d) - 1
            p = [(self.pos[a, k] << d)[:, None] + ((o >> (d * a)) & m)[None] for a in range(3)]
            self.grid[self._at(p, self.cs[k][:, None])] = k[:, None].expand(-1, len(o))
        self.lcs = lcs
        f32 = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)  # noqa: E731
        self.sc, self.sr = f32([list(c.sphere_c) for c in lcs]), f32([c.sphere_r for c in lcs])
        self.has = torch.tensor([bool(c.has_sphere) for c in lcs], device=DEV)
        self.mask = None if mask is None else torch.tensor(mask, device=DEV)

    def _at(self, p, cs):
        e = self.ext[cs] << self.L
        return self.off[cs] + (p[2] * e[..., 1] + p[1]) * e[..., 0] + p[0]

    def leaf(self, S, l, cs):
        """The leaf brick holding level-l site S (inside the domain)."""
        return self.grid[self._at([(v << (self.L - l)) >> 3 for v in S], cs)]

    def solid(self, S, l, cs):
        inv = torch.tensor(1.0 / (1 << l), dtype=torch.float32, device=DEV)
        d = [(S[a].to(torch.float32) + 0.5) * inv - self.sc[cs, a] for a in range(3)]
        out = self.has[cs] & (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] < self.sr[cs] * self.sr[cs])
        if self.mask is not None:  # voxels of level 1
            v = [(x << 1) + 1 if l == 0 else x >> (l - 1) for x in S]
            out = out | self.mask[v[2], v[1], v[0]]
        return out

    def sites(self, k):
        i = torch.arange(512, device=DEV)
        return [8 * self.pos[a, k][:, None] + o[None] for a, o in enumerate((i & 7, (i >> 3) & 7, i >> 6))]


CHILD = (0, 1, 8, 9, 64, 65, 72, 73)


class _Stencil:
    """Where every population of the sites of one level comes from."""

    def __init__(self, T, l):
        k = torch.nonzero(T.level == l)[:, 0]
        self.k, self.l = k, l
        own = (k[:, None] * 512 + torch.arange(512, device=DEV)[None])
        self.own = own.reshape(-1)
        cs = T.cs[k][:, None].expand(-1, 512)
        G = T.sites(k)
        self.is_solid = T.solid(G, l, cs).reshape(-1)
        N = [(T.ext[cs, a] * 8) << l for a in range(3)]
        bc = T.bc[cs]
        self.src, self.lists = [], []
        for q in range(Q):
            S = [G[0] - CX[q], G[1] - CY[q], G[2] - CZ[q]]
            out = torch.zeros_like(cs, dtype=torch.bool)
            kind = {3: out.clone(), 4: out.clone(), 2: out.clone()}
            for a in range(3):
                for side, off in ((0, S[a] < 0), (1, S[a] >= N[a])):
                    t = bc[..., 2 * a + side]
                    off = off & (bc[..., 2 * a] != 0)
                    out = out | off
                    for v in kind:
                        kind[v] = kind[v] | (off & (t == v))
                S[a] = torch.where(out, G[a], S[a] % N[a])
            W = [torch.where(out, g, s) for g, s in zip(G, S)]
            rock = T.solid(W, l, cs) & ~out
            leaf = T.leaf(W, l, cs)
            lv = T.level[leaf]
            p = [T.pos[a, leaf] * 8 for a in range(3)]
            at = lambda x: leaf * 512 + (x[0] - p[0]) + 8 * (x[1] - p[1]) + 64 * (x[2] - p[2])  # noqa: E731
            ok = ~out & ~rock
            same, coarse, fine = ok & (lv == l), ok & (lv == l - 1), ok & (lv == l + 1)
            src = torch.where(same, at(W), own)
            src = torch.where(coarse, at([w >> 1 for w in W]), src)
            src = torch.where(fine, at([w << 1 for w in W]), src)
            inlet = out & kind[3]
            outlet = out & ~kind[3] & kind[4]
            wall = out & ~kind[3] & ~kind[4]
            pick = lambda m: torch.nonzero(m.reshape(-1))[:, 0]  # noqa: E731
            self.src.append(src.reshape(-1))
            self.lists.append({"coarse": pick(coarse), "fine": pick(fine), "bounce": pick(rock | wall),
                               "moving": pick(wall & kind[2]), "inlet": pick(inlet), "outlet": pick(outlet)})
        self.cs = cs.reshape(-1)


def _feq(q, rho, u):
    cu = CX[q] * u[0] + CY[q] * u[1] + CZ[q] * u[2]
    return WQ[q] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))


def _substep(T, st, F, Old, sub):
    l = st.l
    f64 = lambda v: torch.tensor(v, dtype=torch.float64, device=DEV)  # noqa: E731
    g = torch.empty((Q, len(st.own)), dtype=torch.float64, device=DEV)
    wall, inlet = f64([list(c.wall_u) for c in T.lcs]), f64([list(c.inlet_u) for c in T.lcs])
    for q in range(Q):
        v, li = F[q][st.src[q]], st.lists[q]
        if len(i := li["coarse"]):
            s = st.src[q][i]
            v[i] = 0.5 * (Old[q][s] + F[q][s]) if sub else Old[q][s]
        if len(i := li["fine"]):
            v[i] = sum(F[q][st.src[q][i] + o] for o in CHILD) / 8.0
        if len(i := li["bounce"]):
            v[i] = F[OPP[q]][st.own[i]]
        if len(i := li["moving"]):
            w = wall[st.cs[i]]
            v[i] += 6.0 * WQ[q] * (CX[q] * w[:, 0] + CY[q] * w[:, 1] + CZ[q] * w[:, 2])
        if len(i := li["inlet"]):
            v[i] = _feq(q, 1.0, inlet[st.cs[i]].T)
        g[q] = v
    rho = g.sum(0)
    u = [sum(c[q] * g[q] for q in range(Q) if c[q]) / rho for c in (CX, CY, CZ)]
    om = f64([1.0 / (2.0 ** l * (float(c.tau0) - 0.5) + 0.5) for c in T.lcs])[st.cs]
    for q in range(Q):
        v = g[q] + om * (_feq(q, rho, u) - g[q])
        v[st.is_solid] = WQ[q]
        Old[q][st.own] = F[q][st.own]
        F[q][st.own] = v


def _exact_step(case, seed):
    s = _make_pool(case, seed)
    L = case["level"]
    T = _Octree(s["bricks"], s["lcs"], L, _solid_voxels(case) if case["flow"] == "mask" else None)
    F = s["view"].to(torch.float64).reshape(Q, -1)
    torch.cuda.synchronize()  # the pool frees its memory on a stream of its own
    s["pool"].close()
    Old = F.clone()
    st = [_Stencil(T, l) for l in range(L + 1)]

    def level(l, sub):
        if len(st[l].own):
            _substep(T, st[l], F, Old, sub)
        if l < L:
            level(l + 1, 0)
            level(l + 1, 1)

    sums = torch.zeros((case["steps"], case["n"], 4), dtype=torch.float64, device=DEV)
    for k in range(case["steps"]):
        level(0, 0)
        if case["monitor"]:
            j = [F.sum(0)] + [sum(c[q] * F[q] for q in range(Q) if c[q]) for c in (CX, CY, CZ)]
            for x in st:
                for d in range(4):
                    v = torch.where(x.is_solid, torch.zeros((), dtype=torch.float64, device=DEV), j[d][x.own])
                    sums[k, :, d].index_add_(0, x.cs, v * 8.0 ** -x.l)
    out = {"f": F.reshape(Q, -1, 512)}
    if case["monitor"]:
        out["sums"] = sums
    return out


def _moved_rows(a, b):
    """For two octree layouts (x, y, z, level | case << 5) whose levels differ by one at most: per cell
    of b its cell of a (same), its parent there, or its eight children there; -1 where there is none."""
    def key(x, y, z, l):
        return (l << 42) | (x << 28) | (y << 14) | z
    a, b = ([t.to(torch.int64) for t in m] for m in (a, b))
    ka, order = key(*a).sort()

    def find(k):
        i = torch.searchsorted(ka, k).clamp_(max=len(ka) - 1)
        return torch.where(ka[i] == k, order[i], torch.full_like(i, -1))
    x, y, z, l = b
    return (find(key(x, y, z, l)), find(key(x >> 1, y >> 1, z >> 1, l - 1)),
            torch.stack([find(key(2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * z + (c >> 2), l + 1)) for c in range(8)]))


def _exact_regrid(case, seed):
    s = _prepare_regrid(case, seed)
    b0, b1 = s["bricks"], s["bricks1"]
    F = s["view"].to(torch.float64)
    T = _Octree(b0, s["lcs"], case["level"], _solid_voxels(case) if case["flow"] == "mask" else None)
    torch.cuda.synchronize()  # the pool frees its memory on a stream of its own
    s["pool"].close()
    # the indicator: max |curl u| of each brick, central differences inside it, one-sided at its faces
    n = F.shape[1]
    j = [F.sum(0)] + [sum(c[q] * F[q] for q in range(Q) if c[q]) for c in (CX, CY, CZ)]
    rock = torch.zeros((n, 512), dtype=torch.bool, device=DEV)
    for l in range(case["level"] + 1):
        k = torch.nonzero(T.level == l)[:, 0]
        rock[k] = T.solid(T.sites(k), l, T.cs[k][:, None].expand(-1, 512))
    u = [torch.where(rock, torch.zeros_like(j[0]), j[d] / j[0]).reshape(n, 8, 8, 8) for d in (1, 2, 3)]

    def dd(v, axis):  # axis 0: x, the last of (brick, z, y, x)
        v = v.movedim(3 - axis, 3)
        o = torch.empty_like(v)
        o[..., 1:7] = 0.5 * (v[..., 2:] - v[..., :6])
        o[..., 0], o[..., 7] = v[..., 1] - v[..., 0], v[..., 7] - v[..., 6]
        return o.movedim(3, 3 - axis)
    w = [dd(u[2], 1) - dd(u[1], 2), dd(u[0], 2) - dd(u[2], 0), dd(u[1], 0) - dd(u[0], 1)]
    wmax = (w[0] ** 2 + w[1] ** 2 + w[2] ** 2).sqrt().reshape(n, 512).max(1)[0] * 2.0 ** T.level
    # the populations on the other mesh: copied, copied to children, or the mean of eight
    t = [{k: torch.tensor(v.astype(np.int64), device=DEV) for k, v in b.items()} for b in (b0, b1)]
    lay = [(b["x"], b["y"], b["z"], b["level"] | (b["case_id"] << 5)) for b in t]
    same, up, down = _moved_rows(*lay)
    F4 = F.reshape(Q, n, 8, 8, 8)
    out = torch.empty((Q, len(same), 8, 8, 8), dtype=torch.float64, device=DEV)
    i = torch.nonzero(same >= 0)[:, 0]
    out[:, i] = F4[:, same[i]]
    x, y, z, _ = lay[1]
    for c in range(8):
        cx, cy, cz = c & 1, (c >> 1) & 1, c >> 2
        i = torch.nonzero((same < 0) & (up >= 0) & ((x & 1) == cx) & ((y & 1) == cy) & ((z & 1) == cz))[:, 0]
        part = F4[:, up[i], 4 * cz:4 * cz + 4, 4 * cy:4 * cy + 4, 4 * cx:4 * cx + 4]
        out[:, i] = part.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
        i = torch.nonzero((same < 0) & (up < 0))[:, 0]
        v = F4[:, down[c][i]].reshape(Q, len(i), 4, 2, 4, 2, 4, 2).mean((3, 5, 7))
        out[:, i, 4 * cz:4 * cz + 4, 4 * cy:4 * cy + 4, 4 * cx:4 * cx + 4] = v
    return {"indicator": wmax, "flags": None, "f": out.reshape(Q, -1, 512), "x": None, "y": None, "z": None, "level": None}


def _exact_mesh(case, seed):
    if not case["fields"]:
        return None
    s = _prepare_mesh(case, seed)
    n = s["mesh"].m.num_cells
    f = _wrap(s["mesh"], s["fields"].value, (n, case["fields"]), "<f4").to(torch.float64)
    same, up, down = _moved_rows(s["layout0"], s["layout1"])
    v = f[same.clamp(min=0)]
    v = torch.where((same < 0)[:, None], f[up.clamp(min=0)], v)
    i = torch.nonzero((same < 0) & (up < 0))[:, 0]
    v[i] = f[down[:, i]].mean(0)
    out = {k: None for k, _ in COLS}
    out.update({"nbr": None, "counts": None, "fields": v})
    torch.cuda.synchronize()  # before the mesh is freed
    return out


def _exact_ghost(case, seed):
    s = _prepare_ghost(case, seed)
    f = s["field"].to(torch.float64)
    idx = s["idx"].long()
    back = torch.zeros_like(f)
    back[idx] = f[idx]
    e, ghost = s["edge"], torch.zeros((s["flevel"].numel(), case["comp"]), dtype=torch.float64, device=DEV)
    base = [t.long() // 2 for t in s["fine"]]
    for c in range(8):
        p = [base[0] + (c & 1), base[1] + ((c >> 1) & 1), base[2] + (c >> 2)]
        ok = (p[0] < e) & (p[1] < e) & (p[2] < e)
        i = ((p[2] * e + p[1]) * e + p[0]).clamp(max=e ** 3 - 1)
        ghost += torch.where(ok[:, None], 0.125 * f[i], torch.zeros_like(f[:1]))
    return {"pack": f[idx], "back": back, "ghost": ghost, "coarse": f[s["members"].long()].mean(1)}


def _exact_compact(case, seed):
    s = _prepare_compact(case, seed)
    live = torch.nonzero(s["state"])[:, 0]
    order = live[s["keys"][live].sort(stable=True)[1]]
    return {"perm": None, "keys": None, "ids": None, "field": s["field"][order].to(torch.float64)}


EXACT = {"step": _exact_step, "regrid": _exact_regrid, "mesh": _exact_mesh, "ghost": _exact_ghost,
         "compact": _exact_compact}


def exact(case, seed):
    f = EXACT.get(case["kind"])
    return f(case, seed) if f else None
