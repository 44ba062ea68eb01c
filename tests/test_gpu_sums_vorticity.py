"""Conservation sums around the chunk size and the vorticity indicator with solids, extremes and NaN,
against FP64 / FP32 restatements in numpy."""
import numpy as np
import pytest

from fluidloom_gb300 import lbm
from fluidloom_gb300.lbm import Pool

pytestmark = pytest.mark.gpu


def fill(pool, seed):
    n = pool.info().num_bricks
    rng = np.random.default_rng(seed)
    f = (lbm.equilibrium(1 + 0.02 * rng.random((n, 512)), 0.05 * (rng.random((n, 512, 3)) - 0.5))
         + 1e-4 * rng.random((19, n, 512))).astype(np.float32)
    pool.upload(f)
    return f


@pytest.mark.parametrize("ext", [(1, 1, 1), (4, 4, 8), (5, 5, 5), (16, 8, 1), (16, 9, 1), (13, 5, 4)])
def test_sums_around_the_chunk_size(ctx, ext):
    """1 to 260 bricks: below, at and above one, and two, chunks of 128; two cases in a pool."""
    cases = [lbm.periodic_box(8 * ext[0], 8 * ext[1], 8 * ext[2], 0), lbm.cavity(16, 0)]
    pool = Pool(ctx, cases)
    f = fill(pool, sum(ext)).astype(np.float64)
    cs = pool.bricks()["case_id"]
    got = pool.conservation()
    for c in range(2):
        g = f[:, cs == c]
        want = [g.sum()] + [np.tensordot(np.asarray(d, np.float64), g, 1).sum() for d in (lbm.CX, lbm.CY, lbm.CZ)]
        # FP32 moments of a site: at most 19 roundings of sums below 2 each, over all sites
        np.testing.assert_allclose(got[c], want, rtol=0, atol=19 * 2 ** -23 * 512 * g.shape[1])
    pool.close()


def test_vorticity_solids_and_nan(ctx):
    case = lbm.sphere_channel(32, 16, 16, 1, radius=3.0, centre=(8.0, 8.0, 8.0), band=1.0)
    pool = Pool(ctx, [case])
    f = fill(pool, 3)
    b = pool.bricks()
    n = f.shape[1]
    f[:, n - 1] = np.nan                      # every site of a brick
    f[:, n - 2, 100] = np.nan                 # one site
    f[:, n - 3] = np.float32(lbm.WQ[0]) / 19  # uniform
    pool.upload(f)
    _, got = pool.flags()
    # the moments in the kernel's FP32 order
    r = f[0].copy()
    for q in range(1, 19):
        r = r + f[q]
    d = lambda i, j: f[i] - f[j]  # noqa: E731
    jx = ((((d(1, 2)) + d(7, 8)) + d(9, 10)) + d(11, 12)) + d(13, 14)
    jy = ((((d(3, 4)) + d(7, 8)) + d(10, 9)) + d(15, 16)) + d(17, 18)
    jz = ((((d(5, 6)) + d(11, 12)) + d(14, 13)) + d(15, 16)) + d(18, 17)
    inv = np.float32(1) / r
    p = lbm.site_centres(b).astype(np.float32)
    c = np.float32([8, 8, 8])
    e = p - c
    solid = (e[..., 0] * e[..., 0] + e[..., 1] * e[..., 1]) + e[..., 2] * e[..., 2] < np.float32(9)
    u = [np.where(solid, np.float32(0), j * inv).reshape(n, 8, 8, 8) for j in (jx, jy, jz)]

    def dd(v, axis):
        v = np.moveaxis(v, 3 - axis, 3)
        o = np.empty_like(v)
        o[..., 1:7] = (v[..., 2:] - v[..., :6]) * np.float32(0.5)
        o[..., 0], o[..., 7] = v[..., 1] - v[..., 0], v[..., 7] - v[..., 6]
        return np.moveaxis(o, 3, 3 - axis)
    w = [dd(u[2], 1) - dd(u[1], 2), dd(u[0], 2) - dd(u[2], 0), dd(u[1], 0) - dd(u[0], 1)]
    mag = np.sqrt((w[0] * w[0] + w[1] * w[1]) + w[2] * w[2]) * (2.0 ** b["level"].astype(np.float32))[:, None, None, None]
    flat = mag.reshape(n, 512)
    want = np.where(np.isnan(flat).all(1), np.float32(np.nan), np.nanmax(np.where(np.isnan(flat).all(1)[:, None], 0, flat), 1))
    np.testing.assert_array_equal(got, want.astype(np.float32))
    pool.close()
