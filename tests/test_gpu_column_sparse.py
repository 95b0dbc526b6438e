"""Long, nearly empty columns in the column kernel: groups of particles spread over hundreds of cells. A pair's
two forces are exact negations, a pair at the cutoff of a Morse table (0.465 there) acts in full or not at all
by the reference's r^2, and the forces point along the displacement as closely as in a full box."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu

MORSE = (0.2, 5.0, 0.6, 1e-4, 2.0, 1e-3)


def _pairs(nz, share, rng):
    """Isolated pairs: the first particle in every third cell of every third column, a share of them taken."""
    g = np.stack(np.meshgrid([0, 3], [0, 3], np.arange(0, nz - 2, 3), indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.uniform(size=len(g)) < share]
    u = np.abs(rng.normal(size=g.shape))
    u /= np.linalg.norm(u, axis=1)[:, None]
    r = rng.uniform(0.1, 0.98, size=len(g))
    at = rng.uniform(size=len(g)) < 0.5
    r[at] = 1 + rng.integers(-3, 4, size=at.sum()) * 6e-8
    a = g + rng.uniform(0.05, 0.95, size=g.shape)
    return a, a + u * r[:, None], at


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("nz,share", [(45, 1.0), (300, 0.5), (1800, 0.08), (6000, 0.02)])
def test_pairs_in_long_columns(nz, share, variant):
    rng = np.random.default_rng(nz)
    xa, xb, at = _pairs(nz, share, rng)
    n = len(xa)
    dim = np.array([6.0, 6.0, float(nz)])
    x = np.mod(np.concatenate([xa, xb]), dim)
    u = W.build_gpu(dict(dim=list(dim), cells=[6, 6, nz], cutoff=1.0, dt=0.01, bc=("periodic",) * 3,
                         types=[(1.0, 0.7, m.Newtonian)], pots=[("morse", MORSE, 0, 0)], forces=[], x=x,
                         v=np.zeros((2 * n, 3), np.float32), t=np.zeros(2 * n, dtype=np.int32)))
    u.force_config(variant, 1 << 20)
    u.force()
    _, _, f, c, xr = u.state()
    u.close()
    cell = np.stack([c // (6 * nz), c // nz % 6, c % nz], -1)
    off = cell[n:] - cell[:n]
    off -= (dim * np.round(off / dim)).astype(int)
    fa, fb = f[:n], f[n:]
    assert np.array_equal(fa, -fb)
    # the reference's displacement: the first of two cells is the one with the lower offset to the other
    o = off.astype(np.float32)
    first = np.array([tuple(k) >= (0, 0, 0) for k in off])[:, None]
    d = np.where(first, (xr[:n] - o) - xr[n:], -((xr[n:] + o) - xr[:n]))
    r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    assert r2.dtype == np.float32
    inside = r2 <= np.float32(1.0)
    assert 0 < inside[at].sum() < at.sum()
    assert np.array_equal((np.abs(fa).max(axis=1) > 0.1)[at], inside[at])
    assert (fa[at & ~inside] == 0).all()
    # along the displacement: two roundings of 2^-28 of a cell at r >= 0.1 and three of FP32
    d64 = (xr[:n].astype(np.float64) - off) - xr[n:]
    on = (np.linalg.norm(fa, axis=1) > 0.05) & inside
    e = d64[on] / np.linalg.norm(d64[on], axis=1)[:, None]
    h = fa[on].astype(np.float64)
    h /= np.linalg.norm(h, axis=1)[:, None]
    assert on.sum() > 0.9 * inside.sum()
    assert (np.linalg.norm(h - e * np.sign((h * e).sum(axis=1))[:, None], axis=1)).max() <= 5e-7
