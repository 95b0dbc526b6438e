"""Pairs of a column pass whose result hangs on the last bits of the positions: particles closer than
1/64 of the cutoff (the direction of their force) and pairs at the cutoff of a flux with decay (the
decay does not vanish there). They are compared with the displacement rounded as the reference rounds
it, in numpy."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu

CELLS = 8
A = float(np.sqrt(np.finfo(np.float32).eps))  # a of DPD: closer pairs get a random direction of that length


def _reference_d(xa, xb, cell_a, cell_b):
    """d = (x_first - s) - x_second from cell-relative FP32 positions, a's point of view."""
    off = cell_b - cell_a
    if tuple(off) >= (0, 0, 0):
        return (xa - off.astype(np.float32)) - xb
    return -((xb + off.astype(np.float32)) - xa)


@pytest.mark.parametrize("gap", [2e-5, 3e-4, 5e-3, 0.0149])
def test_close_pairs_take_the_reference_displacement(gap):
    """Pairs a gap apart across a face of their cells, alone in the box; DPD with only the conservative
    term: f = alpha (1 - r) d / r. FP32 evaluation of that: a few units in the last place of the
    force, 25 x 1e-6."""
    rng = np.random.default_rng(int(gap * 1e7))
    n = 60
    cell = rng.integers(0, CELLS - 1, size=(n, 3))
    cell = np.unique(2 * (cell // 2), axis=0)  # one pair to a block of 2^3 cells
    n = len(cell)
    axis = rng.integers(0, 3, size=n)
    base = rng.uniform(0.3, 0.7, size=(n, 3))
    step = rng.normal(size=(n, 3))
    step *= gap / np.linalg.norm(step, axis=1)[:, None]
    step[np.arange(n), axis] = np.abs(step[np.arange(n), axis])
    base[np.arange(n), axis] = 1.0 - 0.5 * step[np.arange(n), axis]
    xa, xb = cell + base, cell + base + step
    x = np.concatenate([xa, xb])
    scn = dict(dim=[float(CELLS)] * 3, cells=[CELLS] * 3, cutoff=1.0, dt=0.01, bc=("periodic",) * 3,
               types=[(1.0, 0.1, m.Newtonian)], pots=[("dpd", (25.0, 0.0, 0.0, 1.0), 0, 0)], forces=[],
               x=x, v=np.zeros((2 * n, 3), np.float32), t=np.zeros(2 * n, dtype=np.int32))
    u = W.build_gpu(scn)
    u.force()
    _, _, f, c, xr = u.state()
    loc = np.stack([c // CELLS ** 2, c // CELLS % CELLS, c % CELLS], -1)
    for k in range(n):
        d = _reference_d(xr[k].astype(np.float32), xr[n + k].astype(np.float32), loc[k], loc[n + k]).astype(np.float64)
        r = np.sqrt((d * d).sum())
        if r < A:
            assert abs(np.linalg.norm(f[k].astype(np.float64)) - 25.0 * (1.0 - A)) <= 25e-6
        else:
            assert np.abs(f[k] - 25.0 * (1.0 - r) * d / r).max() <= 25e-6
        assert np.array_equal(f[k], -f[n + k])


def test_flux_decay_at_the_cutoff_follows_the_reference():
    """Pairs whose distance is within a few units in the last place of the cutoff: the decay of a flux acts
    in full or not at all, by the reference's r^2 against its cutoff squared (FP32). rate = -decay/2 * s
    where the pair counts (the weight is below 1e-12 there)."""
    rng = np.random.default_rng(7)
    cell = np.stack(np.meshgrid(*[np.arange(0, 12, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(cell)
    side = 12
    base = rng.uniform(0.1, 0.9, size=(n, 3))
    step = rng.normal(size=(n, 3))
    step = np.abs(step) / np.linalg.norm(step, axis=1)[:, None]
    x = np.concatenate([cell + base, cell + base + step * (1 + rng.integers(-3, 4, size=(n, 1)) * 6e-8)])
    vals = np.ones((2 * n, 1), dtype=np.float32)
    scn = dict(dim=[float(side)] * 3, cells=[side] * 3, cutoff=1.0, dt=0.01, bc=("periodic",) * 3,
               types=[(1.0, 0.1, m.Newtonian)], pots=[("morse", (0.2, 5.0, 0.6, 1e-4, 2.0, 1e-3), 0, 0)], forces=[],
               x=x, v=np.zeros((2 * n, 3), np.float32), t=np.zeros(2 * n, dtype=np.int32),
               sp_nspec=np.array([1], dtype=np.int32), sp_names=[["S1"]], sp_flags=np.array([[0]], dtype=np.uint32),
               sp_values=vals, fluxes=[(0, 0, 0, 0, 0, 1.0, 0.5, 0.0)])
    u = W.build_gpu(scn)
    _, _, _, c, xr = u.state()
    loc = np.stack([c // side ** 2, c // side % side, c % side], -1)
    u.steps(1)
    got = np.asarray(u.species_values(), dtype=np.float64).reshape(2 * n, -1)[:, 0]
    hits = 0
    for k in range(n):
        d = _reference_d(xr[k].astype(np.float32), xr[n + k].astype(np.float32), loc[k], loc[n + k])
        r2 = np.float32(np.float32(d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
        inside = r2 <= np.float32(1.0)
        hits += inside
        want = 1.0 - (0.01 * 0.25 if inside else 0.0)
        assert abs(got[k] - want) <= 1e-6 and abs(got[n + k] - want) <= 1e-6
    assert 0 < hits < n
