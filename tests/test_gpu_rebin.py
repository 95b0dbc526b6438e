"""The re-binning: every cell's particles in one run of slots in ascending id, whatever moved.

Free flight, so the state after k steps is known: velocities unchanged, positions x + k dt v in the
periodic box (FP32 cell-relative sums, a rounding of at most 2^-24 of an edge near one per step and
one on loading: 1e-6 at four steps). The sizes put a block of the re-binning on a part of a cell, one
cell, several, and its most, with more slots than it keeps on chip, buckets that overflow and a last
block with fewer cells. Key bounds: a restored checkpoint computes them anew from its slots, and the
same force pass must come out bit for bit."""
import numpy as np
import pytest
import torch

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu

DT = 0.01


def _scn(n, cells, h, pots, seed, empty=0.0):
    rng = np.random.default_rng(seed)
    box = np.array(cells) * np.array(h)
    x = rng.uniform(0, 1, size=(n, 3)) * [1 - empty, 1, 1] * box * (1 - 1e-6)
    v = np.clip(rng.normal(0, 1.2, size=(n, 3)), -4, 4).astype(np.float32)
    return dict(dim=list(box), cells=list(cells), cutoff=1.0, dt=DT, bc=("periodic",) * 3,
                types=[(1.0, 0.1, m.Newtonian)], pots=pots, forces=[],
                x=x.astype(np.float32).astype(np.float64), v=v, t=np.zeros(n, dtype=np.int32))


@pytest.mark.parametrize("n, cells, empty", [
    (1, (3, 3, 3), 0.0),
    (4000, (3, 3, 3), 0.0),         # 148 in a cell, a block each
    (45000, (3, 3, 3), 0.0),        # 1667 in a cell: beyond the slots kept on chip, buckets overflow
    (3001, (13, 7, 11), 0.6),       # three in a cell, most cells empty
    (9000, (11, 9, 10), 0.0),
    (60000, (18, 17, 16), 0.0),
    (150000, (34, 34, 34), 0.0),    # blocks of 128 threads, 39304 cells
])
def test_slots_follow_the_particles(n, cells, empty):
    scn = _scn(n, cells, (1.0,) * 3, [], n, empty)
    u = W.build_gpu(scn)
    for k in range(1, 5):
        u.steps(1)
        st = u.device_state()
        ids = st["vel"].view(torch.int32)[:, 3].cpu().numpy()
        cell = st["cell"].cpu().numpy()
        assert np.array_equal(np.lexsort((ids, cell)), np.arange(n))
        assert np.array_equal(np.sort(ids), np.arange(n))
        vel, pos = st["vel"].cpu().numpy()[:, :3], st["pos"].cpu().numpy()[:, :3]
        assert np.array_equal(vel, scn["v"][ids])
        c = np.array(cells)
        loc = np.stack([cell // (c[1] * c[2]), cell // c[2] % c[1], cell % c[2]], -1)
        assert (pos >= 0).all() and (pos <= 1).all()
        d = pos.astype(np.float64) + loc - (scn["x"][ids] + k * DT * vel.astype(np.float64))
        assert np.abs(d - c * np.rint(d / c)).max() <= 1e-6
        x, v, f, cid, xr = u.state()                       # through the slot of each id
        assert np.array_equal(cid[ids], cell) and np.array_equal(v[ids], vel)


@pytest.mark.parametrize("n, cells, h", [
    (9000, (8, 8, 10), (1.0, 1.2, 1.4)), (20000, (4, 5, 6), (1.0, 1.3, 1.6)), (700, (9, 8, 3), (1.5, 1.0, 1.1)),
    (1500, (5, 5, 5), (1.0, 1.0, 1.0)),
])
def test_key_bounds_are_those_of_the_slots(n, cells, h):
    u = W.build_gpu(_scn(n, cells, h, [("dpd", (25.0, 4.5, 3.0, 1.0), 0, 0)], n + 1))
    u.steps(3)
    u.force()
    f = u.state()[2].view(np.uint32).copy()
    u.restore(u.checkpoint())
    u.force()
    assert np.array_equal(u.state()[2].view(np.uint32), f)
