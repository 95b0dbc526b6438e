"""The column force kernel (cubic cells no smaller than the cutoff) against the FP64 oracle on the
engine's own cell frame and task list, where its work is cut: columns of 1 to a few groups of 32
particles, three cells along an axis (both periodic images of a neighbour in one column), long sparse
columns (the position unit grows), cells much larger than the cutoff and crowded ones (several
regions of staged particles), walls, particles on the cells' faces (pairs of cells the reference
skips), type pairs without a potential and particles closer than the table's start; with one, four
and eight warps per group."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W
from oracle import restatement as R

from golden_util import rel_rms

pytestmark = pytest.mark.gpu

MORSE = (0.5, 5.0, 1.0, 1e-4, 3.0, 1e-3)
DPD = (25.0, 4.5, 3.0, 1.0, 0)


def _scn(n, cells, h, kind, seed, walls=False, faces=False):
    rng = np.random.default_rng(seed)
    dim = [c * h for c in cells]
    x = rng.uniform(0, 1, size=(n, 3)) * dim
    if faces:  # a tenth of the particles within a key quantum of a cell face, on either side
        k = rng.permutation(n)[: n // 10]
        ax = rng.integers(0, 3, size=len(k))
        near = np.round(x[k, ax] / h) * h + rng.uniform(-1e-4, 1e-4, size=len(k)) * h
        x[k, ax] = np.mod(near, np.asarray(dim)[ax])
    x = np.minimum(x, np.asarray(dim) * (1 - 1e-6)).astype(np.float32).astype(np.float64)
    v = rng.normal(0, 1, size=(n, 3)).astype(np.float32).astype(np.float64)
    pots = [("dpd", DPD, 0, 0), ("dpd", (10.0, 2.0, 1.0, 0.7, 0), 0, 1)] if kind == "dpd" else [("morse", MORSE, 0, 0), ("morse", MORSE, 0, 1)]
    t = (np.arange(n) % 2).astype(np.int32)  # no potential between particles of type 1
    if kind == "one":
        pots, t = [("morse", MORSE, 0, 0)], np.zeros(n, dtype=np.int32)
    types = [(1.0, 0.5, m.Newtonian)] * (1 if kind == "one" else 2)
    bc = ("periodic", "free_slip", "free_slip") if walls else ("periodic",) * 3
    return dict(dim=dim, cells=list(cells), cutoff=1.0, dt=0.01, bc=bc, types=types, pots=pots, forces=[(0, 0.5, -0.25, 2.0)], x=x,
                v=v, t=t)


CASES = [
    (1, (3, 3, 3), 1.0, "morse", {}), (63, (3, 3, 3), 1.0, "one", {}), (300, (3, 4, 3), 1.25, "dpd", {}),
    (291, (3, 3, 8), 1.0, "one", dict(faces=True)), (2000, (5, 4, 7), 1.0, "dpd", dict(faces=True)),
    (1500, (3, 4, 5), 2.5, "morse", {}), (4000, (3, 3, 3), 1.5, "dpd", {}), (700, (3, 5, 100), 1.0, "morse", {}),
    (900, (1, 2, 40), 1.0, "one", dict(walls=True)), (1777, (4, 6, 1), 1.5, "morse", dict(walls=True, faces=True)),
    (3000, (6, 6, 6), 1.0625, "morse", dict(faces=True)),
]


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{'x'.join(map(str, c[1]))}-{c[2]}-{c[3]}")
def test_columns_match_the_oracle(case, variant):
    n, cells, h, kind, opts = case
    if opts.get("walls") and cells[0] < 3:
        opts = dict(opts)
    scn = _scn(n, cells, h, kind, seed=n, **opts)
    if cells[0] < 3:
        scn["bc"] = ("free_slip",) * 3
    u = W.build_gpu(scn)
    u.force_config(variant, 1 << 20)
    u.force()
    x, v, f, c, xr = u.state()
    tasks = u.tasks()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]
    f64, ep64, counts = R.nonbond(scn, xr, v, c, tasks, np.asarray(u.cell_grid()[0], dtype=np.int32), precision=64)[:3]
    # the project's force bar; a pair at the cutoff may fall on either side of it in the last bit, where
    # the Morse force is below 1e-2 of the typical one
    assert rel_rms(f, f64) <= 1e-5 if n > 1 else np.abs(f - f64).max() <= 1e-6
    ep, _ = u.energies()
    assert abs(ep - ep64) <= 1e-6 * max(1.0, abs(ep64))
    u.close()


def test_columns_keep_the_pair_counts_and_the_virial():
    """The statistics and the virial take the cell kernel over the same cells, each pair once."""
    from mechanica_b200._native import check, lib
    import ctypes
    scn = _scn(1777, (5, 5, 5), 1.0, "one", seed=5)
    u = W.build_gpu(scn)
    u.force()
    x, v, f, c, xr = u.state()
    tasks = u.tasks()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]
    out = R.nonbond(scn, xr, v, c, tasks, np.array([5, 5, 5], dtype=np.int32), precision=64, virial=True)
    assert np.linalg.norm(u.virial() - out[3]) <= 1e-5 * np.linalg.norm(out[3])
    cand, inter = ctypes.c_longlong(), ctypes.c_longlong()
    check(lib().mxg_engine_pair_counts(u.handle, ctypes.byref(cand), ctypes.byref(inter)), "pair_counts")
    L = np.asarray(scn["dim"])
    d = scn["x"][:, None] - scn["x"][None]
    d -= L * np.round(d / L)
    r2 = (d ** 2).sum(2)[np.triu_indices(len(scn["x"]), 1)]
    assert inter.value == int((r2 <= 1.0).sum())
    u.close()


@pytest.mark.parametrize("variant", [1, 2, 3])
def test_columns_turn_close_pairs(variant):
    """Isolated pairs closer than the Lennard-Jones table's start get a random direction of that
    length: opposite forces of the table's size there, and its energy once per pair."""
    lo = 0.275
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.0 + 1.0
    x = np.concatenate([g, g + [0.1, 0.05, -0.07]])
    scn = dict(dim=[8.0] * 3, cells=[8] * 3, cutoff=1.0, dt=0.01, bc=("periodic",) * 3, types=[(39.4, 0.1, m.Newtonian)],
               pots=[("lj126", (lo, 1.0, 9.5075e-6, 6.1545e-3, 1e-3), 0, 0)], forces=[], x=x, v=np.zeros_like(x),
               t=np.zeros(len(x), dtype=np.int32))
    u = W.build_gpu(scn)
    u.force_config(variant, 1 << 20)
    u.force()
    f = np.asarray(u.forces, dtype=np.float64)
    e, dv = W.make_potential(*scn["pots"][0][:2])(np.float32(lo))
    size = np.linalg.norm(f, axis=1)
    assert np.allclose(size, abs(dv), rtol=1e-5)
    assert np.abs(f[:64] + f[64:]).max() <= 1e-6 * abs(dv)
    assert np.linalg.norm((f[:64] / size[:64, None]).mean(axis=0)) < 0.5  # not one direction
    assert abs(u.energies()[0] - 64 * e) <= 1e-5 * abs(64 * e)
    u.close()
