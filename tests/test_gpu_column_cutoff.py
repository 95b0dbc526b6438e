"""Decisions of a column pass that hang on the last bits of the positions, by the reference's FP32 arithmetic (the
oracle decides with it): isolated pairs within a few units in the last place of the cutoff where the force does
not vanish, of a table's own end inside the cutoff (shifted, scaled, summed with a DPD term), of a table's start
and of a summed second table's start; across faces of the cells and of the periodic box. Each force is the pair's
in full or not there at all."""
import numpy as np
import pytest

import mechanica_b200 as m
from oracle import restatement as R

pytestmark = pytest.mark.gpu

SIDE = 12


def _morse(lo=1e-4, hi=2.0):  # at radius 0.7: s = r + 0.2, the well at r = 0.8, a force of 0.465 at r = 1
    return m.Potential.morse(0.2, 5.0, 0.6, lo, hi, 1e-3)


def _dpd(cutoff=1.0):  # no random term: the two engines draw differently
    return m.Potential.dpd(25.0, 4.5, 0.0, cutoff)


def _mixed(first, second):
    """A table between particles of one type, DPD between the two."""
    return lambda: ([(first(), None, 0, 0), (second(), None, 0, 1), (first(), None, 1, 1)], 2)


def _one(first, second=None):
    return lambda: ([(first(), second() if second else None, 0, 0)], 1)


# name: (potentials, radius, the distance that decides)
CASES = {
    "cutoff": (_one(_morse), 0.7, lambda p: 1.0),
    "cutoff, with a DPD term": (_one(_morse, _dpd), 0.7, lambda p: 1.0),
    "cutoff, two types": (_mixed(_morse, lambda: _dpd(1.5)), 0.7, lambda p: 1.0),
    "cutoff, DPD that reaches further": (_one(lambda: _dpd(1.5)), 0.7, lambda p: 1.0),
    "end of a shifted table": (_one(lambda: _morse(hi=1.15)), 0.7, lambda p: p.max - p._info()["r0_plusone"] + 1.4),
    "end, with a DPD term": (_one(lambda: _morse(hi=1.15), _dpd), 0.7, lambda p: p.max - p._info()["r0_plusone"] + 1.4),
    "end of a short shifted table": (_one(lambda: _morse(hi=0.6)), 0.7, lambda p: p.max - p._info()["r0_plusone"] + 1.4),
    "end of a scaled table": (_one(lambda: m.Potential.power(10.0, 1.0, 2.0, 0.05, 1.8, 1e-3)), 0.25, lambda p: p.max * 0.5),
    "start of a table": (_one(lambda: _morse(lo=0.1)), 0.7, lambda p: p.min),
    "start, with a DPD term": (_one(lambda: _morse(lo=0.3), _dpd), 0.7, lambda p: p.min),
    "start of a second table": (_one(_dpd, lambda: _morse(lo=0.3)), 0.7, None),
}


@pytest.mark.parametrize("variant", [1, 3])
@pytest.mark.parametrize("name", list(CASES))
def test_decisions_follow_the_reference(name, variant):
    make, radius, where = CASES[name]
    pots, ntypes = make()
    r0 = pots[0][1].min if where is None else where(pots[0][0])
    rng = np.random.default_rng(len(name))
    cell = np.stack(np.meshgrid(*[np.arange(0, SIDE, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(cell)
    u3 = np.abs(rng.normal(size=(n, 3)))
    u3 /= np.linalg.norm(u3, axis=1)[:, None]
    base = np.where(rng.uniform(size=(n, 1)) < 0.5, rng.uniform(0.05, 0.95, size=(n, 3)), 1 - 0.5 * u3 * r0)
    xa = cell + base
    xb = xa + u3 * (r0 + rng.integers(-3, 4, size=(n, 1)) * 6e-8)
    x = np.mod(np.concatenate([xa, xb]) - 1.0, SIDE)  # some pairs across the periodic faces
    t = np.zeros(2 * n, dtype=np.int32)
    if ntypes == 2:
        t[n:] = rng.integers(0, 2, size=n)
        t[:n] = rng.integers(0, 2, size=n)
    v = rng.normal(0, 1, size=(2 * n, 3)).astype(np.float32)
    m.init(dim=[float(SIDE)] * 3, cells=[SIDE] * 3, cutoff=1.0, dt=0.01, bc={k: "periodic" for k in "xyz"})
    types = [type(f"T{k}", (m.Particle,), {"mass": 1.0, "radius": radius}) for k in range(ntypes)]
    u = m.universe
    for (p, q, i, j) in pots:
        u.bind(p if q is None else p + q, types[i], types[j])
    u._add_particles(x, v, t)
    u.handle
    u.force_config(variant, 1 << 20)
    u.force()
    _, _, f, c, xr = u.state()
    tasks = u.tasks()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]

    def entry(p, i, j):
        kind = "dpd" if p._info()["kind"] == 1 else "table"
        return (kind, (25.0, 4.5, 0.0, 0.0), i, j)

    firsts = [p for (p, q, i, j) in pots]
    seconds = [q for (p, q, i, j) in pots if q is not None]
    scn = dict(dim=[float(SIDE)] * 3, cutoff=1.0, dt=0.01, t=t, types=[(1.0, radius, m.Newtonian)] * ntypes,
               pots=[entry(p, i, j) for (p, q, i, j) in pots])
    tables = {}
    for k, p in enumerate(firsts + seconds):
        i = p._info()
        tables[k] = (dict(kind=i["kind"], flags=i["flags"], n=i["n"], alpha=i["alpha"][:3], a=i["a"], b=i["b"],
                          r0p1=i["r0_plusone"]), p.coefficients if i["kind"] == 0 else np.zeros(8, dtype=np.float32))
    f64 = R.nonbond(scn, xr, v, c, tasks, np.array([SIDE] * 3, dtype=np.int32), precision=64, tables=tables,
                    second=[entry(q, i, j) for (p, q, i, j) in pots if q is not None])[0]
    u.close()
    assert np.array_equal(f[:n], -f[n:])
    big = np.abs(f64).max()
    on = np.abs(f64[:n]).max(axis=1)
    if "start" in name and "second" not in name:
        # a pair closer than the start gets a random direction, and none from the oracle's table; with a DPD term
        # that one alone is there
        d = (xr[:n].astype(np.float64) + np.stack([c[:n] // 144, c[:n] // 12 % 12, c[:n] % 12], -1)) - (
            xr[n:].astype(np.float64) + np.stack([c[n:] // 144, c[n:] // 12 % 12, c[n:] % 12], -1))
        d -= SIDE * np.round(d / SIDE)
        h = np.linalg.norm(np.cross(f[:n], d), axis=1) / (np.linalg.norm(f[:n], axis=1) * np.linalg.norm(d, axis=1))
        direct = on > 0.5 * big / np.sqrt(3)
        assert 0 < direct.sum() < n
        assert h[direct].max() <= 1e-5 < h[~direct].min()
        assert np.abs(f[:n] - f64[:n])[direct].max() <= 1e-5 * big
        return
    decided = on[on > 0]
    if "DPD term" not in name and "two types" not in name and "second" not in name:
        assert 0 < len(decided) < n
    assert np.abs(f - f64).max() <= 1e-5 * big
