"""Forms of potentials and engines that the column kernel takes, against the FP64 oracle on the engine's own cell
frame and task list: a DPD term summed with a table (either may come first), DPD shifted by the radii, scaled
tables, small units in which DPD's smallest distance is no small part of the cutoff, replicas by columns, and
replicas by cells and by columns in one engine."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W
from oracle import restatement as R

from golden_util import rel_rms

pytestmark = pytest.mark.gpu


def _table(p):
    i = p._info()
    return (dict(kind=i["kind"], flags=i["flags"], n=i["n"], alpha=i["alpha"][:3], a=i["a"], b=i["b"], r0p1=i["r0_plusone"]),
            p.coefficients if i["kind"] == 0 else np.zeros(8, dtype=np.float32))


def _apart(n, L, least, rng):
    """n random places in a cube of edge L, no two closer than least (minimum image)."""
    x = np.zeros((0, 3))
    while len(x) < n:
        y = rng.uniform(0, L, size=(n, 3))
        for k in range(n):
            d = y[k] - x
            d -= L * np.round(d / L)
            if len(x) < n and (len(x) == 0 or (d * d).sum(1).min() > least * least):
                x = np.vstack([x, y[k]])
    return np.minimum(x, L * (1 - 1e-6)).astype(np.float32).astype(np.float64)


def _morse():
    return m.Potential.morse(0.5, 5.0, 1.0, 1e-4, 3.0, 1e-3)


def _dpd(shifted=False, cutoff=1.0):
    return m.Potential.dpd(25.0, 4.5, 3.0, cutoff, shifted=shifted)


# name: (first and second potential by type pair, radius, unit of length, particles)
FORMS = {
    "table + DPD": ([((0, 0), _morse, _dpd)], 0.5, 1.0, 500),
    "DPD + table": ([((0, 0), _dpd, _morse)], 0.5, 1.0, 500),
    "table + DPD and DPD alone": ([((0, 0), _morse, _dpd), ((0, 1), _dpd, None), ((1, 1), _morse, None)], 0.5, 1.0, 500),
    "shifted DPD": ([((0, 0), lambda: _dpd(True, 0.5), None), ((0, 1), lambda: _dpd(True, 0.3), None)], 0.2, 1.0, 600),
    "scaled table": ([((0, 0), lambda: m.Potential.power(10.0, 1.0, 2.0, 0.05, 1.9, 1e-3), None)], 0.25, 1.0, 500),
    "DPD in small units": ([((0, 0), lambda: _dpd(False, 0.01), None)], 0.003, 0.01, 800),
}


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("name", list(FORMS))
def test_forms_match_the_oracle(name, variant):
    pots, radius, unit, n = FORMS[name]
    ntypes = 1 + max(j for (ij, p, q) in pots for j in ij)
    rng = np.random.default_rng(n + len(name))
    side = 5
    L = side * unit
    x = _apart(n, side, 0.05, rng) * unit
    v = rng.normal(0, unit, size=(n, 3)).astype(np.float32)
    t = (np.arange(n) % ntypes).astype(np.int32)
    m.init(dim=[L] * 3, cells=[side] * 3, cutoff=unit, dt=0.01, bc={k: "periodic" for k in "xyz"})
    types = [type(f"T{k}", (m.Particle,), {"mass": 1.0, "radius": radius}) for k in range(ntypes)]
    u, firsts, seconds = m.universe, [], []
    for (i, j), first, second in pots:
        p, q = first(), second() if second else None
        u.bind(p if q is None else p + q, types[i], types[j])
        firsts.append((p, i, j))
        if q is not None:
            seconds.append((q, i, j))
    u._add_particles(x, v, t)
    u.handle
    u.force_config(variant, 1 << 20)
    u.force()
    _, _, f, c, xr = u.state()
    ep, _ = u.energies()
    tasks = u.tasks()
    u.close()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]

    def entry(p, i, j):
        return ("dpd" if p._info()["kind"] == 1 else "table", (25.0, 4.5, 3.0), i, j)

    scn = dict(dim=[L] * 3, cutoff=unit, dt=0.01, t=t, types=[(1.0, radius, m.Newtonian)] * ntypes,
               pots=[entry(*p) for p in firsts])
    tables = {k: _table(p) for k, (p, i, j) in enumerate(firsts + seconds)}
    f64, ep64, counts = R.nonbond(scn, xr, v, c, tasks, np.array([side] * 3, dtype=np.int32), precision=64, tables=tables,
                                  second=[entry(*q) for q in seconds])[:3]
    assert rel_rms(f, f64) <= 1e-5
    assert abs(ep - ep64) <= 1e-6 * max(1.0, abs(ep64))


def _replicas(sizes, side, seed):
    """Morse fluids of one kind in boxes of side^3 cells of the cutoff."""
    specs = []
    for k, n in enumerate(sizes):
        rng = np.random.default_rng(seed + k)
        s = side[k]
        x = np.minimum(rng.uniform(0, s, size=(n, 3)), s * (1 - 1e-6)).astype(np.float32).astype(np.float64)
        specs.append(dict(dim=[float(s)] * 3, cells=[s] * 3, cutoff=1.0, dt=1e-4, bc=("periodic",) * 3,
                          types=[(1.0, 0.7, m.Newtonian)], pots=[("morse", (0.1 + 0.1 * k, 5.0, 0.6, 1e-4, 2.0, 1e-3), 0, 0)],
                          forces=[], x=x, v=np.zeros_like(x), t=np.zeros(n, dtype=np.int32)))
    return specs


def test_replicas_by_columns_have_their_own_bits():
    """With the variant pinned, replicas of sparse fluids in one engine give the bits they give alone."""
    specs = _replicas([300, 2000, 31], [5, 9, 3], 5)
    for variant in (1, 2, 3):
        u = W.build_gpu_batch(specs)
        u.handle
        u.force_config(variant, 1 << 20)
        u.steps(3)
        _, vb, fb, _, xb = [a.copy() for a in u.state()]
        u.close()
        off = 0
        for sc in specs:
            n = len(sc["t"])
            us = W.build_gpu(sc)
            us.handle
            us.force_config(variant, 1 << 20)
            us.steps(3)
            _, vs, fs, _, xs = us.state()
            for p, q in ((vb, vs), (fb, fs), (xb, xs)):
                assert np.array_equal(p[off:off + n].view(np.uint32), q.view(np.uint32))
            us.close()
            off += n


@pytest.mark.parametrize("sizes,side", [([1500, 300, 900], [4, 5, 4]), ([200, 64 * 14], [6, 4])])
def test_cells_and_columns_in_one_engine(sizes, side):
    """Replicas on either side of the density line (11 a cell): forces, energy, pair counts and virial of each against
    the oracle, and a second pass gives the same bits."""
    specs = _replicas(sizes, side, 9)
    u = W.build_gpu_batch(specs)
    u.force()
    _, v, f, c, xr = [a.copy() for a in u.state()]
    ep, _ = u.energies()
    u.force()
    assert np.array_equal(u.forces, f) and u.energies()[0] == ep
    off, coff, total = 0, 0, 0.0
    for sc, s in zip(specs, side):
        n, cd = len(sc["t"]), np.array([s] * 3, dtype=np.int32)
        us = W.build_gpu(sc)
        us.handle
        tasks = us.tasks()
        us.close()
        tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]
        f64, ep64 = R.nonbond(sc, xr[off:off + n], v[off:off + n], c[off:off + n] - coff, tasks, cd, precision=64)[:2]
        assert rel_rms(f[off:off + n], f64) <= 1e-5
        total += ep64
        off += n
        coff += s ** 3
    assert abs(ep - total) <= 1e-6 * abs(total)
    u.close()
