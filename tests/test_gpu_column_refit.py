"""A table moved by a re-fit so that it ends inside the cutoff, where none did at the start: pairs within a few units in
the last place of its new end act in full or not at all by the reference's FP32 arithmetic, in a force pass
and in captured steps; and a table that ends closer than 1/64 of the cutoff."""
import numpy as np
import pytest

import mechanica_b200 as m
from oracle import restatement as R

pytestmark = pytest.mark.gpu

SIDE = 12


@pytest.mark.parametrize("r0,captured", [(1.5, False), (1.5, True), (2.2, False), (2.39, False)])
def test_end_of_a_refitted_table(r0, captured):
    """Radius 0.7, s = r - 1.4 + r0 + 1 up to 2: the end is at 2.4 - r0."""
    rng = np.random.default_rng(int(100 * r0))
    cell = np.stack(np.meshgrid(*[np.arange(0, SIDE, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = len(cell)
    u3 = np.abs(rng.normal(size=(n, 3)))
    u3 /= np.linalg.norm(u3, axis=1)[:, None]
    end = float(np.float32(2.0)) - float(np.float32(r0 + 1)) + float(np.float32(0.7)) * 2
    xa = cell + np.where(rng.uniform(size=(n, 1)) < 0.5, rng.uniform(0.05, 0.95, size=(n, 3)), 1 - 0.5 * u3 * end)
    xb = xa + u3 * (end + rng.integers(-4, 5, size=(n, 1)) * 6e-8)
    x = np.mod(np.concatenate([xa, xb]) - 1.0, SIDE)
    m.init(dim=[float(SIDE)] * 3, cells=[SIDE] * 3, cutoff=1.0, dt=1e-6, bc={k: "periodic" for k in "xyz"})
    T = type("T", (m.Particle,), {"mass": 1.0, "radius": 0.7})
    u, p = m.universe, m.Potential.morse(0.2, 5.0, 0.6, 1e-4, 2.0, 1e-3)
    u.bind(p, T, T)
    u._add_particles(x, np.zeros((2 * n, 3), np.float32), np.zeros(2 * n, dtype=np.int32))
    u.handle
    if captured:
        u.steps(1)  # r is far from the start's well: the particles hardly move in a microsecond
    u.set_potential_params(p, [0.2, 5.0, r0, 1e-4, 2.0, 1e-3])
    _, v, _, c, xr = [a.copy() for a in u.state()]
    if captured:
        u.steps(1)
    else:
        u.force()
    f = u.forces
    tasks = u.tasks()
    u.close()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]
    i = p._info()
    tables = {0: (dict(kind=0, flags=i["flags"], n=i["n"], alpha=i["alpha"][:3], a=i["a"], b=i["b"], r0p1=i["r0_plusone"]),
                  p.coefficients)}
    assert tables[0][0]["r0p1"] == np.float32(r0 + 1)
    f64 = R.nonbond(dict(dim=[float(SIDE)] * 3, cutoff=1.0, dt=1e-6, t=np.zeros(2 * n, np.int32), types=[(1.0, 0.7, m.Newtonian)],
                         pots=[("table", (), 0, 0)]), xr, v, c, tasks, np.array([SIDE] * 3, dtype=np.int32), precision=64,
                    tables=tables)[0]
    on = np.abs(f64[:n]).max(axis=1) > 0
    assert 0 < on.sum() < n
    assert np.array_equal(np.abs(f[:n]).max(axis=1) > 0, on)
    big = np.abs(f64).max()
    # the displacement's direction: two units in the last place of a cell against the distance
    assert np.abs(f - f64).max() <= (1e-5 + 2.4e-7 / end) * big
    assert np.array_equal(f[:n], -f[n:])
