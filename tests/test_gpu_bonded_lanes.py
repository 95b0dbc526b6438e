"""The bonded pass evaluates a particle's terms over several lanes up to a size and in one lane
above it; the sums are formed in the same order, so both give the same bits. The large system is
the small one and enough far-away free particles to pass the size (37,888 on 148 SMs)."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _build(free, degree, seed=3):
    """A cluster of 60 particles in one cell's neighbourhood, each bonded to up to `degree` others,
    angles over neighbours, every third bond's pair excluded; `free` particles elsewhere."""
    rng = np.random.default_rng(seed)
    n = 60
    L = 60.0
    x = np.concatenate([rng.uniform(2, 4, (n, 3)), rng.uniform(10, L - 1, (free, 3))]).astype(np.float32).astype(np.float64)
    t = np.concatenate([np.zeros(n), np.ones(free)]).astype(np.int32)
    bi, bj = [], []
    for i in range(n):
        for k in range(1, degree + 1):
            if i + k < n:
                bi.append(i)
                bj.append(i + k)
    ai = np.arange(0, n - 2)
    scn = dict(dim=[L] * 3, cells=[20] * 3, cutoff=3.0, dt=0.001, bc=("periodic",) * 3,
               types=[(1.0, 0.1, m.Newtonian), (1.0, 0.1, m.Newtonian)],
               pots=[("morse", (0.5, 3.0, 0.5, 1e-4, 2.5, 1e-3), 0, 0)], forces=[], x=x, v=np.zeros((n + free, 3), np.float32), t=t,
               bi=np.array(bi), bj=np.array(bj), bond_pot=("harmonic", (10.0, 1.0, 0.01, 5.0, 0.01)),
               dissociation=float(np.finfo(np.float64).max),
               ai=ai, aj=ai + 1, ak=ai + 2, angle_pot=("harmonic_angle", (5.0, 2.0, 0.0, np.pi, 0.005 * np.pi)),
               ex_i=np.array(bi[::3]), ex_j=np.array(bj[::3]))
    return W.build_gpu(scn)


@pytest.mark.parametrize("degree", [1, 2, 3, 5, 9])
def test_lanes_give_the_bits_of_one(degree):
    out = []
    for free in (5, 39000):
        u = _build(free, degree)
        u.steps(2)
        u.force()
        x, v, f, c, xr = u.state()
        out.append([a[:60].view(np.uint32 if a.dtype.itemsize == 4 else np.uint64).copy() for a in (x, v, f, xr)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
