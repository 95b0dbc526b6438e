"""Force passes of particles that have no potential at all, by columns: the constant force and no energy."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntypes,n", [(1, 40), (2, 500)])
def test_free_particles(ntypes, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 4, size=(n, 3)).astype(np.float32).astype(np.float64)
    t = np.arange(n, dtype=np.int32) % ntypes
    u = W.build_gpu(dict(dim=[4.0] * 3, cells=[4] * 3, cutoff=1.0, dt=0.01, bc=("periodic",) * 3,
                         types=[(1.0, 0.1, m.Newtonian)] * ntypes, pots=[], forces=[(0, 1.0, -2.0, 0.5)], x=x,
                         v=np.zeros((n, 3), np.float32), t=t))
    u.force()
    want = np.where(t[:, None] == 0, np.float32([1.0, -2.0, 0.5]), np.float32(0))
    assert np.array_equal(u.forces, want)
    assert u.energies()[0] == 0.0
    u.steps(3)
    assert np.allclose(u.velocities, 0.03 * want, rtol=1e-6)
    u.close()
