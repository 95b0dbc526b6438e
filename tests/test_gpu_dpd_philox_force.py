"""Forces of DPD with the Philox random term, where every pair potential is DPD, against the FP64
restatement of the model on the same stream (keyed on the step and the particle ids).

Tolerance: a pair's force is a handful of FP32 operations on FP32 cell-relative positions, each
within a unit or two in the last place (6e-8), and some 45 of them sum to a result of the size of
one: relative RMS within 1e-5, the bar of every force comparison."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W
from oracle import adjoint_ref as R

from golden_util import rel_rms

pytestmark = pytest.mark.gpu

DT = 0.01
A = (25.0, 4.5, 3.0, 1.0)
B = (40.0, 9.0, 2.0, 0.8)


@pytest.mark.parametrize("n, cells, types, pots", [
    (1500, (5, 5, 5), 1, {(0, 0): A}),                              # 12 in a cell
    (700, (9, 4, 6), 1, {(0, 0): A}),                               # 3 in a cell
    (1100, (3, 4, 7), 2, {(0, 0): A, (0, 1): B}),                   # a pair of types without a potential
    (911, (4, 4, 4), 2, {(0, 0): A, (0, 1): B, (1, 1): B}),
])
def test_philox_forces_match_fp64(n, cells, types, pots):
    rng = np.random.default_rng(n)
    box = np.array(cells, dtype=np.float64)
    x = (rng.uniform(0, 1, size=(n, 3)) * box * (1 - 1e-6)).astype(np.float32).astype(np.float64)
    v = rng.normal(0, 1.0, size=(n, 3)).astype(np.float32)
    t = (np.arange(n) % types).astype(np.int32)
    scn = dict(dim=list(box), cells=list(cells), cutoff=1.0, dt=DT, bc=("periodic",) * 3,
               types=[(1.0, 0.5, m.Newtonian)] * types, pots=[("dpd", p, a, b) for (a, b), p in pots.items()],
               forces=[], x=x, v=v, t=t)
    u = W.build_gpu(scn, rng_mode="philox")
    u.force()
    delta = float(np.float32(1.0 / np.sqrt(DT)))
    terms = {k: [R.Dpd(*p, delta)] for k, p in pots.items()}
    ref = R.forces(x, v.astype(np.float64), t, np.arange(n), box, np.full(types, 0.5), terms, 1.0, 0)
    assert rel_rms(u.state()[2], ref) <= 1e-5
