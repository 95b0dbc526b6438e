"""Values that are not finite: a species value reaches the partner of a flux in both directions, a particle whose
position is lost no longer acts on its neighbours, and the key bounds of its cell are the same after a step as
after a restore."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W
from mechanica_b200._native import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_fluxes_pass_on_what_is_not_finite(kind, value):
    """Fick, secretion and uptake of one species between two types: the column kernel against the formula, 0 or 1
    times the driving force, in numpy."""
    x = np.array([[1.2, 1.5, 1.5], [1.7, 1.5, 1.5]])
    k, target, dt = 2.0, 0.5, 0.01
    for ill in (0, 1):
        s = np.array([0.3, 0.4], dtype=np.float32)
        s[ill] = value
        u = W.build_gpu(dict(dim=[4.0] * 3, cells=[4] * 3, cutoff=1.0, dt=dt, bc=("periodic",) * 3,
                             types=[(1.0, 0.1, m.Newtonian)] * 2, pots=[], forces=[], x=x, v=np.zeros((2, 3), np.float32),
                             t=np.array([0, 1], dtype=np.int32), sp_nspec=np.array([1, 1], dtype=np.int32),
                             sp_names=[["S1"], ["S1"]], sp_flags=np.zeros((2, 1), dtype=np.uint32),
                             sp_values=s.reshape(2, 1), fluxes=[(kind, 0, 1, 0, 0, k, 0.0, target)]))
        u.steps(1)
        got = np.asarray(u.species_values()).ravel()
        u.close()
        with np.errstate(invalid="ignore"):
            a, b = s.astype(np.float64)
            drive = k * (a - b) if kind == 0 else k * (a - target) if kind == 1 else k * (target - b) * a
            g = drive if kind == 0 else float(drive > 0) * drive
            want = np.array([a - dt * (0.25 * g + 0.0 * a), b + dt * (0.25 * g - 0.0 * b)])  # no decay: 0 times the value
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        fine = np.isfinite(want)
        assert np.abs(got[fine] - want[fine]).max(initial=0.0) <= 1e-6


def _lost(n, rng, potential):
    """A fluid in which the particles of type 1 lose their positions in the first step."""
    x = rng.uniform(0, 4, size=(n, 3)).astype(np.float32).astype(np.float64)
    t = np.zeros(n, dtype=np.int32)
    t[::40] = 1
    return W.build_gpu(dict(dim=[4.0] * 3, cells=[4] * 3, cutoff=1.0, dt=1e-4, bc=("periodic",) * 3,
                            types=[(1.0, 0.1, m.Newtonian)] * 2, pots=[(*potential, 0, 0), (*potential, 0, 1)],
                            forces=[(1, float("nan"), 0.0, 0.0)], x=x, v=np.zeros((n, 3), np.float32), t=t)), t


POTENTIALS = [("dpd", (25.0, 4.5, 3.0, 1.0, 0)), ("morse", (0.5, 5.0, 1.0, 1e-4, 3.0, 1e-3))]


@pytest.mark.parametrize("potential", POTENTIALS, ids=lambda p: p[0])
@pytest.mark.parametrize("variant", [1, 3])
def test_a_lost_particle_acts_on_nobody(potential, variant):
    """One particle alone with a lost one beside it: after the step that loses it, it moves freely."""
    x = np.array([[1.3, 1.4, 1.5], [1.6, 1.6, 1.6]])
    u = W.build_gpu(dict(dim=[4.0] * 3, cells=[4] * 3, cutoff=1.0, dt=1e-4, bc=("periodic",) * 3,
                         types=[(1.0, 0.1, m.Newtonian)] * 2, pots=[(*potential, 0, 1)],
                         forces=[(1, float("nan"), 0.0, 0.0)], x=x, v=np.zeros((2, 3), np.float32),
                         t=np.array([0, 1], dtype=np.int32)))
    u.force_config(variant, 1 << 20)
    with pytest.raises(m.EngineError):
        u.steps(1)
    v1 = u.velocities[0].copy()
    assert np.isfinite(v1).all() and np.abs(v1).max() > 0 and not np.isfinite(u.positions[1]).all()
    with pytest.raises(m.EngineError):
        u.steps(5)
    assert np.array_equal(u.velocities[0], v1)
    u.close()


@pytest.mark.parametrize("potential", POTENTIALS, ids=lambda p: p[0])
def test_restore_after_a_loss(potential):
    u, t = _lost(1200, np.random.default_rng(3), potential)
    with pytest.raises(m.EngineError):
        u.steps(2)
    check(lib().mxg_engine_clear_status(u.handle), "clear_status")
    ck = u.checkpoint()
    with pytest.raises(m.EngineError):
        u.steps(2)
    a = [k.copy() for k in u.state()]
    check(lib().mxg_engine_clear_status(u.handle), "clear_status")
    u.restore(ck)
    with pytest.raises(m.EngineError):
        u.steps(2)
    for p, q in zip(a, u.state()):
        assert np.array_equal(p, q, equal_nan=True)
    assert np.isfinite(a[1][t == 0]).all()
    u.close()
