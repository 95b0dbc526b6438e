"""The oracle's tables where the reference's builder is not at hand: the golden tables pass the check against the
closed forms, and tables with a fault do not."""
import os

import numpy as np
import pytest

from mechanica_b200 import workloads as W
from oracle import refengine
from oracle import restatement as R

GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "tables.npz"))
NAMES = sorted({k.split("__")[0] for k in GOLD.files})


def _golden(name):
    n, flags = (int(q) for q in GOLD[f"{name}__info"])
    a, b, r0 = GOLD[f"{name}__ab"]
    return (str(GOLD[f"{name}__kind"]), tuple(GOLD[f"{name}__params"]),
            dict(kind=0, flags=flags, n=n, alpha=GOLD[f"{name}__alpha"][:3], a=a, b=b, r0p1=r0),
            np.array(GOLD[f"{name}__coef"], dtype=np.float32))


@pytest.mark.parametrize("name", NAMES)
def test_golden_tables_are_their_potentials(name):
    R.check_table(*_golden(name))


@pytest.mark.parametrize("name", NAMES)
def test_faults_are_seen(name):
    kind, params, info, coef = _golden(name)
    c = coef.reshape(-1, 8).copy()
    k = len(c) // 2
    size = max(1.0, np.abs(c[k, 2:]).sum())
    c[k, 7] += 20 * params[-1] * size  # one interval's values
    with pytest.raises(RuntimeError):
        R.check_table(kind, params, info, c.ravel())
    for key, value in (("alpha", 0 * np.asarray(info["alpha"])), ("b", info["b"] * 1.01), ("n", info["n"] - 1)):
        with pytest.raises(RuntimeError):
            R.check_table(kind, params, dict(info, **{key: value}), coef)


@pytest.mark.skipif(refengine.available(), reason="the reference's own builder is used here")
@pytest.mark.parametrize("kind,params,wrong", [
    ("morse", (0.5, 5.0, 1.0, 1e-4, 3.0, 1e-3), (0.51, 5.0, 1.0, 1e-4, 3.0, 1e-3)),
    ("morse", (0.5, 5.0, 1.0, 1e-4, 3.0, 1e-3), (0.5, 5.0, 1.1, 1e-4, 3.0, 1e-3)),
    ("lj126", (0.275, 1.0, 9.5075e-6, 6.1545e-3, 1e-3), (0.275, 1.0, 9.5075e-6, 6.3e-3, 1e-3)),
    ("dpd", (25.0, 4.5, 3.0, 1.0, 0), (25.0, 4.5, 3.0, 1.1, 0))])
def test_a_builder_with_a_fault_is_not_taken_for_the_reference(monkeypatch, kind, params, wrong):
    assert R.reference_table(kind, params)[0] is not None
    right = W.make_potential
    monkeypatch.setattr(W, "make_potential", lambda k, p: right(kind, wrong))
    with pytest.raises(RuntimeError):
        R.reference_table(kind, params)
