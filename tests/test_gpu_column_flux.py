"""Species fluxes by the column kernel against an FP64 evaluation of every pair: groups at the edges of
32, three cells along an axis, sparse and coarse cells, fluxes within one type in both orders, a type
without species, and carried rates; one, four and eight warps per group."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _expected(x, t, L, values, fluxes, konst, dt):
    d = x[:, None] - x[None]
    d -= L * np.round(d / L)
    r = np.sqrt((d ** 2).sum(2))
    w = np.where((r <= 1.0) & ~np.eye(len(x), dtype=bool), (1 - np.minimum(r, 1.0)) ** 2, 0.0)
    rate = np.zeros_like(values)
    for (kind, ta, tb, ia, ib, k, decay, target) in fluxes:
        sa, sb = values[:, ia][:, None], values[:, ib][None]
        q = k * (sa - sb) if kind == 0 else np.maximum(k * (sa - target), 0) if kind == 1 else np.maximum(k * (target - sb) * sa, 0)
        on = (t[:, None] == ta) & (t[None] == tb)
        if ta == tb:
            on &= np.triu(np.ones_like(on), 1)  # each pair once, the lower id as a (Fick: either way)
        q = w * q * on
        c = (w > 0) * on
        rate[:, ia] -= q.sum(1) + 0.5 * decay * values[:, ia] * c.sum(1)
        rate[:, ib] += q.sum(0) - 0.5 * decay * values[:, ib] * c.sum(0)
    return np.where(konst, values, values + dt * rate)


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("n,cells,h", [(31, 3, 1.0), (500, 3, 1.0), (777, 5, 1.0), (600, 3, 2.5), (300, 9, 1.0)])
def test_fluxes_match_every_pair(n, cells, h, variant):
    rng = np.random.default_rng(n)
    L = cells * h
    x = np.minimum(rng.uniform(0, L, size=(n, 3)), L * (1 - 1e-6)).astype(np.float32).astype(np.float64)
    t = (np.arange(n) % 3).astype(np.int32)  # type 2 carries no species
    fluxes = [(0, 0, 0, 0, 0, 2.0, 0.1, 0.0), (1, 1, 0, 1, 1, 1.0, 0.0, 0.5), (2, 0, 1, 0, 0, 0.5, 0.05, 1.0)]
    values = rng.uniform(0, 1, size=(n, 3)).astype(np.float32)
    values[t == 2] = 0
    values[t == 1, 2] = 0
    scn = dict(dim=[L] * 3, cells=[cells] * 3, cutoff=1.0, dt=0.01, bc=("periodic",) * 3, types=[(1.0, 0.3, m.Newtonian)] * 3,
               pots=[], forces=[], x=x, v=np.zeros_like(x), t=t, sp_nspec=np.array([3, 2, 0], dtype=np.int32),
               sp_names=[["S1", "S2", "$S3"], ["S1", "S2"], []],
               sp_flags=np.array([[0, 0, 4], [0, 0, 0], [0, 0, 0]], dtype=np.uint32), sp_values=values, fluxes=fluxes)
    u = W.build_gpu(scn)
    u.force_config(variant, 1 << 20)
    konst = np.zeros((n, 3), dtype=bool)
    konst[t == 0, 2] = True
    want = values.astype(np.float64)
    for _ in range(2):  # nothing moves, so every particle keeps its cell and its values advance
        u.steps(1)
        want = _expected(x, t, L, want, fluxes, konst, 0.01)
    got = u.species_values()
    # rates of up to a few hundred FP32 terms of order one, times dt
    assert np.abs(got - want).max() <= 0.01 * 300 * 2.0 ** -22 + 2.0 ** -22
    u.force()  # rates accumulate until they are integrated: two passes, then one step with three
    u.force()
    u.steps(1)
    once = _expected(x, t, L, got.astype(np.float64), fluxes, konst, 0.01)
    assert np.abs(u.species_values() - (got + 3 * (once - got))).max() <= 0.03 * 300 * 2.0 ** -22 + 2.0 ** -22
    u.close()
