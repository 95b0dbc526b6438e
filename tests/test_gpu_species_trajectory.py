"""Trajectories of a fluid with species keep the cell kernel's order of the force sums. Two events that the
last bit of a position decides, each within four steps of 50,021 particles: a pair 7e-9 beyond the cutoff,
where the Morse force is 0.465 and not zero (seed 0), and a particle on a face of its cell, whose rates carry
over when it crosses (seed 6). The values are those of the engine with the cell kernel, to the bit."""
import numpy as np
import pytest

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _run(seed, n=50021):
    scn = W.species(n=n, L=(n / 4.0) ** (1 / 3), seed=seed)
    scn["types"] = [(1.0, 0.7, m.Newtonian)] * 2  # the wells at r = 0.8: the fluid does not collapse
    u = W.build_gpu(scn)
    u.steps(4)
    x, v, f, c, xr = u.state()
    s = np.asarray(u.species_values()).reshape(n, -1)
    u.close()
    return v, c, s


def test_a_pair_at_the_cutoff():
    v, c, _ = _run(0)
    want = np.float32([[-1.0663799047470093, -3.4995076656341553, -2.2685887813568115],
                       [-1.5468677282333374, -1.9215521812438965, 3.9688005447387695]])
    assert list(c[[2797, 39790]]) == [8546, 9075]
    assert np.array_equal(v[[2797, 39790]], want)


def test_a_particle_on_the_face_of_its_cell():
    _, c, s = _run(6)
    assert c[18239] == 10023
    # its values are sums of FP32 rates times dt, in another order by another flux kernel: two units in the last
    # place of one, where the carried step is 4e-3
    assert np.abs(s[18239] - np.float32([0.4812968671321869, 0.9137512445449829, 0.6121189594268799])).max() <= 2.4e-7
