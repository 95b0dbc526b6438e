"""The pair statistics are a query: forces, energies, species values and bonds are the same to the bit with it
and without it, before a step and between steps."""
import numpy as np
import pytest

from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _species():
    return W.species(n=2000, L=8.0, seed=3)


def _breaking():  # bond lengths spread around the break threshold: the first force pass decides
    return W.lattice(nx=8, seed=17, noise=5e-3)


@pytest.mark.parametrize("make", [_species, _breaking])
def test_pair_counts_change_nothing(make):
    got = []
    for ask in (False, True):
        scn = make()
        u = W.build_gpu(scn)
        u.force()
        u.steps(1)

        def query():
            if not ask:
                return
            before = [a.copy() for a in u.state()], u.energies()
            assert u.candidate_pairs() > 0
            after = u.state(), u.energies()
            assert all(np.array_equal(p, q) for p, q in zip(before[0], after[0])) and before[1] == after[1]

        query()
        u.steps(1)
        query()
        u.steps(1)
        out = list(u.state()) + [np.array(u.energies())]
        if "sp_values" in scn:
            out.append(np.asarray(u.species_values()))
        if "bi" in scn:
            out.append(u.bond_flags())
        got.append(out)
        u.close()
    assert all(np.array_equal(p, q) for p, q in zip(*got))
    if make is _breaking:
        assert 0 < (got[0][-1] != 0).sum() < len(got[0][-1])


def test_a_query_before_the_first_pass_breaks_no_bond():
    u = W.build_gpu(_breaking())
    u.candidate_pairs()
    assert (u.bond_flags() & 1).all()
    u.close()
