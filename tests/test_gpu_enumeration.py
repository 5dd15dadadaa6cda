"""The pruned enumeration of projected bases at its edges: ranges that do not fill a tile or a work
item, fixed and free Hamming weight, complex sectors under both membership rules, groups of one
element and of more elements than a CTA has threads.  Representatives are whole numbers: equality."""

import numpy as np
import pytest

import oracle as O
from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu


def chain(n, h, inv, momentum, parity=None):
    return ls.SpinBasis(n, h, inv, ls.Symmetries(LAT.chain_symmetries(n, momentum, parity)))


@pytest.mark.parametrize("n,h,inv,momentum,parity", [
    (3, 1, None, 0, None), (9, 4, None, 2, None), (14, 7, -1, 7, 1), (16, 8, 1, 3, None), (17, 5, None, 1, None),
    (20, 10, 1, 0, 0), (21, 10, None, 0, 1), (23, 11, None, 5, None), (24, 12, -1, 12, 1), (40, 4, None, 8, None),
    (63, 3, None, 21, None)])
def test_fixed_weight_matches_oracle(n, h, inv, momentum, parity):
    b = chain(n, h, inv, momentum, parity)
    c = Case(b, LAT.heisenberg(LAT.chain_bonds(n)))
    b.build()
    assert np.array_equal(b.states, c.oracle_states())


@pytest.mark.parametrize("n,momentum", [(5, 0), (12, 0), (13, 4), (16, 8)])
def test_all_weights_match_oracle(n, momentum):
    b = chain(n, None, None, momentum)
    c = Case(b, LAT.heisenberg(LAT.chain_bonds(n)))
    b.build()
    assert np.array_equal(b.states, c.oracle_states())


@pytest.mark.parametrize("momentum,inv", [(1, -1), (3, 1), (5, -1)])
def test_exact_rule_drops_the_zero_norms(momentum, inv):
    loose, exact = chain(16, 8, inv, momentum), chain(16, 8, inv, momentum)
    loose.build()
    exact.build(exact_norms=True)
    c = Case(loose, LAT.heisenberg(LAT.chain_bonds(16)))
    assert np.array_equal(loose.states, c.oracle_states())
    norms = c.oracle_norms_exact(loose.states)
    assert np.array_equal(exact.states, loose.states[norms > 0])


def test_group_larger_than_a_block():
    """Translations x Z2 of four rings of six sites: 6^4 = 1296 elements."""
    n = 24
    gens = []
    for ring in range(4):
        p = list(range(n))
        for i in range(6):
            p[6 * ring + i] = 6 * ring + (i + 1) % 6
        gens.append(ls.Symmetry(p, 0))
    b = ls.SpinBasis(n, 7, None, ls.Symmetries(gens))
    c = Case(b, LAT.heisenberg([(6 * r + i, 6 * r + (i + 1) % 6) for r in range(4) for i in range(6)]))
    assert c.group.order == 1296
    b.build()
    assert np.array_equal(b.states, c.oracle_states())
