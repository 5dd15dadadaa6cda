"""Enumeration with few group elements, where a thread per candidate takes the place of pruned blocks: on
both sides of the rule, ranges that do not fill a tile, complex sectors under both membership rules,
inversion, all weights, fermions.  States against the oracle or a plain restatement (whole numbers:
equality), orbit norms against the square roots of the exact stabiliser counts."""

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu


def shift(n, step, sector=0):
    return ls.Symmetries([ls.Symmetry([(i + step) % n for i in range(n)], sector)])


def mirror(n, sector=0):
    return ls.Symmetries([ls.Symmetry(list(range(n - 1, -1, -1)), sector)])


def device_norms(basis):
    import torch
    return torch.as_tensor(basis.device_norms(), device="cuda").cpu().numpy()


CASES = {
    "mirror20": lambda: ls.SpinBasis(20, 10, None, mirror(20)),
    "odd_mirror21": lambda: ls.SpinBasis(21, 10, None, mirror(21, 1)),
    "mirror20_inversion": lambda: ls.SpinBasis(20, 10, -1, mirror(20)),  # 92378 candidates: the smallest groups
    "four20": lambda: ls.SpinBasis(20, 10, None, shift(20, 5)),
    "four20_complex": lambda: ls.SpinBasis(20, 10, None, shift(20, 5, 1)),
    "five20_inversion": lambda: ls.SpinBasis(20, 10, 1, shift(20, 4)),  # pruned: 1e5 candidates, 8 images
    "seven21_complex": lambda: ls.SpinBasis(21, 9, None, shift(21, 3, 2)),
    "twelve24": lambda: ls.SpinBasis(24, 6, None, shift(24, 2, 6)),  # 134596 candidates
    "fifteen30": lambda: ls.SpinBasis(30, 4, None, shift(30, 2)),  # pruned: few candidates
    "eighteen40": lambda: ls.SpinBasis(40, 4, None, shift(40, 4)),  # 10 images of 40 bits, 91390 candidates
    "twenty40": lambda: ls.SpinBasis(40, 5, None, shift(40, 2)),  # pruned, at the line of 40 bits
    "three18_all": lambda: ls.SpinBasis(18, None, None, shift(18, 6)),
    "two16_all": lambda: ls.SpinBasis(16, None, None, mirror(16)),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("exact", [False, True])
def test_states_and_norms(name, exact):
    basis = CASES[name]()
    c = Case(basis, LAT.heisenberg(LAT.chain_bonds(basis.number_bits)))
    basis.build(exact_norms=exact)
    states = np.array(basis.states)
    expected = c.oracle_states()
    norms = c.oracle_norms_exact(expected)
    if exact:
        expected, norms = expected[norms > 0], norms[norms > 0]
    assert np.array_equal(states, expected)
    assert np.abs(device_norms(basis) - norms).max() <= 2e-16  # one rounding of a root below 1


def _parity(perm, x):
    """Parity of the permutation that `perm` (bit i of g.x = bit perm[i] of x) induces on the set bits."""
    to = {p: i for i, p in enumerate(perm)}
    odd = np.zeros(len(x), dtype=np.uint64)
    for l in range(len(perm)):
        for k in range(l):
            if to[k] > to[l]:
                odd ^= (x >> np.uint64(k)) & (x >> np.uint64(l)) & np.uint64(1)
    return odd.astype(np.int64)


@pytest.mark.parametrize("n,up,down,step,sector", [(10, 4, 5, 5, 0), (10, 5, 5, 5, 1), (12, 4, 4, 3, 0), (12, 3, 5, 3, 2)])
def test_fermions(n, up, down, step, sector):
    """Groups of 2 and 4 elements in real sectors, signs of the permuted orbitals included."""
    symmetries = shift(n, step, sector)
    basis = ls.SpinfulFermionBasis(n, (up, down), symmetries)
    basis.build()

    def weight(h):
        return np.array([s for s in range(1 << n) if bin(s).count("1") == h], dtype=np.uint64)

    x = ((weight(down)[:, None] << np.uint64(n)) | weight(up)[None, :]).reshape(-1)
    smallest, count = np.ones(len(x), dtype=bool), np.zeros(len(x))
    trivial = np.ones(len(x), dtype=bool)
    order = n // step
    for e in range(order):
        site = [(i + e * step) % n for i in range(n)]
        perm = site + [n + i for i in site]
        y = np.zeros_like(x)
        for i, p in enumerate(perm):
            y |= ((x >> np.uint64(p)) & np.uint64(1)) << np.uint64(i)
        chi = np.cos(2 * np.pi * e * sector / order)  # real sectors: +-1
        smallest &= y >= x
        fixed = y == x
        count += fixed
        trivial &= ~fixed | (np.where(_parity(perm, x) == 1, -1.0, 1.0) * chi > 0.5)
    keep = smallest & trivial
    assert np.array_equal(np.array(basis.states), x[keep])
    assert np.abs(device_norms(basis) - np.sqrt(count[keep] / order)).max() <= 2e-16
