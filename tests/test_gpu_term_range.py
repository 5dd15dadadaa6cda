"""Operators whose terms name a site beyond the basis (an open chain written with one bond too many).
Without a permutation group the states that such a term makes have no index and are dropped, so the
product is that of the other terms; bases with lattice symmetries refuse the operator, because the group
does not act on that site.

The products are compared with those of the operator without the stray terms: at most 40 products a row,
FP64 rounding below 40 * 2^-53 = 4.5e-15 relative L2."""

import numpy as np
import pytest

from ls_helpers import LAT, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-13

HOP = "c†₀ c₁ + c†₁ c₀"
FLIP = "σ⁺₀ σ⁻₁ + σ⁻₀ σ⁺₁"


def _bonds(n):
    return [[i, i + 1] for i in range(n)]


BASES = {
    "spinless": (lambda: ls.SpinlessFermionBasis(8, 3), HOP),
    "spinless_all": (lambda: ls.SpinlessFermionBasis(8), HOP),
    "fixed_weight": (lambda: ls.SpinBasis(8, 4), FLIP),
    "inversion": (lambda: ls.SpinBasis(8, 4, -1), FLIP),
    "all_spins": (lambda: ls.SpinBasis(8), FLIP),
    "spins33": (lambda: ls.SpinBasis(33, 2), FLIP),  # wider than 32-bit states
}


@pytest.mark.parametrize("name", sorted(BASES))
@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("complex_", [False, True])
def test_states_beyond_the_basis_are_dropped(name, k, complex_):
    import torch
    make, term = BASES[name]
    basis = make()
    basis.build()
    n = basis.number_bits
    stray = ls.Operator(basis, ls.Expr(term, sites=_bonds(n)))  # the last bond ends at site n
    inside = ls.Operator(basis, ls.Expr(term, sites=_bonds(n - 1)))
    rng = np.random.default_rng(2)
    x = rng.normal(size=(basis.number_states, k)) + (1j * rng.normal(size=(basis.number_states, k)) if complex_ else 0)
    x = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    for adjoint in (False, True):
        y, expected = stray.apply_device(x, adjoint=adjoint), inside.apply_device(x, adjoint=adjoint)
        assert float((y - expected).abs().square().sum()) <= RTOL ** 2 * float(expected.abs().square().sum())


def test_symmetric_bases_refuse_a_flip_beyond_them():
    import torch
    basis = ls.SpinBasis(8, 4, None, ls.Symmetries(LAT.chain_symmetries(8, 0)))
    basis.build()
    op = ls.Operator(basis, LAT.heisenberg(LAT.chain_bonds(8)) + ls.Expr(FLIP, sites=[[7, 8]]))
    x = torch.ones(basis.number_states, dtype=torch.float64, device="cuda")
    with pytest.raises(RuntimeError, match="beyond"):
        op.apply_device(x)
    # a diagonal term there sees an empty site: sigma^z of it is a constant
    H = LAT.heisenberg(LAT.chain_bonds(8))
    x = torch.from_numpy(np.random.default_rng(3).normal(size=basis.number_states)).cuda()
    plain = ls.Operator(basis, H).apply_device(x)
    with_z = ls.Operator(basis, H + ls.Expr("σᶻ₀", sites=[[8]])).apply_device(x)
    free = ls.SpinBasis(8, 4)
    free.build()
    sign = ls.Operator(free, ls.Expr("σᶻ₀", sites=[[8]])).apply_diag_to_basis_state(int(basis.states[0]))
    assert abs(sign) == 1.0
    assert float((with_z - plain - sign * x).norm()) <= RTOL * float(plain.norm())
