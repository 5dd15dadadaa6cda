"""Matvecs on bases without a permutation group (two-table ranks, a thread per row and column) against
the CPU oracle: every kind of complete basis, widths around the 32-bit states and the widest rank
tables, ragged columns, an incomplete set of states (which keeps the search).

Tolerance: rows sum at most a few hundred products, FP64 rounding stays below 3e-14 relative L2; 1e-12
is the bound of the parity tests."""

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-12


def _spins(n):
    return LAT.xxz(LAT.chain_bonds(n), 1.0, 0.7) + LAT.dm_z(LAT.chain_bonds(n), 0.3)


def _case(name):
    if name == "all_states":
        e = _spins(9) + ls.Expr("σˣ₀", sites=[[i] for i in range(9)]).scale(0.4)
        return Case(ls.SpinBasis(9), e)
    if name == "odd_weight":
        return Case(ls.SpinBasis(13, 6), _spins(13))
    if name == "one_site":
        return Case(ls.SpinBasis(1), ls.Expr("σˣ₀", sites=[[0]]))
    if name == "no_particles":
        return Case(ls.SpinBasis(6, 0), _spins(6))
    if name == "inversion":
        return Case(ls.SpinBasis(12, 6, -1), LAT.heisenberg(LAT.chain_bonds(12)))
    if name == "bits26":  # the last width whose tables sit in shared memory
        return Case(ls.SpinBasis(26, 3), _spins(26))
    if name == "bits32":
        return Case(ls.SpinBasis(32, 3), _spins(32))
    if name == "bits33":
        return Case(ls.SpinBasis(33, 3), _spins(33))
    if name == "bits40":
        return Case(ls.SpinBasis(40, 2), _spins(40))
    if name == "bits41":  # wider than the rank tables: the search kernel
        return Case(ls.SpinBasis(41, 2), _spins(41))
    if name == "spinless":
        e = ls.Expr("c†₀ c₁ + c†₁ c₀", sites=[[i, (i + 1) % 11] for i in range(11)]) + \
            ls.Expr("n₀ n₁", sites=[[i, (i + 1) % 11] for i in range(11)]).scale(1.7)
        return Case(ls.SpinlessFermionBasis(11, 4), e)
    if name == "hubbard":
        return Case(ls.SpinfulFermionBasis(7, (3, 4)), LAT.hubbard(LAT.chain_bonds(7), 1.0, 3.0))
    if name == "hubbard_total":
        return Case(ls.SpinfulFermionBasis(5, 4), LAT.hubbard(LAT.chain_bonds(5), 1.0, 3.0))
    if name == "hubbard_all":
        return Case(ls.SpinfulFermionBasis(4), LAT.hubbard(LAT.chain_bonds(4), 1.0, 3.0))
    if name == "diagonal":  # no off-diagonal terms at all
        return Case(ls.SpinBasis(9, 4), ls.Expr("σᶻ₀ σᶻ₁", sites=[list(b) for b in LAT.chain_bonds(9)]))
    if name == "all_pairs":  # more than 32 term slots
        return Case(ls.SpinBasis(12, 5), LAT.heisenberg([(i, j) for i in range(12) for j in range(i)]))
    raise KeyError(name)


NAMES = ["all_states", "odd_weight", "one_site", "no_particles", "inversion", "bits26", "bits32", "bits33", "bits40",
         "bits41", "spinless", "hubbard", "hubbard_total", "hubbard_all", "all_pairs", "diagonal"]


@pytest.mark.parametrize("name", NAMES)
def test_columns_match_oracle(name):
    import torch
    c = _case(name)
    c.basis.build()
    states = np.array(c.basis.states)
    D = len(states)
    rng = np.random.default_rng(7)
    for k in (1, 3, 4, 18):
        x = rng.normal(size=(D, k)) + 1j * rng.normal(size=(D, k))
        xd = torch.from_numpy(x).cuda()
        y = c.op.apply_device(xd).cpu().numpy()
        ya = c.op.apply_device(xd, adjoint=True).cpu().numpy()
        yr = c.op.apply_device(torch.from_numpy(x.real.copy()).cuda()).cpu().numpy()
        for j in {0, k - 1}:
            expected = c.oracle_matvec(states, np.ascontiguousarray(x[:, j]), complex_=True)
            bound = RTOL * np.linalg.norm(expected) + 1e-300
            assert np.linalg.norm(y[:, j] - expected) <= bound
            assert np.linalg.norm(ya[:, j] - expected) <= bound  # all operators here are Hermitian
            real = c.oracle_matvec(states, np.ascontiguousarray(x[:, j].real))
            assert np.linalg.norm(yr[:, j] - real) <= bound


def test_incomplete_states_keep_the_search():
    """Externally installed states that are only part of a fixed-weight fermionic basis."""
    import torch
    b = ls.SpinlessFermionBasis(8, 3)
    full = np.array(sorted(s for s in range(256) if bin(s).count("1") == 3), dtype=np.uint64)
    part = full[::2].copy()
    b._set_representatives(part)
    op = ls.Operator(b, ls.Expr("n₀", sites=[[i] for i in range(3)]))  # diagonal: closed on any set
    x = torch.arange(1.0, len(part) + 1, dtype=torch.float64, device="cuda")
    y = op.apply_device(x).cpu().numpy()
    expected = np.array([bin(int(s) & 7).count("1") for s in part]) * np.arange(1.0, len(part) + 1)
    assert np.array_equal(y, expected)
    hop = ls.Operator(b, ls.Expr("c†₀ c₁ + c†₁ c₀", sites=[[i, i + 1] for i in range(7)]))
    y = hop.apply_device(x).cpu().numpy()  # targets outside the set are dropped
    index = {int(s): i for i, s in enumerate(part)}
    expected = np.zeros(len(part))
    for j, s in enumerate(part):
        for i in range(7):
            t = int(s) ^ (3 << i)
            if ((int(s) >> i) ^ (int(s) >> (i + 1))) & 1 and t in index:
                expected[index[t]] += (j + 1.0)
    assert np.allclose(y, expected, rtol=1e-12)


def test_particle_number_breaking_term_is_reported():
    import torch
    b = ls.SpinBasis(10, 5)
    b.build()
    op = ls.Operator(b, LAT.heisenberg(LAT.chain_bonds(10)) + ls.Expr("σˣ₀", sites=[[3]]))
    with pytest.raises(RuntimeError, match="particle numbers"):
        op.apply_device(torch.ones(b.number_states, dtype=torch.float64, device="cuda"))
