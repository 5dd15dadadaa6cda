"""Representatives installed by the caller on bases without a group: as many states as the complete basis
has, but not those.  The two-table ranks would send their products anywhere; the search finds what is
there and drops the rest.  Against a dictionary of the states."""

import numpy as np
import pytest

from ls_helpers import ls

pytestmark = pytest.mark.gpu
FULL = sorted(s for s in range(256) if bin(s).count("1") == 3)


def _replaced(kind):
    states = list(FULL)
    if kind == "beyond":  # a particle on a site that the basis does not have
        states[-1] = (1 << 8) | 3
    elif kind == "high":
        states[-1] = (1 << 40) | 3
    elif kind == "none":
        pass
    return np.array(sorted(states), dtype=np.uint64)


@pytest.mark.parametrize("kind", ["none", "beyond", "high"])
@pytest.mark.parametrize("k", [1, 3])
def test_hops_within_the_installed_states(kind, k):
    import torch
    states = _replaced(kind)
    basis = ls.SpinlessFermionBasis(8, 3)
    basis._set_representatives(states)
    hop = ls.Operator(basis, ls.Expr("c†₀ c₁ + c†₁ c₀", sites=[[i, i + 1] for i in range(7)]))
    index = {int(s): i for i, s in enumerate(states)}
    x = np.random.default_rng(4).normal(size=(len(states), k))
    expected = np.zeros_like(x)
    for j, s in enumerate(states.tolist()):
        for i in range(7):
            t = s ^ (3 << i)
            if ((s >> i) ^ (s >> (i + 1))) & 1 and t in index:
                expected[index[t]] += x[j]
    y = hop.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    # at most 7 terms a row: 7 * 2^-53
    assert np.linalg.norm(y - expected) <= 1e-15 * np.linalg.norm(expected)
    y = hop.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()  # and once the check has been made
    assert np.linalg.norm(y - expected) <= 1e-15 * np.linalg.norm(expected)


def test_complete_two_species_states():
    import torch
    basis = ls.SpinfulFermionBasis(5, (2, 3))
    basis.build()
    states = np.array(basis.states)
    loaded = ls.SpinfulFermionBasis(5, (2, 3))
    loaded._set_representatives(states)
    e = ls.Expr("c†₀↑ c₁↑ + c†₁↑ c₀↑ + c†₀↓ c₁↓ + c†₁↓ c₀↓", sites=[[i, i + 1] for i in range(4)])
    x = torch.from_numpy(np.random.default_rng(5).normal(size=len(states))).cuda()
    assert torch.equal(ls.Operator(basis, e).apply_device(x), ls.Operator(loaded, e).apply_device(x))


def test_states_enumerated_for_another_basis():
    """56 states of weight 3 of 8 sites installed as those of weight 5, from the enumeration's own array."""
    from ctypes import byref
    import torch
    N = ls._native
    lib = N.lib()
    source, basis = ls.SpinlessFermionBasis(8, 3), ls.SpinlessFermionBasis(8, 5)
    array = N.chpl_external_array(None, 0, None)
    lib.ls_chpl_enumerate_representatives(source._payload, 0, 0, byref(array))
    N.check()
    assert int(array.num_elts) == len(FULL)
    lib.ls_hs_unchecked_set_representatives(basis._payload, byref(array), 22)
    N.check()
    op = ls.Operator(basis, ls.Expr("n₀", sites=[[i] for i in range(4)]))
    x = np.random.default_rng(11).normal(size=len(FULL))
    y = op.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    # at most 3 ones a row
    assert np.allclose(y, x * [bin(s & 15).count("1") for s in FULL], rtol=1e-15)
    assert op.kernel_route(1, False) == ("plain", 0)
