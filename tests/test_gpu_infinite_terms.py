"""Infinite coefficients (hard constraints): rows that no such term matches stay finite, as a sum over the
matching terms has it, with and without a permutation group."""

import numpy as np
import pytest

from ls_helpers import LAT, ls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("k", [1, 5])
def test_only_matching_rows_are_infinite(symmetric, complex_, k):
    import torch
    n = 10
    basis = ls.SpinBasis(n, 4, None, ls.Symmetries(LAT.chain_symmetries(n, 0)) if symmetric else None)
    basis.build()
    states = np.array(basis.states)
    # n_i n_{i+1}, infinite on every bond; and a finite field on single sites
    m = np.array([(1 << i) | (1 << ((i + 1) % n)) for i in range(n)] + [1 << i for i in range(n)], dtype=np.uint64)
    v = np.array([np.inf] * n + [0.5] * n, dtype=np.complex128)
    zero = np.zeros(2 * n, dtype=np.uint64)
    empty = (np.zeros(0, dtype=np.complex128),) + tuple(np.zeros(0, dtype=np.uint64) for _ in range(5))
    op = ls.Operator._from_arrays(basis, empty, (v, m, m, m, zero, zero))
    x = np.random.default_rng(6).uniform(0.5, 1.0, size=(len(states), k)) * (1 + 0j if complex_ else 1)
    y = op.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    pairs = np.array([any((int(s) & int(b)) == int(b) for b in m[:n]) for s in states])
    assert pairs.any() and not pairs.all()
    assert np.isinf(y[pairs].real).all()
    # four particles of 0.5 each: exact
    assert np.array_equal(y[~pairs], 2.0 * x[~pairs])
