"""Basis.build of many states holds the states, their index and 2 bytes per state of stabiliser sizes: the
orbit norms (16 bytes per state) come with the first call that needs them, and are those of the states."""

import numpy as np
import pytest

from ls_helpers import ls

pytestmark = pytest.mark.gpu


def test_large_build_leaves_the_norms_for_later():
    import torch
    n = 26
    reflection = ls.Symmetries([ls.Symmetry(list(range(n - 1, -1, -1)), 0)])
    small = ls.SpinBasis(12, 6, None, ls.Symmetries([ls.Symmetry(list(range(11, -1, -1)), 0)]))
    small.build()  # the library's own scratch and the context
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    basis = ls.SpinBasis(n, n // 2, None, reflection)
    basis.build()
    D = basis.number_states
    assert D == 5200300
    held = before - torch.cuda.mem_get_info()[0]
    # states 8, suffixes of the index 2, stabilisers 2 bytes; at most 2^24 bucket starts of 4 bytes
    assert held < 12 * D + 4 * 2 ** 24 + 4 * 2 ** 20
    norms = torch.as_tensor(basis.device_norms(), device="cuda").cpu().numpy()
    states = basis.states
    pick = np.sort(np.random.default_rng(7).choice(D, size=20000, replace=False))
    expected = basis.state_info(states[pick])[2]
    # the same square root of the same quotient
    assert np.abs(norms[pick] - expected).max() <= 2e-16
    # 13 of 26 spins: a mirror image of itself would have an even weight, so every orbit has two states
    assert np.array_equal(np.unique(norms), [np.sqrt(0.5)])
