"""Representatives enumerated through the plugin table and freed by the caller, no index having been built:
their device copies (states, norms or stabiliser sizes) go with them."""

from ctypes import byref

import numpy as np
import pytest

from ls_helpers import ls

pytestmark = pytest.mark.gpu


def test_freed_states_leave_nothing_on_the_device():
    import torch
    N = ls._native
    lib = N.lib()
    n = 24
    basis = ls.SpinBasis(n, n // 2, None, ls.Symmetries([ls.Symmetry(list(range(n - 1, -1, -1)), 0)]))

    def once():
        array = N.chpl_external_array(None, 0, None)
        lib.ls_chpl_enumerate_representatives(basis._payload, 0, 0, byref(array))
        N.check()
        count = int(array.num_elts)
        lib.ls_hs_internal_destroy_external_array(byref(array))
        return count

    D = once()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(8):
        assert once() == D
    torch.cuda.synchronize()
    # 24 bytes a state would be 0.26 GB over the calls
    assert before - torch.cuda.mem_get_info()[0] < 8 * D
    # a basis built afterwards finds its own states, whatever host address they get
    other = ls.SpinBasis(n, n // 2, None, ls.Symmetries([ls.Symmetry(list(range(n - 1, -1, -1)), 1)]))
    other.build()
    states = np.array(other.states)
    assert np.array_equal(other.index(states[::1000]), np.arange(0, len(states), 1000))
