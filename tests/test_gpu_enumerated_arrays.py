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


@pytest.mark.parametrize("symmetric", [True, False])
def test_part_of_an_enumerated_array(symmetric):
    """The first half of an enumerated array, installed as it lies and from a copy: the same basis."""
    import torch
    from ls_helpers import LAT
    N = ls._native
    lib = N.lib()
    n = 12

    def new():
        return ls.SpinBasis(n, 5, None, ls.Symmetries(LAT.chain_symmetries(n, 0))) if symmetric \
            else ls.SpinlessFermionBasis(n, 5)

    source = new()
    array = N.chpl_external_array(None, 0, None)
    lib.ls_chpl_enumerate_representatives(source._payload, 0, 0, byref(array))
    N.check()
    count = int(array.num_elts)
    full = np.ctypeslib.as_array((N.c_uint64 * count).from_address(array.elts)).copy()
    half = N.chpl_external_array(array.elts, count // 2, None)
    lying, copied = new(), new()
    lib.ls_hs_unchecked_set_representatives(lying._payload, byref(half), 22)
    N.check()
    copied._set_representatives(full[:count // 2].copy())
    expr = LAT.heisenberg(LAT.chain_bonds(n)) if symmetric else ls.Expr("c†₀ c₁ + c†₁ c₀", sites=[[i, i + 1] for i in range(n - 1)])
    x = torch.from_numpy(np.random.default_rng(8).normal(size=(count // 2, 3))).cuda()
    a, b = ls.Operator(lying, expr).apply_device(x), ls.Operator(copied, expr).apply_device(x)
    assert torch.equal(a, b) and float(a.norm()) > 0
    na, nb = (torch.as_tensor(v.device_norms(), device="cuda") for v in (lying, copied))
    assert torch.equal(na, nb)
