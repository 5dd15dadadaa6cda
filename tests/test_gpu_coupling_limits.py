"""ls_gpu_coupling_inner_products refuses numbers of couplings, and bases, that the fused kernels do not
take before it makes anything of that size: callers try the fused form first, with any number."""

import ctypes

import numpy as np
import pytest

from ls_helpers import LAT, ls

pytestmark = pytest.mark.gpu
EMPTY = (np.zeros(0, dtype=np.complex128),) + tuple(np.zeros(0, dtype=np.uint64) for _ in range(5))


def _refused(op, n_couplings, message):
    import torch
    lib = ls._native.lib()
    n_terms = op.number_off_diag_terms + op.number_diag_terms
    ids = np.zeros(max(n_terms, 1), dtype=np.int32)
    v = torch.ones(op.basis.number_states, dtype=torch.complex128, device="cuda")
    out = torch.zeros(4, dtype=torch.complex128, device="cuda")
    rc = lib.ls_gpu_coupling_inner_products(op._payload, n_couplings, ids.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
                                            v.data_ptr(), v.data_ptr(), out.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream)
    assert rc != 0 and message in lib.ls_gpu_last_error().decode()
    assert (out == 0).all()


@pytest.mark.parametrize("n_couplings", [0, -1, 5, 1 << 30])
@pytest.mark.parametrize("empty", [False, True])
def test_number_of_couplings(n_couplings, empty):
    basis = ls.SpinBasis(10, 5, None, ls.Symmetries(LAT.chain_symmetries(10, 0)))
    basis.build()
    if empty:
        op = ls.Operator._from_arrays(basis, EMPTY, EMPTY)
    else:
        op = ls.Operator(basis, LAT.heisenberg(LAT.chain_bonds(10)))
    out_of_range = not empty and n_couplings <= 0  # the ids are checked first
    _refused(op, n_couplings, "out of range" if out_of_range else "1 to 4 couplings")


def test_group_and_basis():
    big = ls.SpinBasis(25, 3, None, ls.Symmetries(LAT.square_symmetries(5, 0, 0)))  # 200 elements
    big.build()
    _refused(ls.Operator(big, LAT.heisenberg(LAT.square_bonds(5))), 2, "128 elements")
    free = ls.SpinBasis(10, 5)
    free.build()
    _refused(ls.Operator(free, LAT.heisenberg(LAT.chain_bonds(10))), 2, "lattice symmetries")
