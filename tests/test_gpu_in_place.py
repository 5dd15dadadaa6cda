"""A product may overwrite its argument on bases with lattice symmetries (apply_device(x, out=x)): the
off-diagonal elements read a scaled copy of x, and a row's diagonal element only its own entry.  Sizes
that read the norms with x when the two are apart, and sizes that always make the copy."""

import numpy as np
import pytest

from ls_helpers import LAT, ls

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def operators():
    out = {}
    for n in (12, 16, 20, 24):
        b = ls.SpinBasis(n, n // 2, 1, ls.Symmetries(LAT.chain_symmetries(n, 0, 0)))
        b.build()
        out[n] = ls.Operator(b, LAT.xxz(LAT.chain_bonds(n), 1.0, 0.5))
    return out


@pytest.mark.parametrize("n", [12, 16, 20, 24])
@pytest.mark.parametrize("k", [1, 3, 4, 16, 20])
@pytest.mark.parametrize("complex_", [False, True])
def test_output_over_the_input(operators, n, k, complex_):
    import torch
    op = operators[n]
    D = op.basis.number_states
    rng = np.random.default_rng(n + k)
    x = torch.from_numpy(rng.normal(size=(D, k)) + (1j * rng.normal(size=(D, k)) if complex_ else 0)).cuda()
    expected = op.apply_device(x)
    for _ in range(5):
        y = x.clone()
        op.apply_device(y, out=y)
        # the same sums from x_j n_j or from x_j and n_j: equal to rounding
        assert float((y - expected).norm()) <= 1e-14 * float(expected.norm())


def test_overlapping_views(operators):
    """x and y as neighbouring columns of one block: their ranges overlap, their entries do not."""
    import torch
    op = operators[16]
    D = op.basis.number_states
    rng = np.random.default_rng(1)
    block = torch.from_numpy(rng.normal(size=(D, 4))).cuda()
    expected = op.apply_device(block[:, :2].contiguous())
    lib, stream = op._lib, torch.cuda.current_stream().cuda_stream
    assert lib.ls_gpu_matvec_f64(op._payload, 2, block.data_ptr(), 4, block.data_ptr() + 16, 4, 0, stream) == 0
    assert float((block[:, 2:] - expected).norm()) <= 1e-14 * float(expected.norm())
