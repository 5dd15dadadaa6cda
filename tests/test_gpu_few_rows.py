"""Which kernels a product runs (Operator.kernel_route): few rows keep a warp per row where that is faster, a
lane per element takes the rest.  Every case on both sides of the line against the oracle.

Tolerance: rows sum at most a few hundred products, FP64 rounding stays below 3e-14 relative L2; 1e-12
is the bound of the parity tests."""

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-12


def shift(n, step):
    return ls.Symmetries([ls.Symmetry([(i + step) % n for i in range(n)], 0)])


def chain(n, h, inversion=None, symmetries=None):
    return Case(ls.SpinBasis(n, h, inversion, symmetries or ls.Symmetries(LAT.chain_symmetries(n, 0))),
                LAT.heisenberg(LAT.chain_bonds(n)))


def square(L, h, point_group=True):
    return Case(ls.SpinBasis(L * L, h, None, ls.Symmetries(LAT.square_symmetries(L, 0, 0, point_group))),
                LAT.heisenberg(LAT.square_bonds(L)))


def triangular5(h):
    return Case(ls.SpinBasis(25, h, None, ls.Symmetries(LAT.triangular_symmetries(5, 0, 0, 0))),
                LAT.heisenberg(LAT.triangular_bonds(5)))


# name: (case, {(k, complex): route})
CASES = {
    "chain24_inversion": (lambda: chain(24, 12, 1, ls.Symmetries(LAT.chain_symmetries(24, 0, 0))),
                          {(1, False): ("rows", 0), (16, True): ("rows", 0)}),
    "chain48_h4": (lambda: chain(48, 4),  # 4060 rows
                   {(1, False): ("packed", 2), (1, True): ("packed", 2), (3, True): ("rows", 2), (16, True): ("packed", 2)}),
    "chain36_h5": (lambda: chain(36, 5), {(1, False): ("rows", 2), (1, True): ("rows", 2), (4, True): ("rows", 2)}),
    "chain48_three": (lambda: chain(48, 3, None, shift(48, 16)), {(1, True): ("rows", 2), (2, False): ("rows", 2)}),
    "chain60_h3": (lambda: chain(60, 3),  # no candidate index fits beside 60 bits: only the kernel without tables
                   {(1, False): ("fallback", 2), (1, True): ("fallback", 2), (2, True): ("rows", 2)}),
    "square6_h3": (lambda: square(6, 3), {(1, False): ("packed", 9), (2, False): ("packed", 9), (2, True): ("rows", 9),
                                          (16, True): ("packed", 9)}),
    "square6_translations": (lambda: square(6, 3, False), {(1, True): ("packed", 2), (5, False): ("rows", 2)}),
    "triangular5_h8": (lambda: triangular5(8), {(1, False): ("rows", 5), (1, True): ("rows", 5), (8, True): ("rows", 5)}),
    "triangular5_h3": (lambda: triangular5(3), {(1, True): ("rows", 0)}),
    "hypercube": (lambda: Case(ls.SpinBasis(16, 8, 1, ls.Symmetries(LAT.hypercube_symmetries(4))),
                               LAT.heisenberg(LAT.hypercube_bonds(4))),
                  {(1, False): ("packed", 12), (16, True): ("packed", 12), (3, True): ("rows", 16)}),
    "square4_inversion": (lambda: Case(ls.SpinBasis(16, 8, -1, ls.Symmetries(LAT.square_symmetries(4, 2, 2))),
                                       LAT.heisenberg(LAT.square_bonds(4))),
                          {(1, False): ("rows", 5), (1, True): ("rows", 5), (3, True): ("rows", 5), (5, False): ("rows", 5)}),
    "triangular4_inversion": (lambda: Case(ls.SpinBasis(16, 8, 1, ls.Symmetries(LAT.triangular_symmetries(4, 0, 0, 0, 0))),
                                           LAT.heisenberg(LAT.triangular_bonds(4))),
                              {(1, True): ("rows", 9), (3, True): ("rows", 9), (2, True): ("rows", 9)}),
    "free": (lambda: Case(ls.SpinBasis(12, 5), LAT.heisenberg(LAT.chain_bonds(12))), {(1, True): ("free", 0)}),
    "free41": (lambda: Case(ls.SpinBasis(41, 2), LAT.heisenberg(LAT.chain_bonds(41))), {(1, True): ("plain", 0)}),
}


@pytest.fixture(scope="module")
def cases():
    out = {}
    for name, (make, routes) in CASES.items():
        out[name] = (make(), routes)
        out[name][0].basis.build(exact_norms=True)
    return out


@pytest.mark.parametrize("name", sorted(CASES))
def test_route_and_product(cases, name):
    import torch
    c, routes = cases[name]
    states = np.array(c.basis.states)
    D = len(states)
    rng = np.random.default_rng(9)
    for (k, complex_), route in routes.items():
        assert c.op.kernel_route(k, complex_) == route
        x = rng.normal(size=(D, k)) + (1j * rng.normal(size=(D, k)) if complex_ else 0)
        xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        y = c.op.apply_device(xd).cpu().numpy()
        ya = c.op.apply_device(xd, adjoint=True).cpu().numpy()  # H is Hermitian
        for j in {0, k - 1}:
            expected = c.oracle_matvec(states, np.ascontiguousarray(x[:, j]), complex_=complex_)
            assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(expected)
            assert np.linalg.norm(ya[:, j] - expected) <= RTOL * np.linalg.norm(expected)


def test_fermions_of_few_rows():
    """128 elements, 2506 rows: blocks of 16 by the packed kernels, one column by 32-bit states; the two
    agree, and with the complex kernels of the other family (three columns)."""
    import torch
    b = ls.SpinfulFermionBasis(16, (2, 2), ls.Symmetries(LAT.square_symmetries(4, 0, 0)))
    b.build()
    op = ls.Operator(b, LAT.hubbard(LAT.square_bonds(4), 1.0, 4.0))
    assert op.kernel_route(16, True) == ("packed", 4)
    assert op.kernel_route(1, True) == op.kernel_route(3, True) == ("rows", 0)
    rng = np.random.default_rng(10)
    x = torch.from_numpy(rng.normal(size=(b.number_states, 16)) + 1j * rng.normal(size=(b.number_states, 16))).cuda()
    y = op.apply_device(x)
    for j in (0, 7, 15):
        one = op.apply_device(x[:, j].contiguous())
        assert float((y[:, j] - one).norm()) <= RTOL * float(one.norm())
    three = op.apply_device(x[:, :3].contiguous())
    assert float((y[:, :3] - three).norm()) <= RTOL * float(three.norm())


def test_kernel_info_is_that_of_the_warp_per_row_kernels(cases):
    """It keeps its meaning where the lane-per-element kernels run: whether the packed tables fit."""
    assert cases["chain60_h3"][0].op.kernel_info() == ("fallback", 2)
    assert cases["chain36_h5"][0].op.kernel_info() == ("packed", 2)
    assert cases["free"][0].op.kernel_info() == ("plain", 0)
