"""The row-group matvec kernels at the edges of their shapes: both scan modes (whole 32-bit states, 16-bit
prefixes), group sizes around the scan's chunks, rows around the group of rows of a warp, ragged
numbers of real and complex columns, flip patterns of one to four sites, non-finite inputs.

Every output against the CPU oracle.  Tolerance: a row sums at most a few hundred products, so FP64
rounding stays below 300 * 2^-53 = 3e-14 relative L2; 1e-12 is the bound of the parity tests."""

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-12


def _case(name):
    S = ls.Symmetries
    if name == "chain9":  # 9 elements: the second chunk holds one
        return Case(ls.SpinBasis(9, 4, None, S(LAT.chain_symmetries(9, 1))), LAT.xxz(LAT.chain_bonds(9), 1.0, 0.3))
    if name == "chain16_inversion":  # 32 elements, whole chunks
        return Case(ls.SpinBasis(16, 8, -1, S(LAT.chain_symmetries(16, 8, 1))), LAT.heisenberg(LAT.chain_bonds(16)))
    if name == "chain32":  # the widest state of the 32-bit scan
        return Case(ls.SpinBasis(32, 3, None, S(LAT.chain_symmetries(32, 5))), LAT.heisenberg(LAT.chain_bonds(32)))
    if name == "chain33":  # the narrowest that needs prefixes; 33 elements: the third chunk holds one
        return Case(ls.SpinBasis(33, 3, None, S(LAT.chain_symmetries(33, 2))), LAT.heisenberg(LAT.chain_bonds(33)))
    if name == "chain63":
        return Case(ls.SpinBasis(63, 2, None, S(LAT.chain_symmetries(63, 7))), LAT.heisenberg(LAT.chain_bonds(63)))
    if name == "all_pairs25":  # 300 flip patterns x 150 elements: too large for whole states, prefixes of 25-bit states
        bonds = [(i, j) for i in range(25) for j in range(i)]
        return Case(ls.SpinBasis(25, 5, None, S(LAT.triangular_symmetries(5, 0, 0, 0))), LAT.heisenberg(bonds))
    if name == "square36":  # prefixes with spin inversion would be 1.6e7 rows: three particles instead
        return Case(ls.SpinBasis(36, 3, None, S(LAT.square_symmetries(6, 0, 0))),
                    LAT.heisenberg(LAT.square_bonds(6)) + LAT.heisenberg(LAT.square_bonds(6, diagonal=True), 0.5))
    if name == "all_pairs20_inversion":  # prefixes with spin inversion
        bonds = [(i, j) for i in range(20) for j in range(i)]
        b = ls.SpinBasis(20, 10, 1, S(LAT.chain_symmetries(20, 0, 0) + [ls.Symmetry([(3 * i) % 20 for i in range(20)], 0)]))
        return Case(b, LAT.heisenberg(bonds))
    if name == "flips":  # one to four flipped sites, no conserved number, several classes and a field
        e = ls.Expr("σˣ₀", sites=[[i] for i in range(10)]).scale(0.7)
        e = e + ls.Expr("σˣ₀ σˣ₁ σˣ₂", sites=[[i, (i + 1) % 10, (i + 2) % 10] for i in range(10)]).scale(-0.2)
        e = e + ls.Expr("σˣ₀ σʸ₁ σˣ₂ σʸ₃", sites=[[i, (i + 1) % 10, (i + 2) % 10, (i + 3) % 10] for i in range(10)])
        e = e + ls.Expr("σᶻ₀ σᶻ₁", sites=[list(b) for b in LAT.chain_bonds(10)]) + \
            ls.Expr("σᶻ₀", sites=[[i] for i in range(10)]).scale(0.4)
        return Case(ls.SpinBasis(10, None, None, S(LAT.chain_symmetries(10, 3))), e)
    if name == "diagonal":  # no off-diagonal terms at all
        return Case(ls.SpinBasis(12, 6, 1, S(LAT.chain_symmetries(12, 0))),
                    ls.Expr("σᶻ₀ σᶻ₁", sites=[list(b) for b in LAT.chain_bonds(12)]))
    if name == "one_row":
        return Case(ls.SpinBasis(12, 1, None, S(LAT.chain_symmetries(12, 0))), LAT.heisenberg(LAT.chain_bonds(12)))
    raise KeyError(name)


NAMES = ["chain9", "chain16_inversion", "chain32", "chain33", "chain63", "all_pairs25", "square36",
         "all_pairs20_inversion", "flips", "one_row", "diagonal"]


@pytest.fixture(scope="module")
def cases():
    out = {}
    for name in NAMES:
        out[name] = _case(name)
        out[name].basis.build(exact_norms=True)
    return out


def _check(y, expected, finite_scale=None):
    scale = np.linalg.norm(expected)
    assert np.linalg.norm(y - expected) <= RTOL * max(scale, 1e-300)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("k", [1, 2, 3, 5, 16, 19])
def test_columns_match_oracle(cases, name, k):
    import torch
    c = cases[name]
    states = c.basis.states
    D = len(states)
    rng = np.random.default_rng(3)
    x = rng.normal(size=(D, k)) + 1j * rng.normal(size=(D, k))
    y = c.op.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    yr = c.op.apply_device(torch.from_numpy(x.real.copy()).cuda()).cpu().numpy()
    for j in range(k):
        expected = c.oracle_matvec(states, np.ascontiguousarray(x[:, j]), complex_=True)
        _check(y[:, j], expected)
        real = c.oracle_matvec(states, np.ascontiguousarray(x[:, j].real))
        assert np.linalg.norm(yr[:, j] - real) <= RTOL * np.linalg.norm(expected)


def test_odd_leading_dimension_and_unaligned_real_columns(cases):
    import torch
    c = cases["chain16_inversion"]
    D = len(c.basis.states)
    x = np.random.default_rng(4).normal(size=(D, 7))
    big = torch.zeros((D, 7), dtype=torch.float64, device="cuda")
    big.copy_(torch.from_numpy(x))
    out = torch.full((D, 7), 7.0, dtype=torch.float64, device="cuda")
    lib = c.op._lib
    # columns 1 .. 5 of rows of 7: an odd leading dimension, 8-byte aligned only
    rc = lib.ls_gpu_matvec_f64(c.op._payload, 5, big.data_ptr() + 8, 7, out.data_ptr() + 8, 7, 0,
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    y = out.cpu().numpy()
    assert (y[:, 0] == 7.0).all() and (y[:, 6] == 7.0).all()
    for j in range(1, 6):
        _check(y[:, j], c.oracle_matvec(c.basis.states, np.ascontiguousarray(x[:, j])))


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_input_reaches_its_rows_only(cases, bad):
    import torch
    c = cases["chain16_inversion"]
    D = len(c.basis.states)
    j = D // 2
    unit = np.zeros(D, dtype=np.complex128)
    unit[j] = 1.0
    reached = c.oracle_matvec(c.basis.states, unit, complex_=True) != 0
    x = np.random.default_rng(5).normal(size=D) + 0j
    x[j] = bad
    y = c.op.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    reached[j] = True
    assert np.array_equal(~np.isfinite(y), reached)


@pytest.mark.parametrize("many", [False, True])
def test_alike_terms_of_several_couplings(many):
    """Couplings that share bonds: their alike terms are one element, summed per class (up to four
    classes) or per coupling (more).  Every coupling's product against the oracle's matvec of it."""
    import importlib
    import torch
    ag = importlib.import_module("lattice-symmetries_gb300.autograd")
    n = 7
    legs, rungs = LAT.ladder(n)
    parts = [LAT.heisenberg(legs), LAT.dm_z(legs, 0.6), LAT.heisenberg(rungs),
             LAT.heisenberg(rungs, 0.5) + LAT.dm_z(legs, 0.3) + LAT.heisenberg(legs, -0.7)]
    if many:  # five classes: both directions of the legs and of the second neighbours, and the rungs
        second = [(leg + i, leg + (i + 2) % n) for leg in (0, n) for i in range(n)]
        parts[2] = parts[2] + LAT.heisenberg(second, 0.2) + LAT.dm_z(second, 0.35)
    b = ls.SpinBasis(2 * n, n, None, ls.Symmetries(LAT.ladder_symmetries(n, 2)))
    b.build(exact_norms=True)
    pop = ag.ParametrizedOperator(b, parts, [0.4, 1.1, -0.7, 0.3])
    D = b.number_states
    rng = np.random.default_rng(8)
    g, x = (rng.normal(size=D) + 1j * rng.normal(size=D) for _ in range(2))
    out = pop.coupling_products(torch.from_numpy(g).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    y = pop.operator.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    total = np.zeros(D, dtype=np.complex128)
    for c, part in enumerate(parts):
        hx = Case(b, part).oracle_matvec(b.states, x, complex_=True)
        total += pop.theta[c] * hx
        # a sum of D products: FP64 rounding below D * 2^-53 * |g| |H x|
        assert abs(out[c] - np.vdot(g, hx)) <= RTOL * np.linalg.norm(g) * np.linalg.norm(hx)
    assert np.linalg.norm(y - total) <= RTOL * np.linalg.norm(total)
