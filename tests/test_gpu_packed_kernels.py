"""The kernels with a warp per row, which remain for tables beyond the lane-per-element ones', for few rows and
for counting, on every number of slots per lane.  They are reached on purpose: a diagonal term on a site
beyond the basis (a constant, or nothing for fermions) gets no lane-per-element tables, and neither do
more than 64 distinct coefficients.

Tolerance: rows sum at most a few hundred products, FP64 rounding stays below 3e-14 relative L2; 1e-12
is the bound of the parity tests."""

import importlib

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-12
ag = importlib.import_module("lattice-symmetries_gb300.autograd")


def beyond(n):
    return ls.Expr("σᶻ₀", sites=[[n]]).scale(0.3)


def spins(n, h, inversion, symmetries, expr):
    return Case(ls.SpinBasis(n, h, inversion, ls.Symmetries(symmetries)), expr + beyond(n))


def chain(n, momentum, inversion=None, h=None):
    return spins(n, n // 2 if h is None else h, inversion, LAT.chain_symmetries(n, momentum), LAT.xxz(LAT.chain_bonds(n), 1.0, 0.7))


CASES = {  # slots per lane
    "chain14_complex": (lambda: chain(14, 3), 1),
    "chain14_inversion": (lambda: chain(14, 7, -1), 1),
    "chain33": (lambda: chain(33, 2, None, 3), 2),
    "chain36_inversion_free": (lambda: chain(36, 0, None, 4), 2),
    "square3": (lambda: spins(9, 4, None, LAT.square_symmetries(3, 0, 0), LAT.heisenberg(LAT.square_bonds(3))), 3),
    "square4": (lambda: spins(16, 8, -1, LAT.square_symmetries(4, 2, 2), LAT.heisenberg(LAT.square_bonds(4))), 4),
    "triangular4": (lambda: spins(16, 8, 1, LAT.triangular_symmetries(4, 0, 0, 0, 0),
                                  LAT.heisenberg(LAT.triangular_bonds(4))), 6),
    "square5": (lambda: spins(25, 5, None, LAT.square_symmetries(5, 0, 0), LAT.heisenberg(LAT.square_bonds(5))), 9),
    "hypercube": (lambda: spins(16, 6, None, LAT.hypercube_symmetries(4), LAT.heisenberg(LAT.hypercube_bonds(4))), 12),
    "triangular6": (lambda: spins(36, 4, None, LAT.triangular_symmetries(6, 0, 0, 0, 0),
                                  LAT.heisenberg(LAT.triangular_bonds(6))), 16),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_every_number_of_slots(name):
    import torch
    make, slots = CASES[name]
    c = make()
    c.basis.build(exact_norms=True)
    states = np.array(c.basis.states)
    D = len(states)
    rng = np.random.default_rng(12)
    for k, complex_ in [(1, True), (4, True), (8, True), (16, True), (13, True), (1, False), (2, False), (4, False),
                        (8, False), (16, False)]:
        assert c.op.kernel_route(k, complex_) == ("packed", slots)
        x = rng.normal(size=(D, k)) + (1j * rng.normal(size=(D, k)) if complex_ else 0)
        xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        y, ya = c.op.apply_device(xd).cpu().numpy(), c.op.apply_device(xd, adjoint=True).cpu().numpy()
        for j in {0, k // 2, k - 1}:
            expected = c.oracle_matvec(states, np.ascontiguousarray(x[:, j]), complex_=complex_)
            scale = RTOL * np.linalg.norm(expected)
            if complex_:
                assert np.linalg.norm(y[:, j] - expected) <= scale
                assert np.linalg.norm(ya[:, j] - expected) <= scale
            else:  # the real part of the elements
                full = c.oracle_matvec(states, x[:, j] + 0j, complex_=True)
                assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(full)


@pytest.mark.parametrize("n,up,slots", [(9, 2, 3), (16, 2, 4)])
def test_fermions(n, up, slots):
    """Against the lane-per-element kernels, which run the same operator without the stray term."""
    import torch
    L = int(round(n ** 0.5))
    b = ls.SpinfulFermionBasis(n, (up, up + 1), ls.Symmetries(LAT.square_symmetries(L, 0, 0)))
    b.build()
    H = LAT.hubbard(LAT.square_bonds(L), 1.0, 4.0)
    op, other = ls.Operator(b, H + ls.Expr("n₀↓", sites=[[n]])), ls.Operator(b, H)
    rng = np.random.default_rng(13)
    for k in (1, 4, 8, 16):
        assert op.kernel_route(k, True) == ("packed", slots)
        x = torch.from_numpy(rng.normal(size=(b.number_states, k)) + 1j * rng.normal(size=(b.number_states, k))).cuda()
        y = op.apply_device(x)
        for j in range(0, k, 3):
            expected = other.apply_device(x[:, j].contiguous())
            assert other.kernel_route(1, True)[0] == "rows"
            assert float((y[:, j] - expected).norm()) <= RTOL * float(expected.norm())


def test_kernel_without_shared_tables():
    import torch
    c = chain(60, 7, None, 2)
    c.basis.build(exact_norms=True)
    states = np.array(c.basis.states)
    assert c.op.kernel_route(3, True) == ("fallback", 2)
    x = np.random.default_rng(14).normal(size=(len(states), 3)) + 0.5j
    y = c.op.apply_device(torch.from_numpy(x).cuda()).cpu().numpy()
    for j in range(3):
        expected = c.oracle_matvec(states, np.ascontiguousarray(x[:, j]), complex_=True)
        assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(expected)


def random_pairs(n, scale=1.0):
    """XXZ on all pairs with a coupling per orbit of the reflection: more than 64 coefficients."""
    rng, e, J = np.random.default_rng(15), None, {}
    for i in range(n):
        for j in range(i):
            key = min((j, i), (n - 1 - i, n - 1 - j))
            if key not in J:
                J[key] = scale * float(rng.uniform(0.2, 1.0))
            t = LAT.xxz([(j, i)], J[key], 0.6)
            e = t if e is None else e + t
    assert len(J) > 64
    return e


def mirrored(n, sector, h):
    return ls.SpinBasis(n, h, None, ls.Symmetries([ls.Symmetry(list(range(n - 1, -1, -1)), sector)]))


def test_many_coefficients_in_plain_and_batched_products():
    n, H = 18, random_pairs(18)
    cases = [Case(mirrored(n, sector, 4), H) for sector in (0, 1)]
    for c in cases:
        c.basis.build(exact_norms=True)
        assert c.op.kernel_route(16, True) == ("packed", 1)
    for k in (1, 4, 8, 16, 21):
        batch = ls.SectorBatch([c.op for c in cases], k=k)
        assert batch.batched
        rng = np.random.default_rng(k)
        import torch
        xs = []
        for s, c in enumerate(cases):
            x = rng.normal(size=(c.basis.number_states, k)) + 1j * rng.normal(size=(c.basis.number_states, k))
            batch.x(s).copy_(torch.from_numpy(x))
            xs.append(x)
        batch.run(check=True)
        for s, c in enumerate(cases):
            y = batch.y(s).cpu().numpy()
            plain = c.op.apply_device(torch.from_numpy(xs[s]).cuda()).cpu().numpy()
            states = np.array(c.basis.states)
            for j in {0, k - 1}:
                expected = c.oracle_matvec(states, np.ascontiguousarray(xs[s][:, j]), complex_=True)
                assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(expected)
                assert np.linalg.norm(plain[:, j] - expected) <= RTOL * np.linalg.norm(expected)


@pytest.mark.parametrize("inversion", [None, 1])
@pytest.mark.parametrize("n,momentum,parity", [(14, 3, None), (18, 0, 0), (20, 5, None)])
def test_batched_products(n, momentum, parity, inversion):
    """Sector batches of one and two slots per lane, real and complex sectors together."""
    import torch
    cases = [spins(n, 4 if inversion is None else n // 2, inversion, LAT.chain_symmetries(n, m, p),
                   LAT.xxz(LAT.chain_bonds(n), 1.0, 0.7))
             for m, p in ((0, parity), (momentum if parity is None else n // 2, parity))]
    for c in cases:
        c.basis.build(exact_norms=True)
    for k in (1, 4, 13):
        batch = ls.SectorBatch([c.op for c in cases], k=k)
        assert batch.batched
        rng = np.random.default_rng(k)
        xs = []
        for s, c in enumerate(cases):
            xs.append(rng.normal(size=(c.basis.number_states, k)) + 1j * rng.normal(size=(c.basis.number_states, k)))
            batch.x(s).copy_(torch.from_numpy(xs[s]))
        batch.run(check=True)
        for s, c in enumerate(cases):
            y, states = batch.y(s).cpu().numpy(), np.array(c.basis.states)
            for j in {0, k - 1}:
                expected = c.oracle_matvec(states, np.ascontiguousarray(xs[s][:, j]), complex_=True)
                assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(expected)


def coupling_case(name):
    if name == "stray":  # every coupling with a term beyond the basis, 16 elements and inversion
        b = ls.SpinBasis(16, 8, 1, ls.Symmetries(LAT.chain_symmetries(16, 8)))
        return b, [LAT.heisenberg(LAT.chain_bonds(16)), LAT.xxz(LAT.chain_bonds(16), 0.3, 2.0) + beyond(16)]
    if name == "stray128":
        b = ls.SpinBasis(16, 6, None, ls.Symmetries(LAT.square_symmetries(4, 0, 0)))
        return b, [LAT.heisenberg(LAT.square_bonds(4)), LAT.heisenberg(LAT.square_bonds(4, diagonal=True)), beyond(16)]
    return mirrored(18, 1, 4), [random_pairs(18), random_pairs(18, -0.4)]


@pytest.mark.parametrize("name", ["stray", "stray128", "many"])
def test_coupling_products(name):
    import torch
    b, parts = coupling_case(name)
    b.build(exact_norms=True)
    pop = ag.ParametrizedOperator(b, parts)
    assert pop.generator.kernel_route(16, True)[0] == "packed"
    D = b.number_states
    rng = np.random.default_rng(16)
    g, x = (rng.normal(size=D) + 1j * rng.normal(size=D) for _ in range(2))
    out = pop.coupling_products(torch.from_numpy(g).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    for c, part in enumerate(parts):
        hx = Case(b, part).oracle_matvec(np.array(b.states), x, complex_=True)
        assert abs(out[c] - np.vdot(g, hx)) <= RTOL * np.linalg.norm(g) * np.linalg.norm(hx)
