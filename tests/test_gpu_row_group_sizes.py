"""Sector batches and coupling products of enough rows for a lane per element (more than 16 and 8 rows per SM
of a 152-SM device; fewer keep a warp per row), against the CPU oracle.

Tolerance: rows sum at most a few hundred products, FP64 rounding stays below 3e-14 relative L2; 1e-12
is the bound of the parity tests."""

import importlib

import numpy as np
import pytest

from ls_helpers import LAT, Case, ls

pytestmark = pytest.mark.gpu
RTOL = 1e-12
ag = importlib.import_module("lattice-symmetries_gb300.autograd")


@pytest.mark.parametrize("n,h,inversions,k", [(16, 8, (1, -1), 1), (16, 8, (1, -1), 4), (16, 8, (1, -1), 16),
                                              (17, 7, (None,), 1), (17, 7, (None,), 5), (17, 7, (None,), 18),
                                              (33, 4, (None,), 1), (33, 4, (None,), 8)])
def test_sector_batches(n, h, inversions, k):
    import torch
    H = LAT.xxz(LAT.chain_bonds(n), 1.0, 1.5)
    momenta = range(n) if n < 30 else (0, 1, 5)
    cases = [Case(ls.SpinBasis(n, h, z, ls.Symmetries(LAT.chain_symmetries(n, m))), H) for m in momenta for z in inversions]
    for c in cases:
        c.basis.build(exact_norms=True)
    batch = ls.SectorBatch([c.op for c in cases], k=k)
    assert batch.batched and sum(batch.sizes) > 16 * 152
    rng = np.random.default_rng(k)
    xs = []
    for s, D in enumerate(batch.sizes):
        xs.append(rng.normal(size=(D, k)) + 1j * rng.normal(size=(D, k)))
        batch.x(s).copy_(torch.from_numpy(xs[s]))
    batch.run(check=True)
    for s, c in enumerate(cases):
        y, states = batch.y(s).cpu().numpy(), np.array(c.basis.states)
        for j in {0, k - 1}:
            expected = c.oracle_matvec(states, np.ascontiguousarray(xs[s][:, j]), complex_=True)
            assert np.linalg.norm(y[:, j] - expected) <= RTOL * np.linalg.norm(expected)


def coupling_case(name):
    if name.startswith("ladder"):  # alike terms of several couplings: at most four classes, or more
        n = 9
        legs, rungs = LAT.ladder(n)
        parts = [LAT.heisenberg(legs), LAT.dm_z(legs, 0.6), LAT.heisenberg(rungs),
                 LAT.heisenberg(rungs, 0.5) + LAT.dm_z(legs, 0.3) + LAT.heisenberg(legs, -0.7)]
        if name == "ladder_many":
            second = [(leg + i, leg + (i + 2) % n) for leg in (0, n) for i in range(n)]
            parts[2] = parts[2] + LAT.heisenberg(second, 0.2) + LAT.dm_z(second, 0.35)
        return ls.SpinBasis(2 * n, n, None, ls.Symmetries(LAT.ladder_symmetries(n, 2))), parts
    if name == "square5":  # translations of 25 sites, bits of planes or whole states
        return (ls.SpinBasis(25, 6, None, ls.Symmetries(LAT.square_symmetries(5, 0, 0, False))),
                [LAT.heisenberg(LAT.square_bonds(5)), LAT.heisenberg(LAT.square_bonds(5, diagonal=True))])
    if name == "inversion":
        return (ls.SpinBasis(18, 9, -1, ls.Symmetries(LAT.chain_symmetries(18, 9))),
                [LAT.xxz(LAT.chain_bonds(18), 1.0, 0.0), LAT.xxz(LAT.chain_bonds(18), 0.0, 1.0)])
    return (ls.SpinBasis(36, 4, None, ls.Symmetries(LAT.square_symmetries(6, 0, 0, False))),  # wider than 32 bits
            [LAT.heisenberg(LAT.square_bonds(6)), LAT.heisenberg(LAT.square_bonds(6, diagonal=True))])


@pytest.mark.parametrize("name", ["ladder", "ladder_many", "square5", "inversion", "square6"])
def test_coupling_products(name):
    import torch
    b, parts = coupling_case(name)
    b.build(exact_norms=True)
    D = b.number_states
    assert D > 8 * 152
    pop = ag.ParametrizedOperator(b, parts)
    rng = np.random.default_rng(21)
    g, x = (rng.normal(size=D) + 1j * rng.normal(size=D) for _ in range(2))
    out = pop.coupling_products(torch.from_numpy(g).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    states = np.array(b.states)
    for c, part in enumerate(parts):
        hx = Case(b, part).oracle_matvec(states, x, complex_=True)
        # a sum of D products: FP64 rounding below D * 2^-53 * |g| |H x|
        assert abs(out[c] - np.vdot(g, hx)) <= RTOL * np.linalg.norm(g) * np.linalg.norm(hx)
