"""The work this package is used for, as cases that can be timed and compared.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  basis, operator and vectors as a program has them before the call
    run(state)           one pass through the public entry points, and its outputs
    work(case)           the bytes and operations that one pass cannot do without
    exact(case, seed)    the outputs of run() by a plain torch restatement in 64 bits

Kinds of case:

    matvec    Operator.apply_device on device vectors: the inner loop of a GPU eigensolver or of a
              time evolution (one vector or a block, real or complex, H or H^dagger)
    host      Operator @ numpy vector: the call scipy's eigsh makes
    sectors   SectorBatch.run: one block product for all momentum / inversion sectors
    lanczos   lanczos_step on all sectors of a SectorBatch from a fixed orthonormal block
    grad      ParametrizedOperator.apply and its backward pass
    build     Basis.build: enumeration, state index and orbit norms of a new basis, and the place in it
              of a few thousand product states (Basis.state_info and Basis.index: how a program sets
              up a start vector)

Models: `chain` (XXZ, `n` sites), `square` and `triangular` (Heisenberg on an L x L torus, `n` =
L * L, next-nearest bonds of strength `j2` on the square), `ladder` (two legs, Dzyaloshinskii-Moriya
term along the legs), `hubbard` (spinful fermions on an L x L torus with lattice symmetries),
`free_chain` and `free_hubbard` (the same chains without any symmetry).
"""

import functools
import importlib
import math
from fractions import Fraction

import numpy as np
import torch

ls = importlib.import_module("lattice-symmetries_gb300")
lattices = importlib.import_module("lattice-symmetries_gb300.lattices")
autograd = importlib.import_module("lattice-symmetries_gb300.autograd")
lanczos = importlib.import_module("lattice-symmetries_gb300.lanczos")

DELTA, T, U, THETA = 1.5, 1.0, 8.0, (1.0, 0.7, 0.2)
LANCZOS_STEPS = 2
PRODUCT_STATES = 4096


def listed():
    return [
        # the smallest call: a 16-site chain in a test or a tutorial (257 states), where launches count
        dict(name="chain16_real", kind="matvec", model="chain", n=16, momentum=0, parity=0, inversion=1,
             complex=False, k=1, adjoint=False),
        # the 24-site Heisenberg chain driven from scipy: numpy vector in, numpy vector out
        dict(name="chain24_host", kind="host", model="chain", n=24, momentum=0, parity=0, inversion=1),
        # one complex vector on the 6x6 J1-J2 torus, (pi, pi) sector: the largest sector in use
        dict(name="square36_complex", kind="matvec", model="square", n=36, momentum=3, j2=0.5, inversion=1,
             complex=True, k=1, adjoint=False),
        # an odd number of sites, a ragged number of columns and H^dagger
        dict(name="triangular25_adjoint5", kind="matvec", model="triangular", n=25, inversion=0, complex=True, k=5,
             adjoint=True),
        # a block of 16 in a complex momentum sector of the 28-site XXZ chain
        dict(name="chain28_block16", kind="matvec", model="chain", n=28, momentum=3, parity=-1, inversion=1,
             complex=True, k=16, adjoint=False),
        # fermions with lattice symmetries: the 4x4 Hubbard model at 7 up + 7 down, 8 columns
        dict(name="hubbard16_block8", kind="matvec", model="hubbard", n=16, up=7, down=7, complex=True, k=8,
             adjoint=False),
        # no symmetries at all: the basis most first programs use
        dict(name="free_chain24_real", kind="matvec", model="free_chain", n=24, complex=False, k=1, adjoint=False),
        dict(name="free_hubbard12_block4", kind="matvec", model="free_hubbard", n=12, up=6, down=6, complex=True,
             k=4, adjoint=False),
        # all sectors of the 24-site XXZ chain in one product, 16 columns each
        dict(name="sectors24_block16", kind="sectors", model="chain", n=24, k=16),
        # the block eigensolver's step over all sectors: product, recurrence, orthonormalisation
        dict(name="lanczos22_block16", kind="lanczos", model="chain", n=22, k=16),
        # a training step: forward and backward through H(theta) x on the 28-site ladder
        dict(name="ladder28_grad", kind="grad", model="ladder", n=28),
        # a new basis: the 6x6 torus enumerated from scratch, product states located in it
        dict(name="build_square36", kind="build", model="square", n=36, momentum=3, j2=0.5, inversion=1),
    ]


def draw(rng):
    def sites(lo, hi):  # any number of sites; a spin chain's states grow as 2^n
        return rng.randint(lo, hi)

    def columns():
        return max(1, min(20, int(2 ** rng.uniform(0.0, 4.33))))

    def chain(lo, hi):
        n = sites(lo, hi)
        momentum = rng.choice([0, 0, n // 2 if n % 2 == 0 else 0, rng.randrange(n)])
        parity = rng.choice([-1, 0, 1]) if 2 * momentum % n == 0 else -1
        return dict(model="chain", n=n, momentum=momentum, parity=parity,
                    inversion=rng.choice([0, 1, -1]) if n % 2 == 0 else 0)

    def torus():
        model = rng.choice(["square", "triangular"])
        n = rng.choice([9, 16, 25]) if model == "triangular" else rng.choice([16, 25])
        case = dict(model=model, n=n, inversion=rng.choice([0, 1, -1]) if n % 2 == 0 else 0)
        if model == "square":
            case.update(momentum=rng.choice([0, 2]) if n == 16 else 0, j2=rng.choice([0.0, 0.5]))
        return case

    def with_vectors(case):
        real_only = case["model"] == "chain" and 2 * case["momentum"] % case["n"] != 0
        return dict(case, kind="matvec", complex=real_only or rng.random() < 0.6, k=columns(),
                    adjoint=rng.random() < 0.3)

    kind = rng.choice(["chain", "chain", "torus", "free_chain", "free_hubbard", "hubbard", "host", "sectors",
                       "lanczos", "grad", "build", "build"])
    if kind == "chain":
        return with_vectors(chain(12, 28))
    if kind == "torus":
        return with_vectors(torus())
    if kind == "free_chain":
        return with_vectors(dict(model="free_chain", n=sites(10, 25)))
    if kind == "free_hubbard":
        n = sites(5, 12)
        return with_vectors(dict(model="free_hubbard", n=n, up=rng.randint(n // 3, n // 2),
                                 down=rng.randint(n // 3, n // 2)))
    if kind == "hubbard":
        n = rng.choice([9, 16])
        return with_vectors(dict(model="hubbard", n=n, up=rng.randint(2, n // 2 - 1), down=rng.randint(2, n // 2 - 1)))
    if kind == "host":
        case = chain(14, 26)
        case["momentum"] = 0
        return dict(case, kind="host")
    if kind == "sectors":
        return dict(kind="sectors", model="chain", n=2 * sites(6, 12), k=columns())
    if kind == "lanczos":
        return dict(kind="lanczos", model="chain", n=2 * sites(8, 11), k=rng.choice([4, 8, 13, 16]))
    if kind == "grad":
        return dict(kind="grad", model="ladder", n=2 * sites(6, 14))
    return dict(chain(14, 30) if rng.random() < 0.5 else torus(), kind="build")


# ---- models -----------------------------------------------------------------------------------


def _weight(case):
    return case["n"] // 2


def _side(case):
    return math.isqrt(case["n"])


def _generators(case):
    """Symmetry generators of the package for this case (empty without symmetries)."""
    n = case["n"]
    if case["model"] == "chain":
        parity = case.get("parity", -1)
        return lattices.chain_symmetries(n, case["momentum"], parity if parity >= 0 else None)
    if case["model"] == "square":
        return lattices.square_symmetries(_side(case), case["momentum"], case["momentum"])
    if case["model"] == "triangular":
        return lattices.triangular_symmetries(_side(case), 0, 0, 0)
    if case["model"] == "ladder":
        return lattices.ladder_symmetries(n // 2, 0, 0)
    if case["model"] == "hubbard":
        return lattices.square_symmetries(_side(case), 0, 0)
    return []


def _basis(case):
    generators = _generators(case)
    symmetries = ls.Symmetries(generators) if generators else None
    if case["model"].endswith("hubbard"):
        return ls.SpinfulFermionBasis(case["n"], (case["up"], case["down"]), symmetries)
    return ls.SpinBasis(case["n"], _weight(case), case.get("inversion") or None, symmetries)


def _built(case):
    basis = _basis(case)
    # in complex momentum sectors states of zero norm are left out
    basis.build(exact_norms=case["model"] == "chain" and 2 * case["momentum"] % case["n"] != 0)
    return basis


def _expressions(case):
    """The couplings of H as expressions of the package."""
    n, model = case["n"], case["model"]
    if model in ("chain", "free_chain"):
        return [lattices.xxz(lattices.chain_bonds(n), 1.0, DELTA)]
    if model == "square":
        e = lattices.heisenberg(lattices.square_bonds(_side(case)))
        if case["j2"]:
            e = e + lattices.heisenberg(lattices.square_bonds(_side(case), diagonal=True), case["j2"])
        return [e]
    if model == "triangular":
        return [lattices.heisenberg(lattices.triangular_bonds(_side(case)))]
    if model == "ladder":
        legs, rungs = lattices.ladder(n // 2)
        return [lattices.heisenberg(legs), lattices.heisenberg(rungs), lattices.dm_z(legs)]
    bonds = lattices.square_bonds(_side(case)) if model == "hubbard" else lattices.chain_bonds(n)
    return [lattices.hubbard(bonds, T, U, n)]


def _sector_cases(case):
    """The chain's momenta times spin inversion as single-sector cases."""
    n = case["n"]
    return [dict(case, momentum=m, parity=-1, inversion=z) for m in range(n) for z in (1, -1)]


def _normal(shape, seed, complex_, salt=0):
    gen = torch.Generator(device=_device()).manual_seed(1000003 * int(seed) + salt)
    x = torch.randn(tuple(shape) + ((2,) if complex_ else ()), generator=gen, dtype=torch.float64, device=_device())
    return torch.view_as_complex(x) if complex_ else x


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _vectors(case, seed, states, salt=0):
    k = case.get("k", 1)
    shape = (states,) if k == 1 else (states, k)
    return _normal(shape, seed, case.get("complex", True), salt)


def _start_blocks(case, seed, sizes, rows):
    """One orthonormal [rows, k] block per sector, zero below the sector's states."""
    q = torch.zeros((len(sizes), rows, case["k"]), dtype=torch.complex128, device=_device())
    for s, d in enumerate(sizes):
        q[s, :d] = torch.linalg.qr(_normal((d, case["k"]), seed, True, s))[0]
    return q


# ---- preparation and one pass -------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "build":
        # random product states of the basis' weight: the w largest of n random numbers point up
        rng = np.random.default_rng(int(seed))
        up = np.argsort(rng.random((PRODUCT_STATES, case["n"])), axis=1)[:, :_weight(case)].astype(np.uint64)
        product = np.bitwise_or.reduce(np.uint64(1) << up, axis=1)
        return dict(kind=kind, case=case, symmetries=ls.Symmetries(_generators(case)), product=product)
    if kind in ("sectors", "lanczos"):
        operators = [ls.Operator(_built(c), _expressions(c)[0]) for c in _sector_cases(case)]
        batch = ls.SectorBatch(operators, k=case["k"])
        if kind == "sectors":
            for s in range(batch.number_sectors):
                batch.x(s).copy_(_normal((batch.sizes[s], case["k"]), seed, True, s))
            return dict(kind=kind, batch=batch)
        start = _start_blocks(case, seed, batch.sizes, batch.X.shape[1])
        small = torch.zeros((len(operators), case["k"], case["k"]), dtype=torch.complex128, device=start.device)
        return dict(kind=kind, batch=batch, start=start, previous=torch.zeros_like(start),
                    blocks=[torch.zeros_like(small) for _ in range(1 + 2 * LANCZOS_STEPS)])
    basis = _built(case)
    D = basis.number_states
    if kind == "grad":
        pop = autograd.ParametrizedOperator(basis, _expressions(case))
        return dict(kind=kind, pop=pop, theta=torch.tensor(THETA, dtype=torch.float64, requires_grad=True),
                    x=_normal((D,), seed, True).requires_grad_(True), v=_normal((D,), seed, True, 1))
    operator = ls.Operator(basis, _expressions(case)[0])
    if kind == "host":
        return dict(kind=kind, operator=operator, x=np.random.default_rng(int(seed)).standard_normal(D))
    x = _vectors(case, seed, D)
    return dict(kind=kind, operator=operator, x=x, y=torch.empty_like(x), adjoint=case["adjoint"])


def run(state):
    kind = state["kind"]
    if kind == "matvec":
        # as an iterative solver calls it: its own output buffer, errors checked once at the end
        return state["operator"].apply_device(state["x"], out=state["y"], adjoint=state["adjoint"], check=False)
    if kind == "host":
        return state["operator"] @ state["x"]
    if kind == "sectors":
        return state["batch"].run()
    if kind == "lanczos":
        batch, previous = state["batch"], state["previous"]
        b, out = state["blocks"][0], state["blocks"][1:]
        batch.X.copy_(state["start"])
        previous.zero_()
        b.zero_()
        for j in range(LANCZOS_STEPS):
            lanczos.lanczos_step(batch.run, batch.X, batch.Y, previous, b, out[2 * j], out[2 * j + 1])
        return dict(a=out[0::2], b=out[1::2], q=batch.X)
    if kind == "grad":
        state["theta"].grad = state["x"].grad = None
        y = state["pop"].apply(state["theta"], state["x"])
        loss = torch.vdot(state["v"], y).real
        loss.backward()
        return dict(y=y.detach(), theta=state["theta"].grad, x=state["x"].grad)
    case = state["case"]
    basis = ls.SpinBasis(case["n"], _weight(case), case.get("inversion") or None, state["symmetries"])
    basis.build(exact_norms=case["model"] == "chain" and 2 * case["momentum"] % case["n"] != 0)
    # the tensors keep the basis that owns the memory
    norms = torch.as_tensor(basis.device_norms(), device="cuda")
    states = torch.as_tensor(basis.device_states(), device="cuda").view(torch.int64)
    representatives, characters, _ = basis.state_info(state["product"])
    return dict(states=states, norms=norms, characters=characters, index=basis.index(representatives))


# ---- what a pass cannot do without --------------------------------------------------------------


def _group_order(case):
    n = case["n"]
    order = {"chain": n * (2 if case.get("parity", -1) >= 0 else 1), "square": 8 * n, "triangular": 6 * n,
             "ladder": n, "hubbard": 8 * n}.get(case["model"], 1)
    return order * (2 if case.get("inversion") else 1)


def _states(case):
    """About the number of representatives (the orbits of size |G| dominate)."""
    n = case["n"]
    if case["model"].endswith("hubbard"):
        full = math.comb(n, case["up"]) * math.comb(n, case["down"])
    else:
        full = math.comb(n, _weight(case))
    return max(1.0, full / _group_order(case))


def _row_elements(case):
    """Mean number of off-diagonal elements in a row: bonds whose two ends differ."""
    n = case["n"]

    def differ(w):
        return 2.0 * w * (n - w) / (n * (n - 1))

    bonds = {"chain": n, "free_chain": n, "square": 4 * n if case.get("j2") else 2 * n, "triangular": 3 * n,
             "ladder": 3 * n // 2, "hubbard": 2 * n, "free_hubbard": n}[case["model"]]
    if case["model"].endswith("hubbard"):
        return bonds * (differ(case["up"]) + differ(case["down"]))
    return bonds * differ(_weight(case))


def _is_real(case):
    return not (case["model"] == "ladder" or (case["model"] == "chain" and 2 * case["momentum"] % case["n"] != 0))


def work(case):
    kind = case["kind"]
    if kind == "build":
        return {"bytes": 16.0 * _states(case) + 32.0 * PRODUCT_STATES, "flops": 0.0}
    if kind in ("sectors", "lanczos"):
        parts = [work(dict(c, kind="matvec", complex=True)) for c in _sector_cases(case)]
        total = {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
        if kind == "sectors":
            return total
        # per step: four Gram products and three updates (five terms) of k x k on D x k blocks
        states = sum(_states(c) for c in _sector_cases(case))
        dense = 8.0 * states * case["k"] ** 2 * 9
        return {"bytes": total["bytes"] * LANCZOS_STEPS, "flops": (total["flops"] + dense) * LANCZOS_STEPS}
    D, row, k = _states(case), _row_elements(case), case.get("k", 1)
    complex_ = kind == "grad" or case.get("complex", False)
    scalar = 16.0 if complex_ else 8.0
    stored = 16.0 if _group_order(case) > 1 else 0.0
    per_element = (4.0 if _is_real(case) else 8.0) if complex_ else 2.0
    one = {"bytes": D * (stored + 2 * scalar * k), "flops": D * (row + 1) * k * per_element}
    if kind == "grad":  # forward, adjoint, and one inner product per coupling
        return {"bytes": D * (stored + 5 * scalar), "flops": 3.0 * one["flops"]}
    return one


# ---- the same outputs in plain torch, 64 bits ---------------------------------------------------


@functools.lru_cache(maxsize=None)
def _byte_tables(perm, device):
    """lut[c][v]: image of the byte v at bits 8c.. under g (bit i of g.x is bit perm[i] of x)."""
    n = len(perm)
    chunks = (n + 7) // 8
    lut = np.zeros((chunks, 256), dtype=np.int64)
    v = np.arange(256, dtype=np.int64)
    for i, p in enumerate(perm):
        lut[p // 8] |= ((v >> (p % 8)) & 1) << i
    return torch.from_numpy(lut).to(device)


def _permute(perm, x):
    lut = _byte_tables(perm, str(x.device))
    y = lut[0][x & 255]
    for c in range(1, lut.shape[0]):
        y = y | lut[c][(x >> (8 * c)) & 255]
    return y


def _popcount(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    x = x + (x >> 8)
    x = x + (x >> 16)
    return (x + (x >> 32)) & 127


class _Group:
    """The closed group of (permutation of the bits, character), with spin inversion."""

    def __init__(self, case):
        n = case["n"]
        generators = [(tuple(g.permutation), Fraction(g.phase)) for g in _generators(case)]
        identity = tuple(range(n))
        found, queue = {identity: Fraction(0)}, [identity]
        while queue:
            a = queue.pop()
            for p, phase in generators:
                b = tuple(p[i] for i in a)
                if b not in found:
                    found[b] = (found[a] + phase) % 1
                    queue.append(b)
        self.fermions = case["model"].endswith("hubbard")
        self.inversion = case.get("inversion") or 0
        self.bits = 2 * n if self.fermions else n
        self.elements = []
        for p, phase in sorted(found.items()):
            perm = p + tuple(n + i for i in p) if self.fermions else p
            chi = complex(math.cos(-2 * math.pi * phase), math.sin(-2 * math.pi * phase))
            self.elements.append((perm, 0, chi))
            if self.inversion:
                self.elements.append((perm, (1 << n) - 1, chi * self.inversion))

    def image(self, element, x):
        return _permute(element[0], x) ^ element[1]

    def sign(self, element, x):
        """Sign of the permutation that the element induces on the occupied orbitals."""
        if not self.fermions:
            return torch.ones(x.shape, dtype=torch.float64, device=x.device)
        to = {p: i for i, p in enumerate(element[0])}
        odd = torch.zeros_like(x)
        for k in range(self.bits):
            passed = sum(1 << l for l in range(k) if to[l] > to[k])
            if passed:
                odd += ((x >> k) & 1) * _popcount(x & passed)
        return 1.0 - 2.0 * (odd & 1).double()

    def representatives(self, x):
        """The states of x that are orbit minima with a non-zero norm, and the norms."""
        for e in self.elements:
            x = x[self.image(e, x) >= x]
        total = torch.zeros(x.shape, dtype=torch.float64, device=x.device)
        for e in self.elements:
            at = torch.nonzero(self.image(e, x) == x)[:, 0]
            total[at] += e[2].real * self.sign(e, x[at])
        keep = total > 0.5
        return x[keep], torch.sqrt(total[keep] / len(self.elements))

    def project(self, x):
        """(representative, conj(character) with the fermionic sign) of generated states."""
        best, which = x.clone(), torch.zeros_like(x)
        for number, e in enumerate(self.elements):
            y = self.image(e, x)
            better = y < best
            best = torch.where(better, y, best)
            which[better] = number
        factor = torch.ones(x.shape, dtype=torch.complex128, device=x.device)
        for number, e in enumerate(self.elements):
            at = torch.nonzero(which == number)[:, 0]
            factor[at] = e[2].conjugate() * self.sign(e, x[at]).to(torch.complex128)
        return best, factor


@functools.lru_cache(maxsize=2)
def _fixed_weight(n, w, device):
    parts = []
    for begin in range(0, 1 << n, 1 << 24):
        x = torch.arange(begin, min(1 << n, begin + (1 << 24)), dtype=torch.int64, device=device)
        parts.append(x[_popcount(x) == w])
    return torch.cat(parts)


def _couplings(case):
    """[(bonds, amplitude, diagonal)]: <..1_i..0_j..|H|..0_i..1_j..> and the coefficient of
    sigma^z sigma^z, per coupling."""
    n, model = case["n"], case["model"]
    if model in ("chain", "free_chain"):
        return [(lattices.chain_bonds(n), 2.0, DELTA)]
    if model == "square":
        both = [(lattices.square_bonds(_side(case)), 2.0, 1.0)]
        if case["j2"]:
            both.append((lattices.square_bonds(_side(case), diagonal=True), 2.0 * case["j2"], case["j2"]))
        return both
    if model == "triangular":
        return [(lattices.triangular_bonds(_side(case)), 2.0, 1.0)]
    legs, rungs = lattices.ladder(n // 2)
    return [(legs, 2.0, 1.0), (rungs, 2.0, 1.0), (legs, 0.5j, 0.0)]


class _Exact:
    """One sector: representatives, norms and products with each coupling of H."""

    def __init__(self, case):
        self.case, self.group = case, _Group(case)
        n, device = case["n"], _device()
        if self.group.fermions:
            up, down = _fixed_weight(n, case["up"], device), _fixed_weight(n, case["down"], device)
            step = max(1, (1 << 25) // len(up))
            found = [self.group.representatives(((d[:, None] << n) | up[None, :]).reshape(-1))
                     for d in torch.split(down, step)]
        else:
            found = [self.group.representatives(s) for s in torch.split(_fixed_weight(n, _weight(case), device), 1 << 25)]
        self.states = torch.cat([f[0] for f in found])
        self.norms = torch.cat([f[1] for f in found])
        self.terms = None

    def _elements(self, parts):
        """Rows, columns and values of all elements, from (rows, flipped bits, amplitudes) per bond."""
        rows, flips, amplitude = (torch.cat(v) for v in zip(*parts))
        out = []
        for r, f, c in zip(*(torch.split(v, 1 << 25) for v in (rows, flips, amplitude))):
            rep, factor = self.group.project(self.states[r] ^ f)
            column = torch.searchsorted(self.states, rep).clamp_max(len(self.states) - 1)
            found = self.states[column] == rep  # else a state of zero norm
            value = c * factor * self.norms[column] / self.norms[r]
            out.append((r[found], column[found], value[found]))
        return [torch.cat(v) for v in zip(*out)]

    def couplings(self):
        """[((rows, columns, values), diagonal)] per coupling."""
        if self.terms is not None:
            return self.terms
        a, n = self.states, self.case["n"]
        everything, out = torch.arange(len(a), device=a.device), []

        def bond(i, j, amplitude):
            rows = everything[((a >> i) & 1) != ((a >> j) & 1)]
            return rows, torch.full_like(rows, (1 << i) | (1 << j)), amplitude(a[rows]).to(torch.complex128)

        if self.group.fermions:
            bonds = (lattices.square_bonds(_side(self.case)) if self.case["model"] == "hubbard"
                     else lattices.chain_bonds(n))
            parts = []
            for base in (0, n):
                for i, j in bonds:
                    i, j = sorted((i + base, j + base))
                    between = ((1 << j) - 1) ^ ((1 << (i + 1)) - 1)
                    parts.append(bond(i, j, lambda s: T * (2.0 * (_popcount(s & between) & 1).double() - 1.0)))
            out.append((self._elements(parts), U * _popcount(a & (a >> n) & ((1 << n) - 1)).double()))
        else:
            for bonds, amplitude, zz in _couplings(self.case):
                c = complex(amplitude)
                parts, diagonal = [], torch.zeros(len(a), dtype=torch.float64, device=a.device)
                for i, j in bonds:
                    parts.append(bond(i, j, lambda s: torch.where((s >> i) & 1 == 1, c, c.conjugate())))
                    diagonal += zz * (1.0 - 2.0 * (((a >> i) ^ (a >> j)) & 1).double())
                out.append((self._elements(parts), diagonal))
        self.terms = out
        return out

    def product(self, x, theta=None, coupling=None):
        """H x (or one coupling's share of it) for complex [D] or [D, k]."""
        total = torch.zeros_like(x)
        for c, ((rows, columns, values), diagonal) in enumerate(self.couplings()):
            if coupling is not None and c != coupling:
                continue
            y = x * (diagonal if x.dim() == 1 else diagonal[:, None])
            for r, j, v in zip(*(torch.split(t, 1 << 23) for t in (rows, columns, values))):
                y.index_add_(0, r, x[j] * (v if x.dim() == 1 else v[:, None]))
            total += y * (1.0 if theta is None else theta[c])
        return total


def _lanczos_exact(sectors, start):
    """The coefficients and the last block of plain block Lanczos, every block kept orthonormal by
    Householder QR (the triangular factors with positive diagonals)."""
    a_out = [[] for _ in range(LANCZOS_STEPS)]
    b_out = [[] for _ in range(LANCZOS_STEPS)]
    last = torch.zeros_like(start)
    for s, sector in enumerate(sectors):
        d = len(sector.states)
        q, previous, b = start[s, :d], None, None
        for j in range(LANCZOS_STEPS):
            w = sector.product(q)
            a = q.mH @ w
            w = w - q @ a - (previous @ b.mH if previous is not None else 0.0)
            w = w - q @ (q.mH @ w)
            previous = q
            q, r = torch.linalg.qr(w)
            phase = torch.diagonal(r) / torch.diagonal(r).abs()
            q, b = q * phase, phase.conj()[:, None] * r
            a_out[j].append(0.5 * (a + a.mH))
            b_out[j].append(b)
        last[s, :d] = q
    return dict(a=[torch.stack(v) for v in a_out], b=[torch.stack(v) for v in b_out], q=last)


def exact(case, seed):
    kind = case["kind"]
    if case["model"] == "square" and case["n"] == 36:
        return None  # 9e9 states: too long to go through one by one
    if kind in ("sectors", "lanczos"):
        sectors = [_Exact(c) for c in _sector_cases(case)]
        sizes = [len(e.states) for e in sectors]
        rows = (max(max(sizes), 1) + 255) // 256 * 256
        if kind == "lanczos":
            return _lanczos_exact(sectors, _start_blocks(case, seed, sizes, rows))
        y = torch.zeros((len(sectors), rows, case["k"]), dtype=torch.complex128, device=_device())
        for s, sector in enumerate(sectors):
            y[s, :sizes[s]] = sector.product(_normal((sizes[s], case["k"]), seed, True, s))
        return y
    sector = _Exact(case)
    D = len(sector.states)
    if kind == "build":
        return dict(states=None, norms=sector.norms, characters=None, index=None)
    if kind == "host":
        x = torch.from_numpy(np.random.default_rng(int(seed)).standard_normal(D)).to(_device())
        return sector.product(x.to(torch.complex128)).real.cpu().numpy()
    if kind == "grad":
        x, v = _normal((D,), seed, True), _normal((D,), seed, True, 1)
        theta = [torch.vdot(v, sector.product(x, coupling=c)).real for c in range(len(THETA))]
        return dict(y=sector.product(x, THETA), theta=torch.stack(theta).cpu(), x=sector.product(v, THETA))
    x = _vectors(case, seed, D)
    y = sector.product(x.to(torch.complex128))  # H is Hermitian: the adjoint product is the same
    return y if case["complex"] else y.real.contiguous()
