"""The work a user of this framework has it do, as cases that can be timed and checked.

Each case is one call (or one short chain of calls) through the public entry points: the Hamiltonian apply
``hamiltonian.dot``, the evolutions ``ExpmMultiplyParallel.dot``, ``MultiSectorExpm.evolve`` and ``hamiltonian.evolve``,
``lanczos_full`` with and without reorthogonalisation, the construction of a symmetry sector with its Hamiltonian, and
the matrix-free ``quantum_LinearOperator.dot``.  Models and sizes are those of the benchmark's configurations and the
tests: XXZ and J1-J2 Heisenberg chains, the mixed-field (and driven) Ising chain and the 4 x 4 Hubbard lattice, from
sectors of a few hundred states, where launches and latency count, to the 4.7 million states of the L = 32 chain.

``exact`` forms the same sector matrices and results with plain torch in 64 bits, from the basis conventions alone:
site i is bit N-1-i, representatives are the largest orbit element in descending order, and the element from ket i to
bra j of a coupling J is J me chi sign sqrt(n_j / n_i).
"""
import math

import numpy as np
import torch

from quspin_gb300 import (hamiltonian, quantum_LinearOperator, spin_basis_general, spinful_fermion_basis_general)
from quspin_gb300.tools import ExpmMultiplyParallel, MultiSectorExpm, lanczos_full

DEV = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64, "complex64": torch.complex64,
          "complex128": torch.complex128}


def listed():
    return [
        # One apply in a sector small enough that launches and host work are all of it: an iterative solver of the
        # user's own over the smallest configuration (XXZ, L = 20).
        dict(name="apply_small", kind="apply", model="xxz", L=20, sym="kp", k=0, dtype="float64", vec="complex128", nvec=1),
        # The apply at scale, real matrix and complex state: a Krylov or Chebyshev loop on a large chain.
        dict(name="apply_large", kind="apply", model="j1j2", L=30, sym="kpz", k=0, dtype="float64", vec="complex128", nvec=1),
        # Several states through a complex momentum sector at once: typicality averages, block solvers.
        dict(name="apply_block", kind="apply", model="ising", L=20, sym="k", k=3, dtype="complex128", vec="complex128", nvec=8),
        # Single precision, which users choose to halve the memory: fermions on the square lattice.
        dict(name="apply_single", kind="apply", model="hubbard", L=16, sym="kxky", k=0, nup=4, ndown=4, dtype="complex64", vec="complex64", nvec=1),
        # A time step of a small system, repeated by the thousand in a user's loop.
        dict(name="expm_small", kind="expm", model="xxz", L=20, sym="kp", k=0, dtype="float64", nvec=1, t=1.0),
        # One long evolution of the largest configuration (J1-J2, L = 32, t = 5): the headline workload.
        dict(name="expm_large", kind="expm", model="j1j2", L=32, sym="kpz", k=0, dtype="float64", nvec=1, t=5.0),
        # Eight states in every momentum sector of the mixed-field Ising chain, evolved together.
        dict(name="expm_sectors", kind="sectors", model="ising", L=16, nvec=8, t=1.0),
        # Ground-state Lanczos with the reference's plain recurrence.
        dict(name="lanczos_plain", kind="lanczos", model="xxz", L=26, sym="kp", k=0, dtype="float64", m=30, reorth=False),
        # Lanczos with full reorthogonalisation of a complex momentum sector: excited states.
        dict(name="lanczos_reorth", kind="lanczos", model="j1j2", L=26, sym="k", k=3, dtype="complex128", m=60, reorth=True),
        # A new sector and its Hamiltonian: the first thing every script does, once per sector and size.
        dict(name="build_sector", kind="build", model="j1j2", L=28, sym="kpz", k=0, dtype="float64"),
        # The matrix-free apply, for sectors whose matrix a user does not want to store.
        dict(name="matrix_free", kind="free", model="j1j2", L=26, sym="kpz", k=0, dtype="float64", nvec=1),
        # A driven chain through the adaptive integrator, static and time-dependent parts.
        dict(name="driven_evolve", kind="driven", model="driven", L=20, sym="kp", k=0, dtype="float64", nvec=1, t=0.5),
    ]


def draw(rng):
    kind = rng.choice(["apply", "apply", "expm", "expm", "sectors", "lanczos", "lanczos", "build", "free", "driven"])
    if kind == "sectors":
        return dict(kind=kind, model="ising", L=rng.choice([8, 10, 12, 14, 16]), nvec=rng.choice([1, 2, 3, 5, 8]), t=round(rng.uniform(0.2, 1.0), 3))
    if kind == "driven":
        return dict(kind=kind, model="driven", L=rng.randint(10, 20), sym="kp", k=0, dtype="float64", nvec=rng.choice([1, 1, 2, 5]), t=round(rng.uniform(0.1, 0.5), 3))
    case = dict(kind=kind, **_draw_sector(rng))
    real = case["dtype"] in ("float32", "float64")
    if kind == "apply":
        case["nvec"] = rng.choice([1, 1, 1, 2, 3, 4, 8, 13])
        if rng.random() < 0.25:
            case["dtype"] = case["vec"] = "float32" if real else "complex64"
        else:
            case["vec"] = rng.choice(["float64", "complex128", "complex128"]) if real else "complex128"
    elif kind == "expm":
        case.update(nvec=rng.choice([1, 1, 1, 2, 4, 7]), t=round(10.0 ** rng.uniform(-1.3, 0.3), 3))
    elif kind == "lanczos":
        case["reorth"] = rng.random() < 0.5
        # without reorthogonalisation a longer run in a small sector amplifies rounding until the vectors say nothing
        case["m"] = max(6, min(rng.randint(10, 60 if case["reorth"] else 20), int(_size(case)[0]) // 8))
    elif kind == "free":
        case["nvec"] = rng.choice([1, 1, 2, 3])
    return case


def _draw_sector(rng):
    """A sector of one of the models, from a few hundred states to about 1.3 million."""
    model = rng.choice(["xxz", "j1j2", "j1j2", "ising", "hubbard"])
    if model == "hubbard":
        nup, ndown = rng.choice([(2, 2), (3, 2), (3, 3), (4, 3), (4, 4), (5, 4)])
        return dict(model=model, L=16, sym="kxky", k=0, nup=nup, ndown=ndown, dtype="complex128")
    if model == "ising":
        L, sym = rng.randint(12, 23), rng.choice(["kp", "k"])
    else:
        sym = rng.choice(["kp", "kpz", "k"]) if model == "xxz" else rng.choice(["kpz", "kpz", "k"])
        L = 2 * rng.randint(7, {"kpz": 15, "kp": 13, "k": 13}[sym])
    if sym == "k":
        return dict(model=model, L=L, sym=sym, k=rng.randint(1, (L - 1) // 2), dtype="complex128")
    return dict(model=model, L=L, sym=sym, k=0, dtype="float64")


# -- models: bonds and symmetry maps --------------------------------------------------------------------------------


def _drive(t, h0, A, w):
    return h0 + A * math.cos(w * t)


DRIVE = (0.8, 0.5, 2 * math.pi)


STRENGTH = {"xxz": 0.5, "j1j2": 0.5, "ising": 0.9, "hubbard": 0.5, "driven": 0.8}


def _terms(case, J2=None):
    """(static operator list, dynamic operator list) of the case's model; J2: its tunable coupling (anisotropy,
    next-nearest exchange, transverse field, an eighth of the repulsion)."""
    J2 = STRENGTH[case["model"]] if J2 is None else J2
    L = case["L"]
    nn = [(i, (i + 1) % L) for i in range(L)]
    nnn = [(i, (i + 2) % L) for i in range(L)]
    if case["model"] == "xxz":
        flip = [[0.5, i, j] for i, j in nn]
        return [["+-", flip], ["-+", flip], ["zz", [[J2, i, j] for i, j in nn]]], []
    if case["model"] == "j1j2":
        flip = [[0.5, i, j] for i, j in nn] + [[0.5 * J2, i, j] for i, j in nnn]
        return [["+-", flip], ["-+", flip], ["zz", [[1.0, i, j] for i, j in nn] + [[J2, i, j] for i, j in nnn]]], []
    if case["model"] == "ising":
        return [["zz", [[-1.0, i, j] for i, j in nn]], ["x", [[-J2, i] for i in range(L)]], ["z", [[-0.5, i] for i in range(L)]]], []
    if case["model"] == "driven":
        return ([["zz", [[-1.0, i, j] for i, j in nn]], ["z", [[-0.2, i] for i in range(L)]]],
                [["x", [[-1.0, i] for i in range(L)], _drive, DRIVE]])
    tx, ty = _lattice()
    pairs = [(i, int(m[i])) for m in (tx, ty) for i in range(16)]
    hop, back = [[-1.0, i, j] for i, j in pairs], [[1.0, i, j] for i, j in pairs]
    return [["+-|", hop], ["-+|", back], ["|+-", hop], ["|-+", back], ["n|n", [[8.0 * J2, i, i] for i in range(16)]]], []


def _lattice():
    """Translations of the 4 x 4 periodic square lattice."""
    s = np.arange(16)
    x, y = s % 4, s // 4
    return (x + 1) % 4 + 4 * y, x + 4 * ((y + 1) % 4)


def _basis(case):
    if case["model"] == "hubbard":
        tx, ty = _lattice()
        return spinful_fermion_basis_general(16, Nf=(case["nup"], case["ndown"]), kxblock=(tx, 0), kyblock=(ty, 0))
    L, k = case["L"], case["k"]
    s = np.arange(L)
    blocks = {"kblock": ((s + 1) % L, k)}
    if "p" in case["sym"]:
        blocks["pblock"] = (s[::-1].copy(), 0)
    if "z" in case["sym"]:
        blocks["zblock"] = (-(s + 1), 0)
    if case["model"] in ("ising", "driven"):
        return spin_basis_general(L, **blocks)
    return spin_basis_general(L, Nup=L // 2, pauli=0, **blocks)


def _hamiltonian(case, basis, J2=None):
    static, dynamic = _terms(case, J2)
    return hamiltonian(static, dynamic, basis=basis, dtype=np.dtype(case["dtype"]))


def _sector_cases(case):
    """The momentum sectors of a chain, with reflection resolved at k = 0 and k = L / 2."""
    L = case["L"]
    for k in range(L):
        for p in ((0, 1) if k in (0, L // 2) else (None,)):
            yield k, p, "float64" if p is not None else "complex128"


def _states(n, nvec, dtype, seed):
    """Normalised Gaussian states, one per column."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    wide = torch.complex128 if DTYPES[dtype].is_complex else torch.float64
    v = torch.randn((n, nvec), generator=g, dtype=wide, device=DEV)
    v = v / torch.linalg.vector_norm(v, dim=0)
    return (v[:, 0] if nvec == 1 else v).to(DTYPES[dtype]).contiguous()


def _coupling(seed):
    """A coupling between 0.3 and 0.7 whose multiples are exact, so that no element is zero by rounding alone."""
    return (2 * int(np.random.default_rng(seed).integers(615, 1433)) + 1) / 4096


# -- the cases ------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    np.random.seed(seed % 2**32)                    # the norm estimator draws from numpy's global generator
    if kind == "build":
        return dict(case=case, J2=_coupling(seed))
    if kind == "sectors":
        L, mats = case["L"], []
        s = np.arange(L)
        for k, p, dtype in _sector_cases(case):
            blocks = {"kblock": ((s + 1) % L, k)}
            if p is not None:
                blocks["pblock"] = (s[::-1].copy(), p)
            basis = spin_basis_general(L, **blocks)
            mats.append(hamiltonian(_terms(case)[0], [], basis=basis, dtype=np.dtype(dtype)).tocsr_gpu())
        plan = MultiSectorExpm(mats, a=-1j * case["t"], nvec=case["nvec"])
        v = [_states(M.shape[0], case["nvec"], "complex128", seed + 1000 * b) for b, M in enumerate(mats)]
        return dict(case=case, plan=plan, v=v)
    basis = _basis(case)
    if kind == "free":
        op = quantum_LinearOperator(_terms(case)[0], basis=basis, dtype=np.dtype(case["dtype"]))
        return dict(case=case, op=op, v=_states(basis.Ns, case["nvec"], "complex128", seed))
    H = _hamiltonian(case, basis)
    state = dict(case=case, H=H)
    if kind == "apply":
        state["v"] = _states(H.Ns, case["nvec"], case["vec"], seed)
    elif kind == "expm":
        state["plan"] = ExpmMultiplyParallel(H.tocsr_gpu(), a=-1j * case["t"])
        state["v"] = _states(H.Ns, case["nvec"], "complex128", seed)
    elif kind == "lanczos":
        state["v"] = _states(H.Ns, 1, case["dtype"], seed)
    elif kind == "driven":
        state["v"] = _states(H.Ns, case["nvec"], "complex128", seed)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        return state["H"].dot(state["v"])
    if kind == "expm":
        return state["plan"].dot(state["v"])
    if kind == "sectors":
        return state["plan"].evolve(state["v"], host=False)
    if kind == "lanczos":
        E, V, Q = lanczos_full(state["H"], state["v"], case["m"], reorth=case["reorth"])
        return {"E": E, "V": V, "Q": Q}
    if kind == "free":
        return state["op"].dot(state["v"])
    if kind == "driven":
        return state["H"].evolve(state["v"], 0.0, case["t"])
    basis = _basis(case)
    A = _hamiltonian(case, basis, state["J2"]).tocsr_gpu()
    return {"states": basis.states, "indptr": A.indptr, "indices": A.indices, "data": A.data}


# -- what a pass cannot do without ----------------------------------------------------------------------------------


def _size(case):
    """(states, stored entries) of a case's sector: the particle sector over the group's order, and the mean row."""
    L = case["L"]
    if case["model"] == "hubbard":
        n = math.comb(16, case["nup"]) * math.comb(16, case["ndown"]) / 16
        row = 64 * (case["nup"] / 16 * (1 - case["nup"] / 16) + case["ndown"] / 16 * (1 - case["ndown"] / 16)) * 16 / 15 + 1
        return n, n * row
    G = L * (2 if "p" in case["sym"] else 1) * (2 if "z" in case["sym"] else 1)
    if case["model"] in ("ising", "driven"):
        return 2**L / G, 2**L / G * (L + 1)
    bonds = L if case["model"] == "xxz" else 2 * L
    n = math.comb(L, L // 2) / G
    return n, n * (bonds * 0.5 * L / (L - 1) + 1)


def _taylor_terms(case):
    """About how many products e^{-iHt} takes in double precision: beyond the norm of H t, a few more by the tolerance."""
    L, t = case["L"], case["t"]
    bound = {"xxz": 0.625 * L, "j1j2": 0.75 * L, "ising": 2.4 * L, "driven": 2.5 * L, "hubbard": 40.0}[case["model"]] * t / 2
    return bound + 6.0 * bound ** (1 / 3) + 10


def work(case):
    kind = case["kind"]
    if kind == "sectors":
        n = sum(2.0 ** case["L"] / (case["L"] * (2 if p is not None else 1)) for _, p, _ in _sector_cases(case))
        cplx, val = 2.0, 16
        nnz = n * (case["L"] + 1)
    else:
        n, nnz = _size(case)
        val = {"float32": 4, "float64": 8, "complex64": 8, "complex128": 16}[case["dtype"]]
        cplx = 2.0 if case["dtype"].startswith("complex") else 1.0
    matrix = nnz * (4 + val) + 4 * n
    k = case.get("nvec", 1)
    if kind == "apply":
        e = {"float32": 4, "float64": 8, "complex64": 8, "complex128": 16}[case["vec"]]
        return {"bytes": matrix + 2 * n * k * e, "flops": 2 * nnz * k * cplx * (2 if case["vec"].startswith("complex") else 1)}
    if kind in ("expm", "sectors"):
        m = _taylor_terms(case)
        return {"bytes": m * (matrix + 64 * n * k), "flops": m * nnz * k * 4 * cplx}
    if kind == "lanczos":
        m, e = case["m"], 8 * cplx
        b = m * (matrix + 7 * n * e) + (m * m * n * e if case["reorth"] else 0)
        return {"bytes": b, "flops": m * 2 * nnz * cplx**2 + (2 * m * m * n * cplx**2 if case["reorth"] else 0)}
    if kind == "build":
        return {"bytes": matrix + n * 4, "flops": nnz}
    if kind == "free":
        return {"bytes": n * (4 + 4 + 32 * k), "flops": 4 * nnz * k * cplx}
    calls = 12 * max(2.0, 0.25 * case["L"] * case["t"] * 2.5)     # right-hand sides of an 8th-order integrator at 1e-9
    return {"bytes": calls * (matrix + 48 * n * k), "flops": calls * 4 * nnz * k}


# -- the same results with plain torch in 64 bits -------------------------------------------------------------------


class _Group:
    """The symmetry group of a sector as site permutations (with inversion), phases and, for fermions, signs."""

    def __init__(self, N, generators, fermion):
        self.N, self.fermion = N, fermion
        elements = [(np.arange(N), False, 0.0)]
        for perm, inv, period, q in generators:
            powers, p, f = [], np.arange(N), False
            for g in range(period):
                powers.append((p, f, -2 * math.pi * q * g / period))
                p, f = np.asarray(perm)[p], f != inv
            elements = [(b[a], fa != fb, pa + pb) for a, fa, pa in elements for b, fb, pb in powers]
        self.elements = elements

    def image(self, s, perm, inv):
        """(image of the states s, sign): the value on site i goes to site perm[i]."""
        N, out = self.N, torch.zeros_like(s)
        table = torch.arange(256, device=s.device)
        for b in range(0, N, 8):
            lut = torch.zeros(256, dtype=s.dtype, device=s.device)
            for t in range(min(8, N - b)):
                lut |= ((table >> t) & 1) << (N - 1 - int(perm[N - 1 - b - t]))
            out |= lut[(s >> b) & 255]
        sign = None
        if self.fermion:
            odd = torch.zeros_like(s)
            for i in range(N):
                for j in range(i + 1, N):
                    if perm[i] > perm[j]:
                        odd ^= (s >> (N - 1 - i)) & (s >> (N - 1 - j)) & 1
            sign = 1.0 - 2.0 * odd.double()
        return (out ^ ((1 << N) - 1) if inv else out), sign

    def sector(self, candidates):
        """(states descending, norms) of the symmetric states."""
        s = candidates
        for perm, inv, _ in self.elements:              # keep the largest of each orbit
            s = s[self.image(s, perm, inv)[0] <= s]
        norm = torch.zeros(s.shape, dtype=torch.float64, device=s.device)
        for perm, inv, phase in self.elements:
            t, sign = self.image(s, perm, inv)
            norm += (t == s) * math.cos(phase) * (1.0 if sign is None else sign)
        norm = torch.round(norm)
        s, order = torch.sort(s[norm > 0.5], descending=True)
        return s, norm[norm > 0.5][order]

    def representative(self, s):
        """(largest orbit element, phase, sign of the element that reaches it)."""
        best, phase, sg = s.clone(), torch.zeros(s.shape, dtype=torch.float64, device=s.device), torch.ones(s.shape, dtype=torch.float64, device=s.device)
        for perm, inv, ph in self.elements:
            t, sign = self.image(s, perm, inv)
            up = t > best
            best = torch.where(up, t, best)
            phase = torch.where(up, ph, phase)
            if sign is not None:
                sg = torch.where(up, sign, sg)
        return best, phase, sg


def _candidates(N, ups):
    """All words of N bits with (ups[0] of N set) or, for two entries, set counts per half; None: every word."""
    if ups is None:
        return torch.arange(2**N, dtype=torch.int64, device=DEV)
    halves = []
    for n, k in zip([N // len(ups)] * len(ups), ups):
        keep = []
        for c in torch.arange(2**n, dtype=torch.int64, device=DEV).split(1 << 25):
            bits = torch.zeros_like(c)
            for b in range(n):
                bits += (c >> b) & 1
            keep.append(c[bits == k])
        halves.append(torch.cat(keep))
    return halves[0] if len(ups) == 1 else (halves[0][:, None] * 2 ** (N // 2) + halves[1]).reshape(-1)


def _group(case, k=None, p=None):
    if case["model"] == "hubbard":
        maps = [np.concatenate([m, m + 16]) for m in _lattice()]
        return _Group(32, [(m, False, 4, 0) for m in maps], True), (case["nup"], case["ndown"])
    L = case["L"]
    gens = [((np.arange(L) + 1) % L, False, L, case["k"] if k is None else k)]
    if p is not None or "p" in case.get("sym", ""):
        gens.append((np.arange(L)[::-1], False, 2, p or 0))
    if "z" in case.get("sym", ""):
        gens.append((np.arange(L), True, 2, 0))
    return _Group(L, gens, False), None if case["model"] in ("ising", "driven") else (L // 2,)


def _bonds(case, terms):
    """(string, coupling, sites) per bond, spin-down sites of the lattice shifted by 16, Pauli factors included."""
    for op, bonds in terms:
        for b in bonds:
            sites = list(b[1:])
            if "|" in op:
                at = op.index("|")
                sites = sites[:at] + [x + 16 for x in sites[at:]]
            yield op.replace("|", ""), b[0] * (2.0 ** len(op) if case["model"] in ("ising", "driven") else 1.0), sites


def _matrix(group, states, norms, bonds):
    """Sector matrix of the bonds as (rows, columns, values), duplicates not summed."""
    N, n = group.N, states.numel()
    col = torch.arange(n, device=DEV)
    rows, cols, vals = [], [], []
    asc = states.flip(0).contiguous()
    for op, J, sites in bonds:
        r, amp = states.clone(), torch.full((n,), float(J), dtype=torch.float64, device=DEV)
        for c, site in zip(op[::-1], sites[::-1]):
            b = N - 1 - site
            bit = (r >> b) & 1
            if c == "z":
                amp = amp * (bit - 0.5)
                continue
            if c == "n":
                amp = amp * bit
                continue
            if c == "x":
                amp = 0.5 * amp
            else:
                amp = amp * ((bit == 0) if c == "+" else (bit == 1))
            if group.fermion:
                above = r >> (b + 1)
                for sh in (32, 16, 8, 4, 2, 1):
                    above = above ^ (above >> sh)
                amp = amp * (1 - 2 * (above & 1))
            r = r ^ (1 << b)
        keep = amp != 0
        r, amp, i = r[keep], amp[keep], col[keep]
        if set(op) <= set("zn"):
            rep, phase, sign = r, torch.zeros_like(amp), torch.ones_like(amp)
        else:
            rep, phase, sign = group.representative(r)
        at = torch.searchsorted(asc, rep).clamp(max=n - 1)
        ok = asc[at] == rep
        j = (n - 1 - at)[ok]
        i = i[ok]
        v = (amp * sign)[ok] * torch.sqrt(norms[j] / norms[i])
        rows.append(j), cols.append(i), vals.append(torch.polar(torch.ones_like(v), phase[ok]) * v)
    return torch.cat(rows), torch.cat(cols), torch.cat(vals)


def _csr(group, states, norms, bonds, real):
    n = states.numel()
    r, c, v = _matrix(group, states, norms, bonds)
    if real:
        v = v.real
    A = torch.sparse_coo_tensor(torch.stack([r, c]), v, (n, n)).coalesce()
    keep = A.values().abs() > 1e-14
    return torch.sparse_coo_tensor(A.indices()[:, keep], A.values()[keep], (n, n)).coalesce().to_sparse_csr()


def _apply(A, x):
    """A x for a real or complex CSR and a real or complex block."""
    x2 = x.reshape(x.shape[0], -1)
    if x2.is_complex() and not A.is_complex():
        y = torch.complex(A @ x2.real.contiguous(), A @ x2.imag.contiguous())
    else:
        y = A @ x2.to(torch.promote_types(A.dtype, x2.dtype))
    return y.reshape(x.shape)


def _expm(A, v, t):
    """e^{-i A t} v by Taylor series over steps of unit norm."""
    steps = max(1, math.ceil(2 * t * float(A.values().abs().max()) + 20 * t))
    F = v.clone()
    for _ in range(steps):
        B, k = F, 1
        while k < 80:
            B = _apply(A, B) * (-1j * t / (steps * k))
            F = F + B
            k += 1
            if float(B.abs().max()) < 1e-18:
                break
    return F


def _lanczos(A, v, m, reorth):
    q = v / torch.linalg.vector_norm(v)
    Q, a, b = [q], [], []
    for i in range(m):
        r = _apply(A, Q[i])
        if i:
            r = r - b[-1] * Q[i - 1]
        a.append(torch.vdot(Q[i], r).real.item())
        r = r - a[-1] * Q[i]
        if reorth:
            B = torch.stack(Q)
            for _ in range(2):
                r = r - B.T @ (B.conj() @ r)
        b.append(torch.linalg.vector_norm(r).item())
        if i + 1 < m:
            Q.append(r / b[-1])
    E, V = np.linalg.eigh(np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1))
    return E, V, torch.stack(Q)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sectors":
        out = []
        for b, (k, p, dtype) in enumerate(_sector_cases(case)):
            group, ups = _group(case, k, p)
            s, norms = group.sector(_candidates(group.N, ups))
            A = _csr(group, s, norms, _bonds(case, _terms(case)[0]), p is not None)
            out.append(_expm(A, _states(s.numel(), case["nvec"], "complex128", seed + 1000 * b).reshape(s.numel(), -1), case["t"]))
        return out
    if case["L"] > 30:
        return None                                            # a minute instead of seconds
    group, ups = _group(case)
    s, norms = group.sector(_candidates(group.N, ups))
    n = s.numel()
    static, dynamic = _terms(case, _coupling(seed) if kind == "build" else None)
    A = _csr(group, s, norms, _bonds(case, static), not case["dtype"].startswith("complex"))
    if kind == "build":
        return {"states": None, "indptr": None, "indices": None, "data": A.values()}
    if kind == "apply":
        return _apply(A, _states(n, case["nvec"], case["vec"], seed).to(torch.complex128 if case["vec"].startswith("complex") else torch.float64))
    if kind == "free":
        return _apply(A, _states(n, case["nvec"], "complex128", seed))
    if kind == "expm":
        return _expm(A, _states(n, case["nvec"], "complex128", seed), case["t"])
    if kind == "lanczos":
        E, V, Q = _lanczos(A, _states(n, 1, case["dtype"], seed), case["m"], case["reorth"])
        return {"E": E, "V": None, "Q": Q}                     # an eigenvector's sign is free
    D = _csr(group, s, norms, _bonds(case, [e[:2] for e in dynamic]), True)
    y, steps = _states(n, case["nvec"], "complex128", seed), 4000
    h = case["t"] / steps
    f = lambda t, y: -1j * (_apply(A, y) + _drive(t, *DRIVE) * _apply(D, y))  # noqa: E731
    for i in range(steps):                                     # classical Runge-Kutta, step error far below 1e-9
        t = i * h
        k1 = f(t, y)
        k2 = f(t + h / 2, y + h / 2 * k1)
        k3 = f(t + h / 2, y + h / 2 * k2)
        y = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + f(t + h, y + h * k3))
    return y
