"""Every form of the symmetry maps and the orbit walk against the oracle, bit
for bit: masked shifts (with and without the bit reversal) and byte tables,
one to four maps in nested loops and the odometer beyond, 32- and 64-bit
states, fermion signs from parity products and from the per-site masks, and
sectors from one state up, through states, norms, representatives and the
canonical CSR (whose merge inserts, joins or drops diagonal entries)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.models import chain_maps, square_maps

pytestmark = pytest.mark.gpu


def _swap(N, i, j):
    m = np.arange(N)
    m[i], m[j] = j, i
    return m


def _cycle(N, sites):
    m = np.arange(N)
    m[sites] = np.roll(sites, -1)
    return m


def _cases():
    c12, c7 = chain_maps(12), chain_maps(7)
    c34 = chain_maps(34)
    sq = square_maps(4, 4)
    scattered = _cycle(12, [0, 5, 3, 10, 2, 7])      # more than four distances: byte tables
    both = [np.concatenate([sq[k], sq[k] + 16]) for k in ("tx", "ty")]
    return {
        "no_maps": (9, 4, {}, False),
        "one_state": (6, 0, dict(t=(chain_maps(6)["t"], 0)), False),
        "odd_chain": (7, 3, dict(t=(c7["t"], 2)), False),
        "three_maps": (12, 6, dict(t=(c12["t"], 0), p=(c12["p"], 1), z=(c12["z"], 0)), False),
        "tables": (12, 5, dict(s=(scattered, 1)), False),
        "tables_and_shifts": (12, None, dict(s=(scattered, 0), z=(c12["z"], 1)), False),
        "four_maps": (16, 8, dict(tx=(sq["tx"], 0), ty=(sq["ty"], 2), px=(sq["px"], 0), z=(sq["z"], 0)), False),
        "five_maps": (10, 5, {"s%d" % i: (_swap(10, i, i + 5), i % 2) for i in range(5)}, False),
        "wide_words": (34, 3, dict(t=(c34["t"], 0), p=(c34["p"], 0)), False),
        "wide_momentum": (34, 2, dict(t=(c34["t"], 5)), False),
        "fermion_ring": (9, 4, dict(t=(chain_maps(9)["t"], 3)), True),
        "fermion_tables": (12, 5, dict(s=(scattered, 2)), True),
        "fermion_reflection": (11, 5, dict(p=(chain_maps(11)["p"], 1)), True),
        "fermion_long": (36, 2, dict(p=(np.arange(36)[::-1].copy(), 0)), True),
        "fermion_lattice": (32, (2, 3), dict(tx=(both[0], 1), ty=(both[1], 0)), True),
    }


def _bases(name):
    from quspin_gb300 import (spin_basis_general, spinful_fermion_basis_general, spinless_fermion_basis_general)
    N, up, blocks, fermion = _cases()[name]
    if isinstance(up, tuple):
        b = spinful_fermion_basis_general(N // 2, Nf=up, simple_symm=False, **blocks)
        return b, O.OracleBasis(N, [(2, *up)], fermion=True, **blocks)
    if fermion:
        return spinless_fermion_basis_general(N, Nf=up, **blocks), O.OracleBasis(N, [(1, up, 0)], fermion=True, **blocks)
    sectors = [(0, 0, 0)] if up is None else [(1, up, 0)]
    return spin_basis_general(N, Nup=up, pauli=0, **blocks), O.OracleBasis(N, sectors, **blocks)


@pytest.mark.parametrize("name", list(_cases()))
def test_orbit_forms_match_oracle(cuda, name):
    from quspin_gb300 import hamiltonian
    b, ob = _bases(name)
    np.testing.assert_array_equal(b.states.astype(np.uint64), ob.states)
    np.testing.assert_array_equal(b._n.astype(np.uint32), ob.norms)
    N, up, _, fermion = _cases()[name]
    rng = np.random.default_rng(7)
    if up is None or isinstance(up, tuple):
        words = rng.integers(0, 2**N, size=300).astype(np.uint64)
    else:
        words = np.array([sum(1 << int(i) for i in rng.choice(N, up, replace=False)) for _ in range(300)], np.uint64)
    reps, g, sign = b.representative(words, return_g=True, return_sign=True)
    for mine, theirs in zip((reps.astype(np.uint64), g, sign), ob.representative(words)):
        np.testing.assert_array_equal(mine, theirs)
    np.testing.assert_array_equal(np.atleast_1d(b.normalization(words)).astype(np.uint32), ob.normalization(words))
    bonds = [[0.7 - 0.05 * i, i, (i + 3) % N] for i in range(N)]
    # hops both ways, diagonal terms that cancel on some rows, and a term the
    # sector may annihilate altogether
    static = [["+-", bonds], ["-+", [[-J if fermion else J, i, j] for J, i, j in bonds]],
              ["zz", [[0.25, i, (i + 1) % N] for i in range(N)]], ["z", [[-0.125, i] for i in range(N)]]]
    H = hamiltonian(static, [], basis=b, dtype=np.complex128).tocsr()
    Ho = O.make_static(ob, static, np.complex128).tocsr()
    for mine, theirs in ((H.indptr, Ho.indptr), (H.indices, Ho.indices), (H.data, Ho.data)):
        np.testing.assert_array_equal(mine, theirs)
