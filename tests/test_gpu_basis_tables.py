"""Basis kernels whose map tables, search queues and binomial table together
pass a shared-memory bound: 48 KB, beyond which a kernel has to opt in by its
static and dynamic part together, and the most a block may use, where the queues
shrink and the binomials are computed instead.  States, norms, the CSR and the
matrix-free product against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.models import square_maps

pytestmark = pytest.mark.gpu


def _pair_swaps(N, count):
    """Commuting maps t_i t_{i+1} of transpositions by three and by one in
    turn: five distances each, so none is a masked shift."""
    t = [((4 * k, 4 * k + 3), (4 * k + 1, 4 * k + 2)) for k in range(N // 4)]
    t = [p for pair in t for p in pair]
    maps = {}
    for i in range(count):
        m = np.arange(N)
        for a, b in (t[i], t[i + 1]):
            m[a], m[b] = b, a
        maps["s%02d" % i] = (m, 0)
    return maps


def _cases():
    sq = square_maps(6, 6)
    lattice = {k: (sq[k], 0) for k in ("tx", "ty", "px", "py")}
    return {
        "lattice": (36, 2, lattice, False),            # 40 KB of tables and 9.3 KB of queues
        "lattice_holes": (36, 34, lattice, False),     # 40 KB and 10 KB of binomials
        "lattice_fermions": (36, 3, lattice, True),
        "three_maps": (56, 54, _pair_swaps(56, 3), False),
        "thirteen_maps": (64, 62, _pair_swaps(64, 13), False),   # 208 KB and 31 KB of binomials
        "thirteen_fermions": (64, 2, _pair_swaps(64, 13), True),
        "fifteen_fermions": (56, 2, _pair_swaps(56, 15), True),  # 220 KB with the sign masks
    }


@pytest.mark.parametrize("name", list(_cases()))
def test_large_tables_match_oracle(cuda, name):
    import torch
    from quspin_gb300 import hamiltonian, quantum_LinearOperator, spin_basis_general, spinless_fermion_basis_general
    N, up, blocks, fermion = _cases()[name]
    make = spinless_fermion_basis_general if fermion else spin_basis_general
    b = make(N, Nf=up, **blocks) if fermion else make(N, Nup=up, pauli=0, **blocks)
    ob = O.OracleBasis(N, [(1, up, 0)], fermion=fermion, **blocks)
    np.testing.assert_array_equal(b.states.astype(np.uint64), ob.states)
    np.testing.assert_array_equal(b._n.astype(np.uint32), ob.norms)
    assert len(ob.states) > 1
    bonds = [[0.7, i, (i + 1) % N] for i in range(N)]
    static = [["+-", bonds], ["-+", [[-J if fermion else J, i, j] for J, i, j in bonds]], ["zz", bonds]]
    Ho = O.make_static(ob, static, np.complex128).tocsr()
    H = hamiltonian(static, [], basis=b, dtype=np.complex128).tocsr()
    for mine, theirs in ((H.indptr, Ho.indptr), (H.indices, Ho.indices), (H.data, Ho.data)):
        np.testing.assert_array_equal(mine, theirs)
    v = torch.randn(b.Ns, dtype=torch.complex128, generator=torch.Generator().manual_seed(1)).numpy()
    got = quantum_LinearOperator(static, basis=b, dtype=np.complex128).dot(v)
    # some tens of products a row, summed in any order
    bound = 100 * np.finfo(np.float64).eps * (abs(Ho) @ abs(v)).max()
    np.testing.assert_allclose(got, Ho @ v, rtol=0, atol=bound)
