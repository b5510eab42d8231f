"""The one-call Lanczos run (float-pair CSR, vectors kept) against the step by
step loop on the same matrix with int64 row pointers, which the run does not
take: coefficients, vectors and the number of valid vectors, real and complex,
plain and packed values, with and without reorthogonalisation, from a handful
of rows to several blocks, and a start vector in a small invariant subspace.

Tolerance: both form the products in float pairs (48 bits, row sums within
1e-13 of their moduli) in the same order and differ in the order of FP64 sums;
12 steps in random matrices amplify that by less than 1e2."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n, cplx, distinct, rng):
    A = sp.random(n, n, density=min(1.0, 9.0 / n), random_state=rng, format="csr")
    A.data = rng.choice(np.array([0.5, -1.0, 0.25, 1.5]), A.nnz) if distinct else rng.normal(size=A.nnz)
    if cplx:
        A = A.astype(complex)
        A.data = A.data * rng.choice(np.array([1.0, 1j, -1j]), A.nnz)
    A = sp.csr_matrix(A + A.conj().T + sp.diags(rng.choice(np.array([-0.5, 0.75, 2.0]), n)))
    A.sum_duplicates()
    return A


@pytest.mark.parametrize("n", [13, 255, 5003, 70001])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("coded", [False, True])
@pytest.mark.parametrize("reorth", [False, True])
def test_run_matches_steps(cuda, n, cplx, coded, reorth):
    import torch
    from quspin_gb300.sparse import DeviceCSR
    from quspin_gb300.tools import lanczos_full
    rng = np.random.default_rng(n + 2 * cplx + coded)
    A = _matrix(n, cplx, coded, rng)
    M = DeviceCSR.from_scipy(A)
    if coded:
        assert M.paired().coded
    M64 = DeviceCSR(M.indptr.to(torch.int64), M.indices, M.data, M.shape, M.dtype)
    v = rng.normal(size=n) + (1j * rng.normal(size=n) if cplx else 0.0)
    m = min(12, n - 1)
    E, V, Q = lanczos_full(M, v, m, reorth=reorth)
    E2, V2, Q2 = lanczos_full(M64, v, m, reorth=reorth)
    assert Q.shape == Q2.shape == (m, n)
    np.testing.assert_allclose(E, E2, rtol=0, atol=1e-11 * abs(E2).max())
    tol = 1e-11 if reorth or n > 1000 else 1e-6        # short of n = 13 the plain recurrence meets converged pairs
    np.testing.assert_allclose(Q, Q2, rtol=0, atol=tol)
    if reorth:
        np.testing.assert_allclose(Q.conj() @ Q.T, np.eye(m), rtol=0, atol=1e-13)
    T = np.einsum("ij,ij->i", Q.conj(), (A @ Q.T).T).real
    np.testing.assert_allclose(np.diag((V * E) @ V.T), T, rtol=0, atol=1e-11 * abs(E2).max())


@pytest.mark.parametrize("reorth", [False, True])
def test_run_stops_in_invariant_subspace(cuda, reorth):
    from quspin_gb300.sparse import DeviceCSR
    from quspin_gb300.tools import lanczos_full
    n = 300
    A = sp.diags([np.ones(n - 1), np.ones(n - 1)], [-1, 1]).tolil()
    A[5, 6] = A[6, 5] = 0.0
    v = np.zeros(n)
    v[0] = 1.0
    E, V, Q = lanczos_full(DeviceCSR.from_scipy(sp.csr_matrix(A)), v, 20, reorth=reorth, eps=1e-12)
    assert Q.shape[0] in (6, 5)                        # b vanishes after the sixth vector
    k = Q.shape[0]
    np.testing.assert_allclose(np.sort(E), np.linalg.eigvalsh(A.toarray()[:k, :k]), rtol=0, atol=1e-13)


@pytest.mark.parametrize("form", ["hamiltonian", "csr", "linop", "mixed"])
@pytest.mark.parametrize("off", [-3, 4])
def test_start_vector_of_another_size_is_refused(cuda, form, off):
    """The run and the steps take the operator's row count for the vectors'
    length, so a start vector of another length is an error before any launch."""
    from quspin_gb300 import hamiltonian, quantum_LinearOperator, spin_basis_general
    from quspin_gb300.tools import lanczos_full, lanczos_iter
    from tests.models import xxz_static
    b = spin_basis_general(10, Nup=5, pauli=0)
    H = hamiltonian(xxz_static(10), [], basis=b, dtype=np.float64)
    A = {"hamiltonian": H, "csr": H.static, "mixed": H,
         "linop": quantum_LinearOperator(xxz_static(10), basis=b, dtype=np.float64)}[form]
    v = np.ones(b.Ns + off)
    for reorth in (False, True):
        with pytest.raises(ValueError, match="mismatch"):
            lanczos_full(A, v, 6, reorth=reorth, precision="mixed" if form == "mixed" else "double")
    with pytest.raises(ValueError, match="mismatch"):
        lanczos_iter(A, v, 6)
