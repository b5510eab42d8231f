"""Several vectors and long rows: rows divided over the lanes of a warp
(vl_split), sweeps of the vectors in blocks of their own, on both sides of
every bound of the rules, with rows from empty to twice the mean, in products
and Taylor terms, float pairs and single precision.

Tolerances: a product of float pairs and its share of the row's sum are within
2^-46 of the row's sum of moduli, FP32 ones within 2^-23; a term's row norm is
a sum of at most 16 moduli."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

# rows, mean entries: dense, few long rows, few short, few of middling length, many long ones
SHAPES = [(23, 20), (300, 150), (1000, 40), (900, 260), (9000, 70), (14000, 140)]


def _matrix(n, mean, cplx):
    rng = np.random.default_rng(n + mean)
    lens = np.minimum(rng.integers(0, 2 * mean + 1, n), n)
    lens[n // 2] = 0
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens])
    vals = rng.choice(np.array([0.5, -1.0, 0.3, 2.0 / 3.0]), len(cols))
    if cplx:
        vals = vals + 1j * rng.choice(np.array([0.0, 0.7, -0.1]), len(cols))
    return sp.csr_matrix((vals, cols, np.concatenate([[0], np.cumsum(lens)])), shape=(n, n))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("cplx", [False, True])
def test_long_rows_many_vectors(cuda, shape, cplx):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    from quspin_gb300.sparse import DeviceCSR, PairedCSR
    A = _matrix(*shape, cplx)
    n, most = A.shape[0], int(np.diff(A.indptr).max())
    M = DeviceCSR.from_scipy(A)
    M1 = M.astype(np.complex64 if cplx else np.float32)
    P = PairedCSR(M, coded=True)
    for k in (2, 3, 5, 6, 8, 13, 16):
        rng = np.random.default_rng(k)
        x = rng.normal(size=(n, k)) + 1j * rng.normal(size=(n, k))
        ref, scale = A @ x, abs(A) @ abs(x)
        xd = D.to_device(x)
        for Q in (P, P.packed(), PairedCSR(M, coded=False)):
            y = torch.full_like(xd, 0.25)
            M.matvec_into(xd, y, operand=Q)
            assert np.all(abs(D.to_host(y) - ref) <= most * 2.0**-46 * scale), (k, Q.vcode)
        x1 = xd.to(torch.complex64)
        y1 = torch.empty_like(x1)
        M1.matvec_into(x1, y1)
        h1 = D.to_host(x1).astype(np.complex128)
        assert np.all(abs(D.to_host(y1) - A @ h1) <= most * 2.0**-23 * (abs(A) @ abs(h1))), k
        # one term: B' = c A B, F += B', and the largest row sum of moduli
        b0, b1 = torch.empty((n, k, 4), dtype=torch.float32, device="cuda"), torch.empty((n, k, 4), device="cuda")
        _lib.call("qs_split_pairs", 2 * n * k, D.ptr(xd), D.ptr(b0), D.stream())
        F = xd.clone()
        ctl = torch.zeros(_lib.load().qs_expm_ctl_bytes() // 8 + 1, dtype=torch.int64, device="cuda")
        c = torch.tensor([0.375 - 0.25j], dtype=torch.complex128, device="cuda")
        Q = P.packed()
        _lib.call("qs_taylor_term", n, M.nnz, D.ptr(Q.indptr), 0, D.ptr(Q.indices), D.ptr(Q.data), Q.vcode, D.ptr(b0),
                  D.ptr(b1), _lib.CPF, D.ptr(F), k, 0.0, 0.0, D.ptr(c), 0, 0.0, D.ptr(ctl), 0, D.stream())
        got = D.to_host(b1).astype(np.float64)
        got = (got[..., 0] + got[..., 1]) + 1j * (got[..., 2] + got[..., 3])
        cr = 0.375 - 0.25j
        assert np.all(abs(got - cr * ref) <= (most + 8) * 2.0**-46 * scale)
        assert np.all(abs(D.to_host(F) - x - got) <= 2.0**-50 * (abs(x) + abs(got)))
        top = ctl[:1].view(torch.float64).item()
        assert abs(top - abs(got).sum(axis=1).max()) <= 1e-12 * top


@pytest.mark.parametrize("n,row", [(20000, 24), (5000, 100), (2000, 400), (400, 400)])
@pytest.mark.parametrize("cplx", [False, True])
def test_single_precision_of_many_vectors(cuda, n, row, cplx):
    """The root mean square error of an FP32 product of several vectors is no
    larger than that of one, whose row sums are spread over lanes.  The bound's
    fifth covers the samples' scatter (a few per cent)."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import DeviceCSR
    rng = np.random.default_rng(row)
    cols = np.sort((np.arange(n)[:, None] + rng.permutation(n)[:row]) % n, axis=1)
    vals = (rng.normal(size=n * row) + (1j * rng.normal(size=n * row) if cplx else 0.0)).astype(
        np.complex64 if cplx else np.float32)
    A = sp.csr_matrix((vals, cols.ravel(), np.arange(n + 1) * row), shape=(n, n))
    M = DeviceCSR.from_scipy(A)
    assert M.dtype == vals.dtype

    def error(k):
        x = (rng.normal(size=(n, k)) + 1j * rng.normal(size=(n, k))).astype(np.complex64)
        xd = D.to_device(x[:, 0].copy() if k == 1 else x)
        y = torch.empty_like(xd)
        M.matvec_into(xd, y)
        ref = A.astype(np.complex128) @ x.astype(np.complex128)
        return np.linalg.norm(D.to_host(y).reshape(n, k) - ref) / np.linalg.norm(ref)
    one = error(1)
    for k in (2, 3, 5, 8, 13):
        assert error(k) <= 1.2 * one, k
