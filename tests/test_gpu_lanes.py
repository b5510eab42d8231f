"""Products of several vectors with the vectors across the lanes, at every
group width (2 to 8 lanes, one and two words fetched per lane, two sweeps),
for plain, coded and packed values, real and complex, int32 and int64 row
pointers, over rows from empty to many batches and a row count that leaves
groups and warps partly filled; and the conversion to float pairs without FP64
instructions, bit for bit the FP64 form.

Tolerance of a product: a float pair carries 48 bits, so a product and its
share of a sum are within 2^-45 of their moduli; rows of up to 70 entries
random in sign stay within 1e-13 of the row's sum of moduli."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n, cplx, rng):
    lens = rng.integers(0, 12, n)
    lens[rng.integers(0, n, n // 7)] = 0
    lens[5], lens[n - 1] = 70, 33
    rows = np.repeat(np.arange(n), lens)
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]) if lens.sum() else []
    vals = rng.choice(np.array([0.5, -1.0, 0.3, 2.0 / 3.0]), len(rows))
    if cplx:
        vals = vals + 1j * rng.choice(np.array([0.0, 0.7, -0.1]), len(rows))
    return sp.csr_matrix((vals, (rows, cols)), shape=(n, n))


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8, 9, 13])
@pytest.mark.parametrize("cplx_A,cplx_x", [(False, False), (False, True), (True, True)])
def test_products_across_lanes(cuda, k, cplx_A, cplx_x):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import DeviceCSR, PairedCSR
    rng = np.random.default_rng(100 * k + 10 * cplx_A + cplx_x)
    n = 421
    A = _matrix(n, cplx_A, rng)
    x = rng.normal(size=(n, k)) * 10.0 ** rng.integers(-9, 9, size=(n, 1))
    if cplx_x:
        x = x + 1j * rng.normal(size=(n, k))
    ref, scale = A @ x, abs(A) @ abs(x)
    M32 = DeviceCSR.from_scipy(A)
    M64 = DeviceCSR(M32.indptr.to(torch.int64), M32.indices, M32.data, M32.shape, M32.dtype)
    coded = PairedCSR(M32, coded=True)
    assert coded.coded
    xd = D.to_device(x)
    first = None
    for M, P in ((M32, PairedCSR(M32, coded=False)), (M64, PairedCSR(M64, coded=False)), (M32, coded),
                 (M32, coded.packed())):
        y = torch.full_like(xd, 0.25)
        M.matvec_into(xd, y, a=1.0, overwrite=True, operand=P)
        h = D.to_host(y)
        assert np.all(abs(h - ref) <= 1e-13 * scale + 1e-300), P.vcode
        first = h if first is None else first
        np.testing.assert_array_equal(h, first)          # the same pairs in the same order
        M.matvec_into(xd, y, a=-1.0, overwrite=False, operand=P)
        assert np.all(abs(D.to_host(y)) <= 1e-15 * scale + 1e-300), P.vcode
    s = (np.complex64 if cplx_x else np.float32)
    M1 = M32.astype(np.complex64 if cplx_A else np.float32)
    x1 = (x / abs(x).max()).astype(s)
    y1 = torch.empty_like(D.to_device(x1))
    M1.matvec_into(D.to_device(x1), y1)
    # FP32 sums of up to 70 products
    assert np.all(abs(D.to_host(y1) - A @ x1.astype(np.complex128)) <= 80 * 6e-8 * (abs(A) @ abs(x1)) + 1e-38)


def test_pairs_without_fp64(cuda):
    """qs_split_pairs: hi = float(x), lo = float(x - hi) on random doubles of
    every exponent, exact halves between floats, powers of two, zeros,
    subnormals, infinities and NaN."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    rng = np.random.default_rng(3)
    x = rng.normal(size=200000) * 2.0 ** rng.integers(-160, 126, size=200000).astype(float)
    h = rng.normal(size=1000).astype(np.float32).astype(np.float64)
    half = np.spacing(np.abs(h).astype(np.float32)).astype(np.float64) / 2
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.2e-308, 1e300, 1.0, -1.0, 2.0**-126, 2.0**-149,
                     2.0**127, 2.0 - 2.0**-52, 2.0**-73, 2.0**-74])
    x = np.concatenate([x, h + half, h - half, h * (1 + 2.0**-52), edge])
    out = torch.empty(2 * len(x), dtype=torch.float32, device="cuda")
    xd = D.to_device(x)
    _lib.call("qs_split_pairs", len(x), D.ptr(xd), D.ptr(out), D.stream())
    got = D.to_host(out).reshape(-1, 2)
    with np.errstate(all="ignore"):
        hi = x.astype(np.float32)
        lo = (x - hi.astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(got[:, 0].view(np.uint32)[~np.isnan(hi)], hi.view(np.uint32)[~np.isnan(hi)])
    fine = ~np.isnan(lo)
    np.testing.assert_array_equal(got[fine, 1], lo[fine])
    assert np.all(np.isnan(got[~fine, 1]))


@pytest.mark.parametrize("n", [3, 245, 4752, 30000])
@pytest.mark.parametrize("k", [1, 2, 5])
def test_small_products_default_form(cuda, n, k):
    """The default product of a small matrix is the IEEE form, at every lane
    count its row count picks, within FP64 rounding of each row; a large one
    stays in float pairs."""
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import DeviceCSR
    rng = np.random.default_rng(n + k)
    A = sp.random(n, n, density=min(1.0, 12.0 / n), random_state=rng, format="csr")
    x = rng.normal(size=(n, k)) + 1j * rng.normal(size=(n, k))
    x = x[:, 0].copy() if k == 1 else x
    M = DeviceCSR.from_scipy(A)
    assert M._small(k, True) == (2 * M.nnz * k <= (3_000_000 if k <= 2 else 1_000_000))
    y = M.dot(D.to_device(x))
    # up to 30 entries a row: at most 64 roundings of 2^-53 in the IEEE form, 48-bit pairs otherwise
    assert np.all(abs(D.to_host(y) - A @ x) <= (1e-14 if M._small(k, True) else 1e-13) * (abs(A) @ abs(x)))
    assert ("_paired" in M.__dict__) == (not M._small(k, True))
