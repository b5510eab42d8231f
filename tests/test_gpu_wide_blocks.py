"""Blocks of so many vectors that a row of them passes 4 GB: the kernels'
strides leave 32 bits.  Two rows, all columns checked on the device."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vec,power", [("complex128", 28), ("float64", 29), ("complex64", 29), ("float32", 30),
                                       ("complex128", 27)])
def test_products_of_wide_blocks(cuda, vec, power):
    import torch
    from quspin_gb300.sparse import DeviceCSR
    k = 2**power + 3
    tdt = getattr(torch, vec)
    M = DeviceCSR.from_scipy(sp.csr_matrix(np.array([[1.0, 2.0], [0.5, -1.0]])))
    if vec in ("float32", "complex64"):
        M = M.astype(np.float32)
    x = torch.empty((2, k), dtype=tdt, device="cuda")
    for r in range(2):                                      # whole numbers: no rounding anywhere
        real = x[r] if not tdt.is_complex else torch.view_as_real(x[r]).view(-1)
        torch.arange(real.numel(), out=real)
        real.remainder_(4093 + 4 * r)
    y = torch.empty_like(x)
    M.matvec_into(x, y)
    for c0 in range(0, k, 1 << 26):
        a, b = x[0, c0:c0 + (1 << 26)], x[1, c0:c0 + (1 << 26)]
        assert bool((y[0, c0:c0 + (1 << 26)] == a + 2 * b).all()) and bool((y[1, c0:c0 + (1 << 26)] == a / 2 - b).all())
    del x, y, a, b
    torch.cuda.empty_cache()


@pytest.mark.parametrize("dtype", ["PF", "PF8"])
def test_terms_of_wide_blocks_are_taken(cuda, dtype):
    """A launch after the stopping test fired returns at once: the call is
    accepted with 2^27 vectors, with and without a launch shape."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    from quspin_gb300.sparse import DeviceCSR, PairedCSR
    from quspin_gb300.tune import encode, lanes_operand
    P = PairedCSR(DeviceCSR.from_scipy(sp.csr_matrix(np.array([[1.0, 2.0], [0.5, -1.0]]))), coded=dtype == "PF8")
    assert P.vcode == getattr(_lib, dtype)
    k = 1 << 27
    b = torch.empty((2, 2, k), dtype=torch.complex128, device="cuda")
    F = torch.ones((2, k), dtype=torch.complex128, device="cuda")
    ctl = torch.zeros(_lib.load().qs_expm_ctl_bytes() // 8 + 1, dtype=torch.int64, device="cuda")
    ctl.view(torch.int32)[6] = 1                            # done
    c = torch.ones(1, dtype=torch.complex128, device="cuda")
    for code in (0, encode(2, 2) | (1 << 20)):
        A = lanes_operand(P, k, code)
        _lib.call("qs_taylor_term", 2, A.nnz, D.ptr(A.indptr), 0, D.ptr(A.indices), D.ptr(A.data), A.vcode,
                  D.ptr(b[0]), D.ptr(b[1]), _lib.CPF, D.ptr(F), k, 0.0, 0.0, D.ptr(c), 0, 0.0, D.ptr(ctl), code,
                  D.stream())
    assert bool((F == 1).all())
    del b, F
    torch.cuda.empty_cache()
