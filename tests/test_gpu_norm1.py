"""The single-vector norm of the Taylor loop (taylor_norm1_kernel in
csrc/expm_lp.cu): F scaled by eta and its largest modulus, at sizes around a
warp, a block and a grid's sweep, with moduli of one size, of a wide range,
mostly zero, subnormal, infinite and NaN elements.

Tolerance: the scaled elements are two rounded products and a sum, compared at
4 units in the last place of the products' size; the norm is the largest hypot
of the elements that the device stored, within the 2 units in the last place
that CUDA documents for hypot."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(kind, n, rng):
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    if kind == "wide":
        v *= 10.0 ** rng.integers(-290, 290, n)
    if kind == "sparse":
        v *= rng.random(n) < 3.0 / n
    if kind == "tiny":
        v *= 1e-310
    if kind == "equal":                       # moduli that differ in the last places only
        ph = rng.random(n) * 2 * np.pi
        v = (1.0 + 1e-15 * rng.integers(0, 4, n)) * np.exp(1j * ph)
    if kind == "ascending":
        v = np.arange(1, n + 1) * np.exp(1j * rng.random(n))
    return v


@pytest.mark.parametrize("kind", ["normal", "wide", "sparse", "tiny", "equal", "ascending"])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 70001, 700001])
@pytest.mark.parametrize("use_eta", [False, True])
def test_norm_and_scaling(cuda, kind, n, use_eta):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    rng = np.random.default_rng(n)
    v = _values(kind, n, rng)
    eta = 0.6 - 0.8j if use_eta else 1.0
    F = D.to_device(v.astype(np.complex128))
    b0 = torch.empty_like(F)
    ctl = torch.zeros(_lib.load().qs_expm_ctl_bytes() // 8 + 1, dtype=torch.int64, device="cuda")
    e = torch.tensor([eta], dtype=torch.complex128, device="cuda")
    _lib.call("qs_taylor_rescale", n, 1, D.ptr(F), D.ptr(b0), _lib.CPF, D.ptr(e), D.ptr(ctl), 0, D.stream())
    out = D.to_host(F)
    if use_eta:
        size = 0.6 * np.maximum(abs(v.real), abs(v.imag)) + 0.8 * np.maximum(abs(v.real), abs(v.imag))
        assert (abs(out - v * eta) <= 8 * 2.0 ** -53 * size + 2e-323).all()
    else:
        np.testing.assert_array_equal(out, v)
    want = np.hypot(out.real, out.imag).max()
    c1 = float(ctl.view(torch.float64)[0])
    assert abs(c1 - want) <= 4 * np.spacing(want)


def test_norm_of_infinity_and_nan(cuda):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    for bad, want in ((np.inf, np.inf), (np.nan, 3.0)):           # a NaN counts as nothing
        v = np.full(5000, 3.0 + 0j)
        v[4321] = bad
        F = D.to_device(v)
        b0 = torch.empty_like(F)
        ctl = torch.zeros(_lib.load().qs_expm_ctl_bytes() // 8 + 1, dtype=torch.int64, device="cuda")
        e = torch.ones(1, dtype=torch.complex128, device="cuda")
        _lib.call("qs_taylor_rescale", 5000, 1, D.ptr(F), D.ptr(b0), _lib.CPF, D.ptr(e), D.ptr(ctl), 0, D.stream())
        assert float(ctl.view(torch.float64)[0]) == want
