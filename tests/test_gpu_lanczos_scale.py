"""The scaling of a Lanczos vector, x / b by b's reciprocal and a correction,
bit for bit against the division: random significands over all exponents, the
bounds of the range in which the short form is used, powers of two, zeros of
both signs, subnormals, infinities and NaN.  The short form is correctly rounded
and so is a division: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [s * f * 2.0**e for s in (1.0, -1.0) for f in (1.0, 1.0 + 2.0**-52, 1.5, 2.0 - 2.0**-52)
         for e in (-1022, -901, -900, -899, -501, -500, -499, -1, 0, 1, 499, 500, 501, 899, 900, 1023)]
SPECIAL = [0.0, -0.0, 5e-324, -2.2e-308, np.inf, -np.inf, np.nan]


@pytest.mark.parametrize("scale", [0, -480, 499, -900, 1000])
def test_scaling_is_a_division(cuda, scale):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    rng = np.random.default_rng(scale + 2000)
    near = rng.normal(size=20000)
    wide = rng.normal(size=20000) * 2.0 ** rng.integers(-1060, 1020, size=20000).astype(float)
    x = np.concatenate([near, near * 2.0 ** float(min(scale, 900)), wide, EDGES, SPECIAL])
    xd = D.to_device(x)
    q = torch.empty_like(xd)
    divisors = np.concatenate([rng.uniform(1.0, 2.0, 40) * 2.0 ** float(scale), [2.0 ** float(scale), np.inf, 0.0]])
    if scale == 0:
        divisors = np.concatenate([divisors, EDGES, [2.0 - 2.0**-52, 1.0 + 2.0**-52, 5e-324, np.nan]])
    for b in divisors:
        _lib.call("qs_lanczos_scale", x.size, D.ptr(xd), D.ptr(D.to_device(np.array([b]))), D.ptr(q), None, D.stream())
        with np.errstate(all="ignore"):
            want = x / b
        got = D.to_host(q)
        fine = ~np.isnan(want)
        np.testing.assert_array_equal(got.view(np.uint64)[fine], want.view(np.uint64)[fine], err_msg=str(b))
        assert np.isnan(got[~fine]).all(), b
