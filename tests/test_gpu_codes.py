"""Value codes on the device (csrc/codes.cu) against the one-dimensional sorts of
the host path: the same table, bytes and count for 1 to 256 distinct values,
refusal of 257 and of NaN, infinities and signed zeros, counts around a
thread's four values and a block's share.  Whole bytes: no tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _values(count, distinct, cplx, rng):
    if cplx:
        side = int(np.ceil(np.sqrt(distinct)))
        table = (rng.normal(size=side)[:, None] + 1j * rng.normal(size=side)[None, :]).ravel()[:distinct]
    else:
        table = rng.normal(size=distinct) * 10.0 ** rng.integers(-300, 300, distinct)
        table[:3] = [0.0, np.inf, -np.inf][:len(table[:3])]
    x = table[rng.integers(0, distinct, count)]
    x[:min(count, distinct)] = table[:min(count, distinct)]
    return torch.tensor(rng.permutation(x))


@pytest.mark.parametrize("count", [1, 3, 4, 5, 1023, 4097, 300001])
@pytest.mark.parametrize("distinct", [1, 3, 255, 256])
@pytest.mark.parametrize("cplx", [False, True])
def test_codes_match_sorts(cuda, count, distinct, cplx):
    from quspin_gb300.sparse import value_codes
    src = _values(count, distinct, cplx, np.random.default_rng(count + distinct + cplx))
    want, got = value_codes(src), value_codes(src.cuda())
    assert got is not None and got[2] == want[2]
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1])


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("count", [257, 5000, 300001])
def test_codes_refused(cuda, count, cplx):
    from quspin_gb300.sparse import value_codes
    rng = np.random.default_rng(count)
    src = _values(count, 257, cplx, rng)
    assert value_codes(src) is None and value_codes(src.cuda()) is None
    every = torch.tensor(rng.normal(size=count) + (1j * rng.normal(size=count) if cplx else 0.0))
    assert value_codes(every.cuda()) is None
    src = _values(count, 5, cplx, rng)
    src[count // 2] = float("nan")
    assert value_codes(src.cuda()) is None


def test_codes_zeros(cuda):
    """Both zeros are one value."""
    from quspin_gb300.sparse import value_codes
    vals, codes, distinct = value_codes(torch.tensor([0.0, -0.0, 1.0, -0.0], dtype=torch.float64).cuda())
    assert distinct == 2 and codes.tolist() == [0, 0, 1, 0] and vals[:2].tolist() == [0.0, 1.0]
