"""The sliced operand and its single-vector kernels (csrc/sell.cu): the words
of every row survive the re-ordering, at slice edges, with empty, even, uneven
and over-long rows; the product, the Taylor term and the Lanczos product against
the row hand-out kernels on the same packed operand; padding never reads into
a result.

Tolerance: the same float-pair products summed in another order, 48-bit
roundings over at most 128 nonzeros: 1e-13 of the row's absolute sum."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n, cplx, kind, rng):
    m = min(n, 9)
    if kind == "uneven":                                  # empty rows among rows of up to 12
        lens = rng.integers(0, min(n, 12) + 1, n)
    elif kind == "long":
        lens = np.full(n, min(n, 128))
    else:
        lens = np.full(n, m)
    cols = [np.sort(rng.choice(n, l, replace=False)) for l in lens]
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    vals = rng.choice(np.array([0.5, -1.25, 2.0, 1.0 / 3.0]), ip[-1])
    if cplx:
        vals = vals * rng.choice(np.array([1.0, 1j, 0.6 + 0.8j]), ip[-1])
    return sp.csr_matrix((vals, np.concatenate(cols) if ip[-1] else np.zeros(0, np.int32), ip), shape=(n, n))


def _packed(A):
    from quspin_gb300.sparse import DeviceCSR
    M = DeviceCSR.from_scipy(A)
    return M, M.paired().packed()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 1024, 5000])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["even", "uneven", "long"])
def test_sliced_words_and_product(cuda, n, cplx, kind):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import SLICED, SlicedCSR
    from quspin_gb300.tune import encode
    rng = np.random.default_rng(n + 7 * cplx + len(kind))
    A = _matrix(n, cplx, kind, rng)
    if A.nnz == 0:
        pytest.skip("no nonzeros")
    M, P = _packed(A)
    limit, SlicedCSR.MAX_PADDING = SlicedCSR.MAX_PADDING, 40.0
    try:
        S = P.sliced()
    finally:
        SlicedCSR.MAX_PADDING = limit
    # every row's words, as a set, and nothing else
    sptr, words = D.to_host(S.indptr), D.to_host(S.indices).view(np.uint32)
    src = D.to_host(P.indices).view(np.uint32)
    for s in range((n + 31) // 32):
        block = words[sptr[s] * 128:sptr[s + 1] * 128].reshape(-1, 32, 4)
        for lane in range(32):
            got = block[:, lane, :].reshape(-1)
            got = np.sort(got[got != 0xffffffff])
            r = s * 32 + lane
            want = src[A.indptr[r]:A.indptr[r + 1]] if r < n else src[:0]
            np.testing.assert_array_equal(got, np.sort(want))
    group = encode(2, 1)
    for xc in ([True] if cplx else [False, True]):
        x = rng.normal(size=n) + (1j * rng.normal(size=n) if xc else 0.0)
        xd = D.to_device(x)
        scale = abs(A) @ np.abs(x) + 1e-300
        for a, over in ((1.0, True), ((0.3 - 0.7j) if xc else -0.7, False)):
            y0 = rng.normal(size=n) + (1j * rng.normal(size=n) if xc else 0.0)
            y1, y2 = D.to_device(y0.astype(x.dtype)), D.to_device(y0.astype(x.dtype))
            M.matvec_into(xd, y1, a=a, overwrite=over, group=group, precision="double", operand=P)
            M.matvec_into(xd, y2, a=a, overwrite=over, group=group | SLICED, precision="double", operand=P)
            y1, y2 = D.to_host(y1), D.to_host(y2)
            assert (np.abs(y1 - y2) <= 1e-13 * (scale + np.abs(y0))).all()
    # a PAD reads column 0 and adds nothing: infinity there stays in the rows that hold it
    x = np.ones(n, complex)
    x[0] = np.inf
    y = D.to_device(np.zeros(n, complex))
    M.matvec_into(D.to_device(x), y, group=group | SLICED, precision="double", operand=P)
    holds = np.asarray((A[:, 0] != 0).todense()).ravel()
    assert np.isfinite(D.to_host(y)[~holds]).all()


def test_sliced_refused(cuda):
    rng = np.random.default_rng(0)
    n = 4000
    A = sp.random(n, n, density=0.0005, random_state=rng, format="lil")
    A[5, :129] = 1.0                                        # one row too long for a slice
    A = A.tocsr()
    A.data = rng.choice(np.array([1.0, 2.0]), A.nnz)
    assert _packed(A)[1].sliced() is None
    rows = np.arange(0, n, 32)                              # one long row in every slice
    C = sp.csr_matrix((np.ones(rows.size * 100), (np.repeat(rows, 100), np.tile(np.arange(100), rows.size))), shape=(n, n))
    assert _packed(sp.csr_matrix(C + sp.eye(n)))[1].sliced() is None


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1000, 70001])
def test_sliced_evolution_and_lanczos(cuda, cplx, n):
    """A whole evolution and a Lanczos run on the sliced form against the row
    hand-out forms: the same partition and stopping, states within 1e-13, the
    recurrence's coefficients within 1e-12 of its norm."""
    import torch
    from quspin_gb300 import _lib
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import SLICED, DeviceCSR
    from quspin_gb300.tools import ExpmMultiplyParallel, lanczos_full
    from quspin_gb300.tune import encode
    rng = np.random.default_rng(n + cplx)
    A = _matrix(n, cplx, "even", rng)
    A = sp.csr_matrix(A + A.conj().T)
    A.sum_duplicates()
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    v /= np.linalg.norm(v)
    old, ExpmMultiplyParallel.SMALL_MAX_ROWS = ExpmMultiplyParallel.SMALL_MAX_ROWS, 0
    try:
        out, terms = [], []
        for sliced in (False, True):
            op = ExpmMultiplyParallel(DeviceCSR.from_scipy(A), a=-0.4j)
            P = op.A_device.paired().packed()
            code = encode(2, 2) | (4 << 20)
            if sliced:
                P, code = P.sliced(), encode(2, 2) | SLICED
            op._pick = P
            P.__dict__.setdefault("_tuned", {})[("taylor", 1, _lib.CPF)] = code
            F = D.to_device(v * 1e150)
            op.run_device(F)
            out.append(D.to_host(F) / 1e150)
            terms.append(op.terms_executed)
    finally:
        ExpmMultiplyParallel.SMALL_MAX_ROWS = old
    assert np.linalg.norm(out[1] - out[0]) <= 1e-13 * np.linalg.norm(out[0])
    assert terms[0] == terms[1]
    E = []
    m = 12
    for sliced in (False, True):
        M = DeviceCSR.from_scipy(A)
        P = M.paired().packed()
        key = ("spmv", 1, np.dtype(np.complex128).str, "double", P.vcode)
        M._tuned = {key: encode(2, 1) | (SLICED if sliced else 0)}
        E.append(lanczos_full(M, D.to_device(v), m)[0])
    assert np.abs(E[1] - E[0]).max() <= 1e-12 * np.abs(E[0]).max()


@pytest.mark.parametrize("kind", ["even", "uneven"])
def test_tuned_pick(cuda, kind):
    """At tuned sizes the evolution takes the sliced or the packed form where
    slices apply, else a row hand-out form, with the same result."""
    from quspin_gb300 import _lib
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import DeviceCSR
    from quspin_gb300.tools import ExpmMultiplyParallel
    from quspin_gb300.tune import encode
    rng = np.random.default_rng(3)
    n = 66001
    A = _matrix(n, False, kind, rng)
    if kind == "uneven":                                    # a row of 100 in every slice
        rows = np.arange(0, n, 32)
        A = A + sp.csr_matrix((np.ones(100 * rows.size), (np.repeat(rows, 100), np.tile(np.arange(100) * 7, rows.size))),
                              shape=(n, n))
    A = sp.csr_matrix(A + A.T)
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    v /= np.linalg.norm(v)
    op = ExpmMultiplyParallel(DeviceCSR.from_scipy(A), a=-0.1j)
    op.set_partition(8, 2)
    P, _ = op._operand(1)
    assert (op.A_device.paired().packed().sliced() is None) == (kind == "uneven")
    sliced = (_lib.PF8P, _lib.PF8S)
    assert P.vcode in (sliced if kind == "even" else (_lib.PF8, _lib.PF8P))
    out = D.to_host(op.dot(D.to_device(v)))
    ref = ExpmMultiplyParallel(DeviceCSR.from_scipy(A), a=-0.1j)
    ref.set_partition(8, 2)
    ref._pick = ref.A_device.paired()
    ref._pick.__dict__.setdefault("_tuned", {})[("taylor", 1, _lib.CPF)] = encode(4, 1)
    assert np.linalg.norm(out - D.to_host(ref.dot(D.to_device(v)))) <= 1e-13 * np.linalg.norm(out)


@pytest.mark.parametrize("power", [0, -40, -62, -63, -64, -70, -74, -100])
def test_term_norm_is_the_largest_modulus(cuda, power):
    """The stopping test's norm of a term, bit for bit, however small the term
    is next to its scale: the first half of the rows hold the modulus whose FP32
    square is the larger near 2^-140, the second half the larger one."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import _lib
    from quspin_gb300.sparse import SLICED, SlicedCSR
    from quspin_gb300.tune import encode
    n = 640000                                              # several slices to every warp
    M, P = _packed(sp.identity(n, format="csr"))
    limit, SlicedCSR.MAX_PADDING = SlicedCSR.MAX_PADDING, 40.0
    try:
        S = P.sliced()
    finally:
        SlicedCSR.MAX_PADDING = limit
    small, large = np.float32([1.0064243, 1.0005476]), np.float32([1.0052148, 1.0023396])
    b = np.zeros((n, 4), np.float32)
    b[:n // 2, 0::2], b[n // 2:, 0::2] = small, large
    b0 = D.to_device(b)
    b1, F = torch.empty_like(b0), torch.ones(n, dtype=torch.complex128, device="cuda")
    ctl = torch.zeros(_lib.load().qs_expm_ctl_bytes() // 8 + 1, dtype=torch.int64, device="cuda")
    c = torch.tensor([2.0**power + 0j], dtype=torch.complex128, device="cuda")
    _lib.call("qs_taylor_term", n, S.nnz, D.ptr(S.indptr), 0, D.ptr(S.indices), D.ptr(S.data), S.vcode, D.ptr(b0),
              D.ptr(b1), _lib.CPF, D.ptr(F), 1, 0.0, 0.0, D.ptr(c), 0, 0.0, D.ptr(ctl), encode(2, 2) | SLICED,
              D.stream())
    np.testing.assert_array_equal(D.to_host(b1), b * np.float32(2.0**power))
    h = large.astype(np.float64)
    assert ctl[:1].view(torch.float64).item() == np.sqrt(h[0] * h[0] + h[1] * h[1]) * 2.0**power


@pytest.mark.parametrize("wins", [False, True])
def test_sliced_words_kept_only_where_they_win(cuda, monkeypatch, wins):
    """The words are as large as the packed operand: the tuner, which builds
    them to time them, keeps them for the products and the terms that run on
    them and gives them back otherwise; a second evolution does not build them
    again to find the same."""
    from quspin_gb300 import _device as D
    from quspin_gb300 import tune
    from quspin_gb300.sparse import SLICED, DeviceCSR, SlicedCSR
    from quspin_gb300.tools import ExpmMultiplyParallel
    built, build = [], SlicedCSR.build.__func__
    monkeypatch.setattr(SlicedCSR, "build", classmethod(lambda cls, P: built.append(1) or build(cls, P)))
    clock = [1e3]

    def time(fn, reps=5):                                   # the sliced form is timed last
        fn()
        clock[0] *= 0.99 if wins else 1.01
        return clock[0]
    monkeypatch.setattr(tune, "_time", time)
    rng = np.random.default_rng(5)
    n = 65600
    A = _matrix(n, False, "even", rng)
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    M = DeviceCSR.from_scipy(A)
    P = M.paired().packed()
    y = M.dot(D.to_device(x))                               # small: no float pairs, no tuning
    M.matvec_into(D.to_device(x), y, precision="double")
    assert bool(M._tuned[("spmv", 1, np.dtype(np.complex128).str, "double", P.vcode)] & SLICED) == wins
    assert ("_sliced" in P.__dict__) == wins and len(built) == 1
    assert np.all(abs(D.to_host(y) - A @ x) <= 1e-13 * (abs(A) @ abs(x)))
    M = DeviceCSR.from_scipy(A)
    P = M.paired().packed()
    built.clear()
    for _ in range(2):
        op = ExpmMultiplyParallel(M, a=-0.1j)
        op.set_partition(6, 1)
        assert (op._operand(1)[0] is P.__dict__.get("_sliced")) == wins
    assert ("_sliced" in P.__dict__) == wins and len(built) == 1


@pytest.mark.parametrize("what", ["packed", "sliced", "pointers"])
def test_forms_without_memory(cuda, monkeypatch, what):
    """No memory for the packed words, the sliced words or the slice pointers:
    the operand of before serves, for one vector and several."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300 import sparse
    from quspin_gb300.sparse import DeviceCSR
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(6)
    n = 65600
    A = _matrix(n, False, "even", rng)
    M = DeviceCSR.from_scipy(A)
    P = M.paired()
    V = rng.normal(size=(n, 3)) + 1j * rng.normal(size=(n, 3))
    op = ExpmMultiplyParallel(DeviceCSR.from_scipy(A), a=-0.1j)
    op.set_partition(6, 1)
    want = [D.to_host(op.dot(D.to_device(v))) for v in (V[:, 0].copy(), V)]

    class Full:                                             # the allocations of the class under test fail
        OutOfMemoryError = torch.OutOfMemoryError
        def __getattr__(self, name):
            if name == {"packed": "zeros", "sliced": "empty", "pointers": "zeros"}[what]:
                return self.fail
            return getattr(torch, name)
        @staticmethod
        def fail(*a, dtype=None, **k):
            if dtype is {"packed": torch.int32, "sliced": torch.int32, "pointers": torch.int64}[what] and a[0] > 1:
                raise torch.OutOfMemoryError("no memory")
            return getattr(torch, {"packed": "zeros", "sliced": "empty", "pointers": "zeros"}[what])(*a, dtype=dtype, **k)
    op = ExpmMultiplyParallel(M, a=-0.1j)
    op.set_partition(6, 1)
    monkeypatch.setattr(sparse, "torch", Full())
    got = [D.to_host(op.dot(D.to_device(v))) for v in (V[:, 0].copy(), V)]
    assert (P.packed() is None) == (what == "packed")
    assert what == "packed" or P.packed().sliced() is None
    for g, w in zip(got, want):
        assert np.linalg.norm(g - w) <= 1e-13 * np.linalg.norm(w)
    y = torch.empty(n, dtype=torch.complex128, device="cuda")
    M.matvec_into(D.to_device(V[:, 0].copy()), y, precision="double")
    assert np.all(abs(D.to_host(y) - A @ V[:, 0]) <= 1e-13 * (abs(A) @ abs(V[:, 0])))


def test_tuner_times_every_shape_of_smaller_operands(cuda, monkeypatch):
    """Below the row counts from which the sliced form always leads, it is
    timed against all row hand-out shapes of the packed operand; from there on
    against a few of them."""
    from quspin_gb300 import _lib, tune
    from quspin_gb300.sparse import DeviceCSR
    n = 65600
    A = _matrix(n, False, "even", np.random.default_rng(7))
    timed = []
    monkeypatch.setattr(tune, "_time", lambda fn, reps=5: timed.append(1) or 1.0)
    count = {}
    for few in (False, True):
        monkeypatch.setattr(tune, "FEW_ROWS_PRODUCT", n + (not few))
        monkeypatch.setattr(tune, "FEW_ROWS_TERM", n + (not few))
        M = DeviceCSR.from_scipy(A)
        P = M.paired().packed()
        for xdtype in (np.complex128, np.float64):
            timed.clear()
            tune.tune_spmv(M, 1, xdtype, "double", operand=P)
            count[few, xdtype] = len(timed)
        timed.clear()
        tune.tune_taylor(P, 1, _lib.CPF)
        count[few, "term"] = len(timed)
    full = len(tune._candidates(n, A.nnz, 1))
    assert count[False, np.complex128] == full + 3 and count[False, np.float64] == full + 1
    assert count[True, np.complex128] == 3 and count[True, np.float64] == 5
    assert count[False, "term"] == len(tune.r32_candidates(P, 1, _lib.CPF)) and count[True, "term"] == 3
