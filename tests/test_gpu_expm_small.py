"""The one-launch evolution of small problems (csrc/expm_small.cu) against the
launch per term on the same operand: sizes around a block's and a sweep's rows,
real and complex, coded and plain values, one and several substeps, a
substep that runs out of terms, a zero matrix and repeated calls on the same
scratch; and against scipy.

Tolerance: the same float-pair arithmetic with the row sums split over another
number of lanes: 48-bit rounding, at most a few hundred terms."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import expm_multiply

pytestmark = pytest.mark.gpu


def _hermitian(n, cplx, coded, rng):
    A = sp.random(n, n, density=min(1.0, 6.0 / n), random_state=rng, format="csr")
    A.data = rng.choice(np.array([0.5, -1.0, 0.25]), A.nnz) if coded else rng.normal(size=A.nnz)
    if cplx:
        A = A.astype(complex)
        A.data = A.data * rng.choice(np.array([1.0, 1j]), A.nnz)
    A = sp.csr_matrix(A + A.conj().T + sp.diags(rng.choice(np.array([-0.5, 1.0]), n)))
    A.sum_duplicates()
    return A


@pytest.mark.parametrize("n", [1, 2, 31, 255, 4751, 19457, 65535])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("coded", [False, True])
def test_small_matches_launch_per_term(cuda, n, cplx, coded):
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(n + 2 * cplx + coded)
    A = _hermitian(n, cplx, coded, rng)
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    scale = 10.0 ** rng.integers(-200, 200)
    u = v / np.linalg.norm(v)
    v = u * scale
    for t in (0.02, 1.7):
        op = ExpmMultiplyParallel(A, a=-1j * t)
        assert op._small_operand() is not None and op._small_operand().coded == (coded or n <= 31)
        one = D.to_host(op.dot(D.to_device(v)))
        terms, missed = op.terms_executed, op.nonconverged_substeps
        np.testing.assert_array_equal(one, D.to_host(op.dot(D.to_device(v))))       # the scratch is left as it was
        ExpmMultiplyParallel.SMALL_MAX_ROWS, old = 0, ExpmMultiplyParallel.SMALL_MAX_ROWS
        try:
            ref = D.to_host(op.dot(D.to_device(v)))
        finally:
            ExpmMultiplyParallel.SMALL_MAX_ROWS = old
        one, ref = one / scale, ref / scale                    # norms of 1e200 overflow when squared
        assert np.linalg.norm(one - ref) <= 1e-13 * np.linalg.norm(ref)
        assert abs(terms - op.terms_executed) <= op.s and missed == op.nonconverged_substeps
        if n <= 4751:
            exact = expm_multiply(-1j * t * A, u)
            assert np.linalg.norm(one - exact) <= 1e-12 * np.linalg.norm(exact)


def test_small_edges(cuda):
    """A substep cut off after three terms is counted; m* = 0 and a zero
    matrix leave the state; a NaN stays a NaN and the next call is clean."""
    from quspin_gb300 import _device as D
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(1)
    n = 1000
    A = _hermitian(n, False, True, rng)
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    op = ExpmMultiplyParallel(A, a=-1j)
    full = op.dot(v)
    op.set_partition(3, 4)
    cut = op.dot(v)
    assert op.nonconverged_substeps == 4 and op.terms_executed == 12
    B, F = None, v.copy()
    mu = A.diagonal().mean()
    for _ in range(4):
        B = F
        for j in range(3):
            B = -1j / (4 * (j + 1)) * (A @ B - mu * B)
            F = F + B if j else F + B
        F = F * np.exp(-1j * mu / 4)
    assert np.linalg.norm(cut - F) <= 1e-12 * np.linalg.norm(F)
    w = v.copy()
    w[3] = np.nan
    assert np.isnan(op.dot(w)).any()
    op._calculate_partition()
    np.testing.assert_array_equal(op.dot(v), full)
    Z = ExpmMultiplyParallel(sp.csr_matrix((n, n)), a=-1j)
    assert Z.m_star == 0
    np.testing.assert_allclose(Z.dot(v), v, rtol=0, atol=0)
    assert D.to_device(v).shape == (n,)


@pytest.mark.parametrize("row,one", [(39, True), (41, False)])
def test_small_form_by_entries(cuda, row, one):
    """Many entries in few rows go to the launch per term: its rule counts
    both, and the two agree."""
    from quspin_gb300 import _device as D
    from quspin_gb300.sparse import DeviceCSR
    from quspin_gb300.tools import ExpmMultiplyParallel
    n = 60000
    rng = np.random.default_rng(row)
    cols = (np.arange(n)[:, None] + rng.choice(n, row, replace=False)[None, :]) % n
    A = sp.csr_matrix((rng.choice(np.array([0.5, -1.0, 0.25]), n * row) / row, np.sort(cols, axis=1).ravel(),
                       np.arange(n + 1) * row), shape=(n, n))
    op = ExpmMultiplyParallel(DeviceCSR.from_scipy(A), a=-0.5j)
    assert (op._small_operand() is not None) == one
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    got = op.dot(D.to_device(v))
    old = ExpmMultiplyParallel.SMALL_MAX_NNZ
    ExpmMultiplyParallel.SMALL_MAX_NNZ = 0 if one else 1 << 30
    try:
        ref = op.dot(D.to_device(v))
    finally:
        ExpmMultiplyParallel.SMALL_MAX_NNZ = old
    assert float((got - ref).norm() / ref.norm()) <= 1e-13


@pytest.mark.parametrize("n", [200, 20000])
def test_small_barrier_gives_up(cuda, monkeypatch, n):
    """Barriers that may not look even once: the kernel ends by itself, F is NaN
    as a whole, the counters raise, settle and host results evolve the kept
    input launch by launch, and the next call is clean."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300._lib import QsError
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(n)
    A = _hermitian(n, True, True, rng)
    v = rng.normal(size=n) + 1j * rng.normal(size=n)
    op = ExpmMultiplyParallel(A, a=-0.7j)
    want = D.to_host(op.dot(D.to_device(v)))
    assert not op.gave_up
    terms = op.terms_executed
    monkeypatch.setattr(ExpmMultiplyParallel, "SMALL_POLLS", 0)
    F = D.to_device(v).clone()
    assert op.dot(F, overwrite_v=True) is F and op.gave_up
    assert bool(torch.isnan(torch.view_as_real(F)).all())
    for name in ("terms_executed", "nonconverged_substeps"):
        with pytest.raises(QsError, match="gave up"):
            getattr(op, name)
    assert op.settle(F) is F and not op.gave_up
    assert np.linalg.norm(D.to_host(F) - want) <= 1e-13 * np.linalg.norm(want)
    assert abs(op.terms_executed - terms) <= op.s
    host = op.dot(v)                                       # read back: settled by itself
    assert np.linalg.norm(host - want) <= 1e-13 * np.linalg.norm(want)
    monkeypatch.setattr(type(op), "partition_source", property(lambda self: "learned"))
    F = op.run_device(D.to_device(v).clone())              # the learned selection reads its counter
    assert np.linalg.norm(D.to_host(F) - want) <= 1e-13 * np.linalg.norm(want)
    monkeypatch.undo()
    np.testing.assert_array_equal(D.to_host(op.dot(D.to_device(v))), want)
    assert not op.gave_up and op.terms_executed == terms


@pytest.mark.parametrize("n", [300, 30000])
def test_small_uses_the_callers_work_array(cuda, n):
    """A device work_array of the result's type holds the term vectors of the
    one-launch form, as it does those of the other forms."""
    import torch
    from quspin_gb300 import _device as D
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(n)
    op = ExpmMultiplyParallel(_hermitian(n, False, True, rng), a=-0.7j)
    assert op._small_operand() is not None
    v = D.to_device(rng.normal(size=n) + 1j * rng.normal(size=n))
    want = op.dot(v)
    for shape in ((2 * n,), (2, n)):
        work = torch.full(shape, np.pi, dtype=torch.complex128, device="cuda")
        assert torch.equal(op.dot(v, work_array=work), want)
        assert not bool((work == np.pi).any())
    with pytest.raises(ValueError, match="twice"):
        op.dot(v, work_array=work[0])


def test_small_buffers_outlive_other_calls(cuda):
    """What a launch of the one-launch form reads and writes is not freed by
    later calls of the same object, which another stream may issue while it
    runs: a call with several vectors, or with another factor."""
    from quspin_gb300 import _device as D
    from quspin_gb300.tools import ExpmMultiplyParallel
    rng = np.random.default_rng(3)
    n = 50000
    op = ExpmMultiplyParallel(_hermitian(n, False, True, rng), a=-0.5j)
    op.GRAPH_MAX_ELEMS = 0
    v = D.to_device(rng.normal(size=n) + 1j * rng.normal(size=n))
    want = op.dot(v)
    held = [t.data_ptr() for t in (*op._small_state, op._keep, op._small_work, *op._small_consts.values())]
    op.dot(v.reshape(n, 1).expand(n, 3).contiguous())
    op.set_a(-0.25j)
    op.dot(v)
    op.set_a(-0.5j)
    assert bool((op.dot(v) == want).all())
    now = [t.data_ptr() for t in (*op._small_state, op._keep, op._small_work, *op._small_consts.values())]
    assert now[:len(held)] == held
    for i in range(op.SMALL_TABLES + 3):
        op.set_a(-0.01j * (i + 1))
        op.dot(v)
    assert len(op._small_consts) <= op.SMALL_TABLES
