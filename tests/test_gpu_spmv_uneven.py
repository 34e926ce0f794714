"""The direct FP64 SpMV on matrices with rows longer than one thread sums (its
rows by length): bit for bit the staged form's, whose rows go in matrix order;
tiles of empty rows, of rows of all lengths around 64, of one long row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["mixed", "empty", "steps", "powerlaw"])
def test_rows_by_length_are_bitwise_the_staged_rows(kind):
    import scipy.sparse as sp

    from mexk import synthetic as S
    from mexk.api import Context

    n = 90001
    rng = np.random.default_rng(11)
    if kind == "mixed":
        lengths = rng.integers(0, 130, n)
    elif kind == "empty":
        lengths = np.where(rng.random(n) < 0.02, 200, 0)
    elif kind == "steps":
        lengths = np.arange(n) % 67
        lengths[n // 2] = 3000
    else:
        lengths = None
    if lengths is None:
        A = S.power_law(n, seed=3)
    else:
        rows = np.repeat(np.arange(n), lengths)
        M = sp.csr_matrix((rng.uniform(-1, 1, len(rows)), (rows, rng.integers(0, n, len(rows)))), shape=(n, n))
        M.sum_duplicates()
        M.sort_indices()
        A = S.CSR(n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
    v = rng.standard_normal(n)
    t = 1e-3 / A.max_abs()
    with Context(A, m_alloc=5) as ctx:
        assert ctx.spmv_form("fp64") == "direct"
        a, _ = ctx.expmv(v, t, 5)
        Va = ctx.get_basis(6)
        ctx.set_spmv_form("staged")
        b, _ = ctx.expmv(v, t, 5)
        Vb = ctx.get_basis(6)
    assert np.array_equal(Va, Vb) and np.array_equal(a, b)
