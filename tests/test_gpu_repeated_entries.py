"""Matrices that store a column of a row twice (unsummed assemblies): every
entry counts, in each form of the window-2 basis in mixed precision (up to
8,192 rows and beyond, where the recurrence stays on chip)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(N, kind):
    """A 5-point grid of N^2 rows. halves: the diagonal stored as two equal
    entries; some: on every 13th row a second entry equal to the diagonal's;
    last: as halves, the second one after the row's other entries."""
    from mexk import synthetic as S

    A = S.laplacian_2d(N)
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    cols, vals = A.col_idx.astype(np.int64), A.values.copy()
    diag = rows == cols
    if kind != "some":
        vals[diag] *= 0.5
    again = diag & (rows % 13 == 5) if kind == "some" else diag
    rows, cols = np.concatenate([rows, rows[again]]), np.concatenate([cols, cols[again]])
    vals = np.concatenate([vals, vals[again]])
    late = np.arange(len(rows)) >= A.nnz
    order = np.lexsort((cols, late, rows)) if kind == "last" else np.lexsort((cols, rows))
    rp = np.zeros(A.n + 1, dtype=np.int32)
    np.cumsum(np.bincount(rows, minlength=A.n), out=rp[1:])
    return S.CSR(A.n, rp, cols[order].astype(np.int32), vals[order])


@pytest.mark.parametrize("N", [90, 131, 301])
@pytest.mark.parametrize("kind", ["halves", "some", "last"])
def test_every_entry_counts(N, kind):
    import scipy.sparse as sp

    from mexk.api import Context

    A = grid(N, kind)
    v = np.random.default_rng(N).standard_normal(A.n)
    M = sp.csr_matrix((A.values, A.col_idx, A.row_ptr), shape=(A.n, A.n), copy=True)
    M.sum_duplicates()  # in place: of the copy
    t = 0.5 / abs(M).sum(axis=1).max()
    ref, term = v.copy(), v.copy()
    for i in range(1, 24):
        term = (t / i) * (M @ term)
        ref += term
    with Context(A, m_alloc=30) as ctx:
        assert ctx.spmv_form("mixed") == "pattern"
        y, res = ctx.expmv(v, t, 30, precision="mixed", controller="search", window=2)
    assert res["converged"] == 1
    assert np.linalg.norm(y - ref) <= 1e-6 * np.linalg.norm(ref)  # the mixed form's bound
