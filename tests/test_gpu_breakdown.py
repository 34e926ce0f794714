"""FP64 bases that end early (an invariant subspace), in a cluster and in a
grid: every block takes the step for the basis's last one, and nothing of it
is left for the next basis of the same or another solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 5000, 20001, 150001])
@pytest.mark.parametrize("reortho", [1, 0])
def test_repeated_breakdowns_leave_nothing_behind(n, reortho):
    import scipy.sparse as sp

    from mexk import synthetic as S
    from mexk.api import Context

    # tridiagonal but for five rows that only see one another
    d = -1.0 - np.arange(n) / n
    off = np.full(n - 1, 0.25)
    c = n // 2
    off[[c - 1, c + 4]] = 0.0
    M = sp.lil_matrix(sp.diags([off, d, off], [-1, 0, 1]))
    M[c, c + 4] = 0.5
    M = M.tocsr()
    M.eliminate_zeros()
    M.sort_indices()
    A = S.CSR(n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
    few = np.zeros(n)
    few[c] = 2.0
    ref, term = few.copy(), few.copy()
    for i in range(1, 40):
        term = (1.0 / i) * (M @ term)
        ref += term
    v = np.random.default_rng(n).standard_normal(n)
    with Context(A, m_alloc=20) as ctx:
        full, _ = ctx.expmv(v, 1.0, 20, reorthogonalize=bool(reortho))
        first, res = ctx.expmv(few, 1.0, 20, reorthogonalize=bool(reortho))
        assert res["converged"] == 1 and max(s[3] for s in ctx.steps()) == 5
        assert np.linalg.norm(first - ref) <= 1e-12 * np.linalg.norm(ref)
        for _ in range(20):
            assert np.array_equal(ctx.expmv(few, 1.0, 20, reorthogonalize=bool(reortho))[0], first)
            assert np.array_equal(ctx.expmv(v, 1.0, 20, reorthogonalize=bool(reortho))[0], full)
