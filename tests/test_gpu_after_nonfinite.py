"""A solve with a non-finite vector leaves nothing behind where the FP64 basis
keeps w in memory (more than 3.4 million rows): the next solve and the next
step on the same context give the bits they gave before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tridiagonal(n, symmetric):
    """Random values: no row patterns, so the context's SpMV takes the products."""
    from mexk import synthetic as S

    rng = np.random.default_rng(n)
    vals = np.empty((n, 3))
    vals[:, 1] = -2.0 + 0.1 * rng.uniform(size=n)
    vals[:, 2] = rng.uniform(0.5, 1.0, n)
    vals[1:, 0] = vals[:-1, 2] if symmetric else rng.uniform(0.5, 1.0, n - 1)
    cols = np.arange(n)[:, None] + np.array([-1, 0, 1])
    keep = (cols >= 0) & (cols < n)
    rp = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(keep.sum(axis=1), out=rp[1:])
    return S.CSR(n, rp, cols[keep].astype(np.int32), vals[keep])


@pytest.mark.parametrize("kind,window,reortho", [("tridiagonal", 0, 1), ("tridiagonal", 0, 0), ("tridiagonal", 2, 1),
                                                 ("tridiagonal", 2, 0), ("tridiagonal", 3, 1), ("heat", 0, 1),
                                                 ("heat", 2, 1)])
def test_next_solve_and_step_are_unchanged(kind, window, reortho):
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.laplacian_2d(1851) if kind == "heat" else tridiagonal(3450003, window > 0)
    assert A.n > 3423000 and A.n % 64 != 0
    v = np.random.default_rng(6).standard_normal(A.n)
    t = 0.05 / A.max_abs()
    with Context(A, m_alloc=6) as ctx:
        def solve(x):
            return ctx.expmv(x, t, 5, window=window, reorthogonalize=bool(reortho))

        def step():
            ctx.set_basis((v / np.linalg.norm(v))[None])
            return ctx.arnoldi_step(0)

        y, res = solve(v)
        ok, h, beta = step()
        assert ok and y.any() and res["converged"] == 1
        for bad in (np.nan, np.inf):
            w = v.copy()
            w[A.n - 1] = bad
            assert not solve(w)[0].any()
            ok2, h2, beta2 = step()
            assert ok2 and np.array_equal(h, h2) and beta == beta2
            assert not solve(w)[0].any()
            assert np.array_equal(solve(v)[0], y)
