"""The one-launch FP64 basis against the step-by-step kernels, from the same
first column: bit for bit where the sums keep their order (even n up to 4096,
at most 32 columns), to rounding beyond; around the edges of sub-blocks (64
rows), blocks, the cluster (4096 rows) and the grid, for each form of the
product, with and without reorthogonalisation and with a window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(kind, n):
    from mexk import synthetic as S

    if kind == "heat":
        return S.laplacian_2d(n)
    if kind == "powerlaw":
        return S.power_law(n, seed=n)
    if kind == "longrow":  # one row longer than a tile of the product
        A = S.random_diag_dominant(n, 3, seed=n)
        rows = [A.col_idx[A.row_ptr[i]:A.row_ptr[i + 1]] for i in range(n)]
        vals = [A.values[A.row_ptr[i]:A.row_ptr[i + 1]] for i in range(n)]
        rows[7] = np.arange(n, dtype=np.int32)
        vals[7] = np.random.default_rng(1).uniform(-1, 1, n) / n
        rp = np.zeros(n + 1, dtype=np.int32)
        np.cumsum([len(r) for r in rows], out=rp[1:])
        return S.CSR(n, rp, np.concatenate(rows).astype(np.int32), np.concatenate(vals))
    return S.random_diag_dominant(n, 8, seed=n)


CASES = [("random", n, 12, 1, 0) for n in (14, 64, 65, 130, 1000, 2047, 2048, 4094, 4095, 4096, 4097, 4160, 9728, 9729,
                                          20011)]
CASES += [("random", 2000, 32, 1, 0), ("random", 2000, 64, 1, 0), ("random", 6001, 100, 1, 0),
          ("random", 3000, 20, 0, 0), ("random", 30000, 20, 0, 0), ("random", 210000, 9, 1, 0),
          ("powerlaw", 2048, 20, 1, 0), ("powerlaw", 12345, 20, 1, 0), ("longrow", 3000, 8, 1, 0),
          ("longrow", 6000, 8, 1, 0), ("heat", 40, 30, 1, 0), ("heat", 64, 30, 1, 2), ("heat", 64, 20, 0, 3),
          ("heat", 131, 17, 1, 0), ("heat", 131, 30, 1, 2), ("heat", 301, 30, 1, 4)]
# sweeps on digit columns (rows x allocated columns >= 3 million): full and window, one and two rows per thread,
# own product and the SpMV's, every group size
CASES += [("random", 300011, 10, 1, 0), ("random", 150003, 23, 1, 0), ("random", 40007, 75, 1, 0),
          ("random", 150003, 20, 0, 0), ("powerlaw", 160001, 19, 1, 0), ("heat", 601, 17, 1, 0),
          ("heat", 601, 30, 1, 6)]
# a window of 2 in three passes (256 rows a block or more), w on chip and not
CASES += [("heat", 198, 30, 1, 2), ("heat", 301, 30, 1, 2), ("heat", 777, 20, 0, 2), ("heat", 1851, 6, 1, 2)]


@pytest.mark.parametrize("kind,n,m,reortho,window", CASES)
def test_basis_matches_stepwise(kind, n, m, reortho, window):
    from mexk.api import Context

    A = make(kind, n)
    n = A.n
    v = np.random.default_rng(n).standard_normal(n)
    t = 1e-3 / A.max_abs()  # one accepted step: the context keeps that cycle's basis
    with Context(A, m_alloc=m) as ctx:
        y, res = ctx.expmv(v, t, m, reorthogonalize=bool(reortho), window=window)
        assert res["cycles"] == 1
        V = ctx.get_basis(m + 1)
        ctx.set_basis(V[:1])
        if window:
            W = V  # the stepping API has no window: check the recurrence itself
        else:
            for j in range(m):
                assert ctx.arnoldi_step(j, reorthogonalize=bool(reortho))[0]
            W = ctx.get_basis(m + 1)
    if window:
        # neighbours within the window orthonormal to rounding, and A v_j in the span of the window
        import scipy.sparse as sp

        M = sp.csr_matrix((A.values, A.col_idx, A.row_ptr), shape=(n, n))
        for j in range(1, m):
            lo = max(0, j + 1 - window)
            G = V[lo:j + 2] @ V[lo:j + 2].T
            assert np.abs(G - np.eye(len(G))).max() < (1e-12 if reortho else 1e-8)
            w = M @ V[j]
            r = w - V[lo:j + 2].T @ (V[lo:j + 2] @ w)
            assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(w)
        return
    if n <= 4096 and n % 2 == 0 and (m <= 32 or n <= 2048):
        assert np.array_equal(V, W)
    elif reortho:
        # two bases of the same recurrence rounded in different orders: the bound of the oracle comparison
        assert np.abs(V - W).max() < 1e-12
    else:
        # one Gram-Schmidt pass amplifies rounding by |w| / h(j+1, j) each step, so two bases drift apart;
        # the result does not (the FP64 bound of the parity tests)
        import scipy.sparse as sp

        M = sp.csr_matrix((A.values, A.col_idx, A.row_ptr), shape=(n, n))
        ref, term = v.copy(), v.copy()
        for i in range(1, 12):  # |tA| < 0.02
            term = (t / i) * (M @ term)
            ref += term
        assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("n,m", [(150001, 21), (40007, 80)])
def test_localised_vector_keeps_fp64_orthogonality(n, m):
    """One large entry and a tail 1e-9 of it: digits share an exponent over a
    block's rows, and the basis stays orthonormal to the bound FP64 is held to."""
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.random_diag_dominant(n, 8, seed=3)
    v = 1e-9 * np.random.default_rng(4).standard_normal(n)
    v[n // 3] = 1.0
    with Context(A, m_alloc=m) as ctx:
        _, res = ctx.expmv(v, 1e-3 / A.max_abs(), m)
        assert res["cycles"] == 1
        V = ctx.get_basis(m)
    assert np.abs(V @ V.T - np.eye(m)).max() < 1e-13


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n,m", [(6000, 20), (150001, 21)])
def test_non_finite_vector_breaks_down_at_once(n, m, bad):
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.random_diag_dominant(n, 8, seed=5)
    v = np.random.default_rng(6).standard_normal(n)
    with Context(A, m_alloc=m) as ctx:
        y_ok, _ = ctx.expmv(v, 0.1, m)
        w = v.copy()
        w[n - 3] = bad
        y, res = ctx.expmv(w, 0.1, m)
        steps = ctx.steps()
        y2, _ = ctx.expmv(v, 0.1, m)
    assert not y.any() and res["converged"] == 1 and res["cycles"] == 1 and steps[0][3] == 1
    assert np.array_equal(y_ok, y2)  # nothing of the failed solve is left behind
