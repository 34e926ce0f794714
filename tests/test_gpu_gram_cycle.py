"""The one-launch FP32 basis (rows on chip, Gram-corrected steps) around the
edges of its sub-blocks (128 rows), blocks (32), the cluster (4096 to 8192
rows) and the grid, with columns on and off chip, for each form of the product, with and
without reorthogonalisation and with a window.

With u = 2^-24, rows of at most 64 entries and at most 64 columns, one step's
rounding is bounded by (64 + 64 + 4) u ||A||v_j||: the product's and the
update's sums. That bounds A v_j's distance from the span of the columns; the
loss of orthogonality is the same divided by what the projection leaves of
A v_j."""
import numpy as np
import pytest

from test_gpu_arnoldi_cycle import make as make_general

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def make(kind, n):
    """heat3d: a 7-point stencil on n^3 points. patches: a 5-point one on n^2 with another
    diagonal on some rows (patterns that are no part of the main one)."""
    import scipy.sparse as sp

    from mexk import synthetic as S

    if kind not in ("heat3d", "patches"):
        return make_general(kind, n)
    T = sp.diags([np.ones(n - 1), np.full(n, -2.0), np.ones(n - 1)], [-1, 0, 1])
    one = sp.identity(n)
    if kind == "heat3d":
        M = sp.kron(sp.kron(T, one), one) + sp.kron(sp.kron(one, T), one) + sp.kron(sp.kron(one, one), T)
    else:
        M = sp.kron(T, one) + sp.kron(one, T) - sp.diags(np.random.default_rng(n).integers(0, 12, n * n) // 11 * 0.5)
    M = sp.csr_matrix(M)
    M.sort_indices()
    return S.CSR(M.shape[0], M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)

CASES = [("random", n, 12, 1, 0) for n in (14, 64, 129, 511, 512, 513, 2000, 2047, 4095, 4096, 4097, 4865, 9729, 20011)]
CASES += [("random", 2000, 1, 1, 0), ("random", 2000, 33, 1, 0), ("random", 2000, 64, 1, 0), ("random", 9000, 64, 1, 0),
          ("random", 2000, 20, 0, 0), ("random", 30000, 9, 0, 0), ("random", 120001, 30, 1, 0),
          ("random", 300007, 40, 1, 0), ("powerlaw", 2048, 20, 1, 0), ("powerlaw", 12345, 20, 1, 0),
          ("longrow", 2000, 8, 1, 0), ("longrow", 6000, 8, 1, 0), ("heat", 7, 30, 1, 0), ("heat", 64, 30, 1, 3),
          ("heat", 64, 20, 0, 3), ("heat", 131, 17, 1, 0), ("heat", 131, 30, 1, 5), ("heat", 401, 40, 1, 0)]
# the cluster's end: 8192 rows, 90,000 CSR entries, no long rows
CASES += [("random", 8192, 12, 1, 0), ("random", 8193, 12, 1, 0), ("random", 9000, 40, 1, 0), ("random", 7001, 64, 1, 0),
          ("powerlaw", 6001, 20, 1, 0), ("heat", 90, 40, 1, 0), ("heat", 91, 40, 1, 0), ("heat", 90, 30, 1, 2),
          ("heat", 91, 30, 1, 2)]
# a window of 2 in the row-pattern form: the recurrence on chip past 4096 rows (blocks of one edge, of two, with
# row groups between them; a stencil that reaches past the edges)
CASES += [("heat", N, 30, 1, 2) for N in (64, 65, 97, 131, 556, 700, 801, 1303)]
CASES += [("heat", 300, 2, 1, 2), ("heat", 300, 64, 1, 2), ("heat", 801, 20, 0, 2), ("heat3d", 31, 20, 1, 2),
          ("heat3d", 40, 20, 1, 2), ("heat3d", 100, 20, 1, 2), ("patches", 150, 20, 1, 2), ("patches", 801, 20, 1, 2)]


@pytest.mark.parametrize("kind,n,m,reortho,window", CASES)
def test_basis(kind, n, m, reortho, window):
    import scipy.sparse as sp

    from mexk.api import Context

    A = make(kind, n)
    n = A.n
    v = np.random.default_rng(n).standard_normal(n)
    t = 1e-3 / A.max_abs()  # one accepted step: the context keeps that cycle's basis
    with Context(A, m_alloc=m) as ctx:
        y, res = ctx.expmv(v, t, m, precision="mixed", controller="search", reorthogonalize=bool(reortho),
                           window=window)
        assert res["cycles"] == 1
        V = ctx.get_basis(m + 1, "mixed")
        y2, _ = ctx.expmv(v, t, m, precision="mixed", controller="search", reorthogonalize=bool(reortho),
                          window=window)
    assert np.array_equal(y, y2)
    M = sp.csr_matrix((A.values, A.col_idx, A.row_ptr), shape=(n, n))
    longest = int(np.diff(A.row_ptr).max())
    step = (min(longest, 64) + longest // 32 + m + 4) * U
    for j in range(m):
        lo = max(0, j + 1 - window) if window else 0
        B = V[lo:j + 2]
        w = M @ V[j]
        size = np.linalg.norm(abs(M) @ np.abs(V[j]))
        coef = np.linalg.lstsq(B.T, w, rcond=None)[0]
        assert np.linalg.norm(w - B.T @ coef) <= step * size
        left = abs(coef[-1])
        loss = np.abs(B @ B.T - np.eye(len(B)))[-1].max()
        if reortho:
            assert loss <= 4 * U + step * size / left, j
    if m <= 2:
        return  # one or two columns do not reach the bound below
    ref, term = v.copy(), v.copy()
    for i in range(1, 12):  # |tA| < 0.1
        term = (t / i) * (M @ term)
        ref += term
    assert np.linalg.norm(y - ref) <= 1e-6 * np.linalg.norm(ref)  # the mixed form's bound


@pytest.mark.parametrize("n", [3000, 6000])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_vector_breaks_down_at_once(n, bad):
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.random_diag_dominant(n, 8, seed=5)
    v = np.random.default_rng(6).standard_normal(n)
    with Context(A, m_alloc=20) as ctx:
        good, _ = ctx.expmv(v, 0.1, 20, precision="mixed", controller="search")
        w = v.copy()
        w[n // 2] = bad
        try:
            y, _ = ctx.expmv(w, 0.1, 20, precision="mixed", controller="search")
            assert not np.isfinite(y).all()
        except Exception:
            pass
        again, _ = ctx.expmv(v, 0.1, 20, precision="mixed", controller="search")
    assert np.array_equal(good, again)


@pytest.mark.parametrize("n", [2000, 6000])
def test_invariant_subspace_breaks_down(n):
    """A = diag + a cycle of five rows; a start vector inside them spans five columns."""
    import scipy.sparse as sp

    from mexk import synthetic as S
    from mexk.api import Context

    M = sp.lil_matrix((n, n))
    M.setdiag(-1.0)
    for i in range(5):
        M[n // 2 + i, n // 2 + (i + 1) % 5] = 0.5
    M = M.tocsr()
    M.sort_indices()
    A = S.CSR(n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
    v = np.zeros(n)
    v[n // 2] = 2.0
    with Context(A, m_alloc=20) as ctx:
        y, _ = ctx.expmv(v, 1.0, 20, precision="mixed", controller="search")
    ref, term = v.copy(), v.copy()
    for i in range(1, 40):
        term = (1.0 / i) * (M @ term)
        ref += term
    assert np.linalg.norm(y - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("kind,window", [("random", 0), ("heat", 2)])
def test_wait_that_runs_out_reports_and_the_context_survives(kind, window):
    """Block 0 leaves before the first meeting: the others' waits end, the solve
    reports it, and the same context then solves as before."""
    from mexk._lib import MexkError, check, lib
    from mexk.api import Context

    A = make(kind, 300 if kind == "heat" else 20000)
    v = np.random.default_rng(8).standard_normal(A.n)
    t = 1.0 / A.max_abs()
    with Context(A, m_alloc=20) as ctx:
        good, _ = ctx.expmv(v, t, 20, precision="mixed", controller="search", window=window)
        check(lib().mexk_test_force_wait_timeout(0, 1))
        try:
            with pytest.raises(MexkError, match="device wait gave up"):
                ctx.expmv(v, t, 20, precision="mixed", controller="search", window=window)
        finally:
            check(lib().mexk_test_force_wait_timeout(0, 0))
        again, _ = ctx.expmv(v, t, 20, precision="mixed", controller="search", window=window)
    assert np.array_equal(good, again)


@pytest.mark.parametrize("kind,n,precision,window,one", [("random", 2000, "fp64", 0, True), ("random", 2000, "mixed", 0, True),
                                                         ("heat", 300, "mixed", 2, True), ("random", 300007, "mixed", 0, False),
                                                         ("random", 300007, "fp64", 0, False)])
def test_basis_launches_and_profile(kind, n, precision, window, one):
    from mexk.api import Context

    A = make(kind, n)
    v = np.random.default_rng(2).standard_normal(A.n)
    ctrl = "reference" if precision == "fp64" else "search"
    with Context(A, m_alloc=20) as ctx:
        ctx.expmv(v, 1e-3 / A.max_abs(), 20, precision=precision, controller=ctrl, window=window)
        assert (ctx.basis_launches(20, precision, window) == 1) == one
        assert ctx.basis_launches(5, precision, window) <= ctx.basis_launches(20, precision, window)
        t5, t20 = (ctx.profile_kernel("basis", j, 3, precision) for j in (4, 19))
        assert 0.0 < t5 < t20 < 50.0


def test_contexts_in_threads_share_the_gpu():
    """Cooperative, cluster and tensor-memory bases of several contexts at once: every
    thread gets the bits it gets alone."""
    import threading

    from mexk.api import Context

    jobs = []
    for i, (kind, n, kw) in enumerate([("random", 20000, {}), ("random", 60000, dict(precision="mixed", controller="search")),
                                       ("heat", 300, dict(precision="mixed", controller="search", window=2)),
                                       ("heat", 120, dict(window=2)), ("random", 3000, {}),
                                       ("heat", 500, dict(precision="mixed", controller="search", window=2))]):
        A = make(kind, n)
        jobs.append((A, 0.5 / A.max_abs(), kw, np.random.default_rng(i).uniform(0, 1, A.n)))
    alone = []
    for A, t, kw, v in jobs:
        with Context(A, m_alloc=20) as ctx:
            alone.append(ctx.expmv(v, t, 20, **kw)[0])
    wrong = []

    def work(i):
        A, t, kw, v = jobs[i]
        try:
            with Context(A, m_alloc=20) as ctx:
                for _ in range(10):
                    if not np.array_equal(ctx.expmv(v, t, 20, **kw)[0], alone[i]):
                        wrong.append((i, "differs"))
        except Exception as e:  # reported below
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong, wrong
