"""One-launch bases that the device refuses: the solve takes the separate
kernels and returns their bits, and the context goes back to one launch when
it can. The refusal is made on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("kind,n,kw", [("random", 3000, {}), ("random", 20000, {}), ("random", 300007, {}),
                                       ("heat", 150, dict(window=2)), ("random", 3000, dict(precision="mixed")),
                                       ("random", 20000, dict(precision="mixed", controller="search")),
                                       ("heat", 150, dict(precision="mixed", controller="search", window=2))])
def test_refused_launch_takes_the_separate_kernels(monkeypatch, kind, n, kw, graphs):
    from mexk import synthetic as S
    from mexk._lib import check, lib
    from mexk.api import Context

    if not graphs:
        monkeypatch.setenv("MEXK_NO_GRAPH", "1")
    A = S.laplacian_2d(n) if kind == "heat" else S.random_diag_dominant(n, 8, seed=n)
    v = np.random.default_rng(n).standard_normal(A.n)
    t = 0.5 / A.max_abs()
    prec, window = kw.get("precision", "fp64"), kw.get("window", 0)
    with Context(A, m_alloc=20) as ctx:
        one, r1 = ctx.expmv(v, t, 20, **kw)
        k1 = ctx.basis_launches(20, prec, window)
        ctx.set_basis_form("separate")
        apart, r2 = ctx.expmv(v, t, 20, **kw)
        assert ctx.basis_launches(20, prec, window) > k1
        ctx.set_basis_form("one_launch")
        check(lib().mexk_test_refuse_one_launch(ctx.handle, 1))
        refused, r3 = ctx.expmv(v, t, 20, **kw)
        again, _ = ctx.expmv(v, t, 20, **kw)
        check(lib().mexk_test_refuse_one_launch(ctx.handle, 0))
        last, _ = ctx.expmv(v, t, 20, **kw)
        assert ctx.basis_launches(20, prec, window) == k1
    assert r1["converged"] == r2["converged"] == r3["converged"] == 1
    assert np.array_equal(refused, apart) and np.array_equal(again, apart) and np.array_equal(last, one)
    bound = 1e-12 if prec == "fp64" else 2e-6  # each within the form's bound of the exact result
    assert np.linalg.norm(one - apart) <= bound * np.linalg.norm(one)
