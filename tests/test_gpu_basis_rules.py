"""The sizes at which a solve's bases go from one launch to separate kernels:
either side of each rule gives the result to its form's bound, and above it
the bits of the separate kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(N, m, precision, window, one):
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.laplacian_2d(N)
    v = np.random.default_rng(N).standard_normal(A.n)
    t = 1e-3 / A.max_abs()
    kw = dict(precision=precision, window=window, controller="search" if precision == "mixed" else "reference")
    with Context(A, m_alloc=m) as ctx:
        y, res = ctx.expmv(v, t, m, **kw)
        assert (ctx.basis_launches(m, precision, window) == 1) == one
        ctx.set_basis_form("separate")
        apart, res2 = ctx.expmv(v, t, m, **kw)
    if m > 3:  # three columns do not reach the controller's tolerance
        assert res["converged"] == res2["converged"] == 1
    if one and m > 3:
        bound = 1e-12 if precision == "fp64" else 2e-6
        assert np.linalg.norm(y - apart) <= bound * np.linalg.norm(apart)
    elif not one:
        assert np.array_equal(y, apart)


@pytest.mark.parametrize("N,window,one", [(1850, 6, True), (1851, 4, True), (1851, 5, False), (1851, 8, False),
                                          (1851, 9, True), (1851, 0, True)])
def test_fp64_windows_where_w_leaves_the_chip(N, window, one):
    check(N, 10, "fp64", window, one)


@pytest.mark.parametrize("N,m,one", [(547, 3, True), (548, 3, False), (548, 4, True), (1341, 5, True), (1342, 5, False)])
def test_mixed_bases_of_few_columns(N, m, one):
    check(N, m, "mixed", 0, one)
