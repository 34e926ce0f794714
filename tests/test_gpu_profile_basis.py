"""The basis's profile starts from clean meeting words and says so when there
is no basis to time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,precision,window", [("random", 3000, "fp64", 0), ("random", 20000, "fp64", 0),
                                                     ("random", 20000, "mixed", 0), ("heat", 301, "mixed", 2)])
def test_profile_basis(kind, n, precision, window):
    from mexk import synthetic as S
    from mexk._lib import MexkError, check, lib
    from mexk.api import Context

    A = S.laplacian_2d(n) if kind == "heat" else S.random_diag_dominant(n, 8, seed=n)
    v = np.random.default_rng(n).standard_normal(A.n)
    t = 0.5 / A.max_abs()
    kw = dict(precision=precision, window=window, controller="search" if precision == "mixed" else "reference")
    with Context(A, m_alloc=20) as ctx:
        with pytest.raises(MexkError, match="broke down"):  # no start vector yet
            ctx.profile_kernel("basis", 19, 3, precision)
        y, _ = ctx.expmv(v, t, 20, **kw)
        ms = ctx.profile_kernel("basis", 19, 3, precision)
        if A.n > 4096:
            check(lib().mexk_test_force_wait_timeout(0, 1))
            try:
                with pytest.raises(MexkError, match="device wait gave up"):
                    ctx.expmv(v, t, 20, **kw)
            finally:
                check(lib().mexk_test_force_wait_timeout(0, 0))
            ctx.set_basis((v / np.linalg.norm(v))[None], precision)
            again = ctx.profile_kernel("basis", 19, 3, precision)
            assert 0.2 * ms < again < 5.0 * ms  # launches that return at once take a few microseconds
        assert np.array_equal(ctx.expmv(v, t, 20, **kw)[0], y)
