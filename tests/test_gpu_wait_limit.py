"""The bounded waits of the one-launch bases give up by their own limit: block
0 leaves before the first meeting and tells nobody, every other block's wait
runs out, the solve reports it, and the same context then solves as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,kw", [("random", 20000, {}), ("random", 300007, {}), ("heat", 150, {}),
                                       ("heat", 301, dict(window=2)), ("random", 20000, dict(precision="mixed")),
                                       ("heat", 301, dict(precision="mixed", controller="search", window=2))])
def test_every_block_gives_up(kind, n, kw):
    from mexk import synthetic as S
    from mexk._lib import MexkError, check, lib
    from mexk.api import Context

    A = S.laplacian_2d(n) if kind == "heat" else S.random_diag_dominant(n, 8, seed=n)
    v = np.random.default_rng(n).standard_normal(A.n)
    t = 0.5 / A.max_abs()
    with Context(A, m_alloc=20) as ctx:
        good, _ = ctx.expmv(v, t, 20, **kw)
        check(lib().mexk_test_force_wait_timeout(0, 1))
        try:
            with pytest.raises(MexkError, match="device wait gave up"):
                ctx.expmv(v, t, 20, **kw)
        finally:
            check(lib().mexk_test_force_wait_timeout(0, 0))
        again, _ = ctx.expmv(v, t, 20, **kw)
    assert np.array_equal(good, again)
