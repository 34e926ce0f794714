"""A context's first solves while the legacy default stream has work queued:
the buffers that they allocate are cleared on the context's own stream, so
that the bits are those of a context that had the GPU to itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,m,kw", [("random", 150003, 23, {}), ("random", 300007, 20, dict(precision="mixed")),
                                         ("heat", 301, 20, dict(precision="mixed", controller="search", window=2))])
def test_first_solve_does_not_wait_for_nor_race_with_it(kind, n, m, kw):
    import torch

    from mexk import synthetic as S
    from mexk.api import Context

    A = S.laplacian_2d(n) if kind == "heat" else S.random_diag_dominant(n, 8, seed=n)
    v = np.random.default_rng(n).standard_normal(A.n)
    t = 0.5 / A.max_abs()
    with Context(A, m_alloc=m) as ctx:
        alone, _ = ctx.expmv(v, t, m, **kw)
    with Context(A, m_alloc=m) as ctx:
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
        first, _ = ctx.expmv(v, t, m, **kw)
        torch.cuda.synchronize()
        second, _ = ctx.expmv(v, t, m, **kw)
    assert np.array_equal(first, alone) and np.array_equal(second, alone)
