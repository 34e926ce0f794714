"""Window-2 stencil bases of several contexts at once, of few rows a block (so
that two grids could share SMs by their sizes): each keeps all of an SM's
tensor memory, and every thread gets the bits it gets alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_stencil_bases_side_by_side():
    from mexk import synthetic as S
    from mexk.api import Context

    A = S.laplacian_2d(97)
    t = 0.5 / A.max_abs()
    kw = dict(precision="mixed", controller="search", window=2)
    vs = [np.random.default_rng(i).uniform(0, 1, A.n) for i in range(6)]
    with Context(A, m_alloc=20) as ctx:
        alone = [ctx.expmv(v, t, 20, **kw)[0] for v in vs]
        assert ctx.basis_launches(20, "mixed", 2) == 1
    wrong = []

    def work(i):
        try:
            with Context(A, m_alloc=20) as ctx:
                for _ in range(40):
                    if not np.array_equal(ctx.expmv(vs[i], t, 20, **kw)[0], alone[i]):
                        wrong.append((i, "differs"))
        except Exception as e:  # reported below
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(vs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong, wrong
