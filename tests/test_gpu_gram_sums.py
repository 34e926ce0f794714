"""The FP32 sums of a one-launch basis over a block's rows: many small terms
after a large one still count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def test_small_terms_after_a_large_one():
    """A cyclic shift keeps the start vector's values, one row on: all columns
    are orthogonal and their stored norms are one sum each. In each block the
    first 128 rows have ones and the others values whose squares, 4e-8, are
    below half a unit in the last place of 1: 51 of them added one by one to a
    lane's 1 would leave no trace (2e-6 of the sum). The bound: 16 roundings
    of U (a float4's four products, four of them, the total, the warp's five
    and the column's normalisation)."""
    from mexk import synthetic as S
    from mexk.api import Context

    n, m = 1_000_000, 40
    rows = (-(-n // 152) + 31) // 32 * 32  # of a block
    r = np.arange(n)
    v = np.where(r % rows < 128, 1.0, 2e-4) * (r % 64 == 0)
    A = S.CSR(n, np.arange(n + 1, dtype=np.int32), ((r - 1) % n).astype(np.int32), np.ones(n))
    with Context(A, m_alloc=m) as ctx:
        _, res = ctx.expmv(v, 0.01, m, precision="mixed", controller="search")
        assert res["cycles"] == 1 and ctx.basis_launches(m, "mixed") == 1
        V = ctx.get_basis(m, "mixed")
    assert np.abs((V * V).sum(axis=1) - 1.0).max() <= 16 * U
