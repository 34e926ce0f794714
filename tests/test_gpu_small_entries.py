"""FP64 solves hold every entry to FP64's rounding, not the vector's norm
alone: one large entry and a tail many orders below it (a point source on a
quiet background), away from the large one, against a Taylor sum.

The bound: a cycle's columns hold such an entry with the rounding of m + 3
products and two corrections of m terms each, relative to the entries around
it, so that 4 m 2^-53 a cycle (2e-14 at 50 columns) is generous; the Taylor
sum's own 30 terms add 30 2^-53 exp(|tA|) < 1e-14. 1e-12 is the bound that
FP64 results are held to in norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tridiagonal(n):
    from mexk import synthetic as S

    rng = np.random.default_rng(n)
    lower, diag, upper = rng.uniform(0.5, 1.0, n - 1), -2.0 + 0.1 * rng.uniform(size=n), rng.uniform(0.5, 1.0, n - 1)
    cols = np.arange(n)[:, None] + np.array([-1, 0, 1])
    vals = np.stack([np.r_[0.0, lower], diag, np.r_[upper, 0.0]], axis=1)
    keep = (cols >= 0) & (cols < n)
    rp = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(keep.sum(axis=1), out=rp[1:])
    return S.CSR(n, rp, cols[keep].astype(np.int32), vals[keep]), (lower, diag, upper)


def exponential(bands, v, t):
    lower, diag, upper = bands
    out, term = v.copy(), v.copy()
    for i in range(1, 30):
        w = diag * term
        w[1:] += lower * term[:-1]
        w[:-1] += upper * term[1:]
        term = w * (t / i)
        out += term
    return out


# one cluster; a grid of few and of many rows a block; the context's SpMV, w in memory
@pytest.mark.parametrize("n,m", [(4001, 30), (40007, 80), (150003, 30), (900001, 20), (3450001, 20)])
@pytest.mark.parametrize("level", [1e-6, 1e-12])
def test_entries_far_below_the_largest(n, m, level):
    from mexk.api import Context

    A, bands = tridiagonal(n)
    v = level * np.random.default_rng(4).uniform(0.5, 1.0, n)
    v[n // 3] = 1.0
    t = 0.2 / A.max_abs()
    ref = exponential(bands, v, t)
    with Context(A, m_alloc=m) as ctx:
        y, res = ctx.expmv(v, t, m)
    assert res["converged"] == 1
    err = np.abs((y - ref) / ref)
    err[n // 3 - 400:n // 3 + 400] = 0.0  # what the large entry spreads to in a few cycles
    assert err.max() <= 1e-12
