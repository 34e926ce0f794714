"""The Pade exponential over a thread-block cluster at the sizes where its
column shares, warp rows and back substitution change: one row per lane to
four, columns that do not divide by the blocks, k up to the largest, and
Hessenberg matrices (whose denominator polynomial is zero below a band, so
that the elimination meets zero numerators)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [3, 15, 16, 17, 31, 32, 33, 63, 65, 96, 97, 127, 128])
@pytest.mark.parametrize("scale", [1e-2, 0.2, 0.9, 2.0, 8.0, 60.0])
def test_hessenberg_expm_vs_oracle(oracle_mod, k, scale):
    import torch

    from mexk._lib import check, lib

    rng = np.random.default_rng(k)
    M = np.triu(rng.standard_normal((k, k)), -1)
    M *= scale / np.abs(M).sum(axis=0).max()  # |M|_1 = scale: every degree, scaling and squarings
    E_ref = oracle_mod.expm(M)
    Md = torch.from_numpy(np.asfortranarray(M).ravel(order="F")).cuda()
    Ed = torch.zeros(k * k, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    check(lib().mexk_expm_f64(k, Md.data_ptr(), k, Ed.data_ptr(), k, None))
    E = Ed.cpu().numpy().reshape(k, k, order="F")
    # two evaluations of the same method: each within k u per product and solve, squared |M|_1 / 5.4 times
    tol = 1e-13 * max(10.0, scale)
    assert np.abs(E - E_ref).max() <= tol * max(1.0, np.abs(E_ref).max())
