"""Batch results where the device has no memory for their transposition: the
host transposes them, to the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 5, 16])
def test_results_without_a_device_buffer(nrhs):
    from mexk import synthetic as S
    from mexk._lib import check, lib
    from mexk.batch import Batch

    probs = [S.random_diag_dominant(n, 5, seed=n) for n in (65, 256, 257, 512, 513)]
    rng = np.random.default_rng(nrhs)
    with Batch(m=20, tol=1e-8) as b:
        for A in probs:
            b.add(A, rng.standard_normal((nrhs, A.n)), 0.5)
        b.upload()
        b.run()
        kept = [b.result(i) for i in range(len(probs))]
        check(lib().mexk_test_refuse_columns(b._h, 1))
        without = [b.result(i) for i in range(len(probs))]
        check(lib().mexk_test_refuse_columns(b._h, 0))
        after = [b.result(i) for i in range(len(probs))]
    for (Y, res), (Yw, resw), (Ya, _) in zip(kept, without, after):
        assert Y.any() and np.array_equal(Y, Yw) and np.array_equal(Y, Ya) and res == resw
