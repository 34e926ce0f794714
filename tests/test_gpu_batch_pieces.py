"""Batch results transposed on the device, and the streaming sweeps' pieces,
at sizes around their 64-row and 512-row edges and for fewer than 16
right-hand sides: against the row-major results and dense exponentials."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs", [(33, 1), (63, 3), (64, 16), (65, 16), (511, 2), (512, 16), (513, 5), (1025, 16)])
def test_columns_and_rows_agree_with_dense(n, nrhs):
    from scipy.linalg import expm

    from mexk import synthetic as S
    from mexk._lib import Result, check, lib
    from mexk.batch import Batch

    probs = [S.random_diag_dominant(n, 5, seed=n), S.random_diag_dominant(700, 4, seed=7)]
    rng = np.random.default_rng(n)
    Vs = [rng.standard_normal((nrhs, A.n)) for A in probs]
    with Batch(m=20, tol=1e-8) as b:
        for A, V in zip(probs, Vs):
            b.add(A, V, 0.5)
        b.upload()
        b.run()
        for i, (A, V) in enumerate(zip(probs, Vs)):
            Y, res = b.result(i)
            assert Y.shape == (nrhs, A.n) and Y.flags["C_CONTIGUOUS"]
            rows = np.empty((A.n, nrhs))
            r = (Result * nrhs)()
            check(lib().mexk_batch_result(b._h, i, rows.ctypes.data_as(C.POINTER(C.c_double)), r))
            assert np.array_equal(Y, rows.T)
            assert all(x["converged"] == 1 for x in res)
            ref = (expm(0.5 * A.to_dense()) @ V.T).T
            err = np.linalg.norm(Y - ref, axis=1) / np.linalg.norm(ref, axis=1)
            assert err.max() <= 1e-6  # the batch's bound
