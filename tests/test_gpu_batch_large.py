"""Batches of systems above 100,000 rows: the mixed form takes the launch shape that shares SMs (two row
blocks per CTA) where that saves rounds, FP64 keeps the single solve's; every solution is the one astg_solve returns, bit for
bit, so the tolerance is zero."""
import numpy as np
import pytest

from fixtures import csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs,precision", [(100000, 9, "mixed"), (100001, 9, "mixed"), (100001, 9, "fp64"), (250000, 10, "mixed"), (250000, 18, "mixed"), (500000, 9, "mixed")])
def test_batches_equal_single_solves(n, nrhs, precision):
    import ast_solver

    k = np.arange(n)
    rp, col, val = csr(n, np.concatenate([np.stack([k[:-d], k[d:]], 1) for d in (3, 61, 3600)]), 0.3)
    B = np.random.default_rng(n).standard_normal((nrhs, n))
    s = ast_solver.OctreeSmoke3(64, 3)
    X, stats = s.solve_batch(rp, col, val, B, precision=precision)[:2]
    for q in range(nrhs):
        np.testing.assert_array_equal(X[q], s.solve(rp, col, val, B[q], precision=precision)[0])
    s.close()
