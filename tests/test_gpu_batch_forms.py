"""Batches of more right-hand sides than solves fit side by side take another launch shape of the
preconditioner (and more lanes); every solution is the one astg_solve returns, bit for bit, so the
tolerance is zero.  One CTA per solve, a cluster, and a cluster whose single form has more warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs,precision", [(1000, 27, "fp64"), (6000, 21, "fp64"), (6000, 21, "mixed"), (31000, 12, "fp64")])
def test_batches_equal_single_solves(n, nrhs, precision):
    import ast_solver

    k = np.arange(n)
    off = (1, 19, 361)
    i = np.concatenate([k] + [k[:-d] for d in off] + [k[d:] for d in off])
    j = np.concatenate([k] + [k[d:] for d in off] + [k[:-d] for d in off])
    v = np.full(len(i), -1.0)
    v[:n] = np.bincount(i[n:], minlength=n) + 0.1
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    col, val = j[o].astype(np.int32), v[o]
    B = np.random.default_rng(n).standard_normal((nrhs, n))
    s = ast_solver.OctreeSmoke3(32, 2)
    X = s.solve_batch(rp, col, val, B, precision=precision)[0]
    for q in range(nrhs):
        np.testing.assert_array_equal(X[q], s.solve(rp, col, val, B[q], precision=precision)[0])
    s.close()
