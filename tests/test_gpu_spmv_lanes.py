"""The PCG's product kernel where the lanes of its reducing warp have different numbers of rows (the last
chunk of 2048 rows ends inside a warp's 32 lanes): FP64 solutions and iteration counts equal the
oracle's bit for bit, so the tolerance is zero.  More rows than the one-cluster form of an iteration
takes, so that this kernel runs."""
import numpy as np
import pytest

from fixtures import csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", [1, 31, 33, 255, 257, 511 + 16, 1793, 2047])
def test_last_chunk_ends_inside_a_warp(last):
    import ast_solver
    from oracle.oracle import Oracle

    n = 8 * 2048 + last
    k = np.arange(n)
    rp, col, val = csr(n, np.concatenate([np.stack([k[:-d], k[d:]], 1) for d in (1, 26, 676)]), 0.1)
    b = np.random.default_rng(last).standard_normal(n)
    s, o = ast_solver.OctreeSmoke3(24, 2), Oracle(8, 2, reduce_mode=1)
    x, st = s.solve(rp, col, val, b)
    xo, ito = o.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    s.close()
    o.close()
