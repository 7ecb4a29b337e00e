"""The MIC(0) factorisation at the sizes where its rows per warp change (1, 2, 4, 32): the solution and
the iteration count equal the oracle's bit for bit (the same operations in the same order), so the
tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 129, 14000, 14001, 28000, 28001, 56000, 56001])
def test_factor_at_the_changes_of_rows_per_warp(n):
    import ast_solver
    from oracle.oracle import Oracle

    k = np.arange(n)
    off = [d for d in (1, 29, 811) if d < n]
    i = np.concatenate([k] + [k[:-d] for d in off] + [k[d:] for d in off])
    j = np.concatenate([k] + [k[d:] for d in off] + [k[:-d] for d in off])
    v = np.full(len(i), -1.0)
    v[:n] = np.bincount(i[n:], minlength=n) + 0.2
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    b = np.random.default_rng(n).standard_normal(n)
    s, h = ast_solver.OctreeSmoke3(40, 2), Oracle(8, 2, reduce_mode=1)
    x, st = s.solve(rp, j[o].astype(np.int32), v[o], b)
    xo, ito = h.solve(rp, j[o].astype(np.int32), v[o], b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    s.close()
    h.close()
