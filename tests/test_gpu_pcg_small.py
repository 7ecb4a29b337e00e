"""PCG iterations whose light work is one cluster's kernel, at the edges of its range (16384 rows) and
of its split (chunks of 2048 rows, 16 lanes of the fixed tree and 128 rows per CTA and chunk), one
column of rows more or less: FP64 solutions and iteration counts equal the oracle's bit for bit, so
the tolerance is zero; the mixed form meets the FP64 stopping test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 15, 17, 2047, 2064, 4096, 14337, 16383, 16384, 16385]


@pytest.mark.parametrize("n", SIZES)
def test_solutions_at_the_edges_of_the_small_form(n):
    import ast_solver
    from oracle.oracle import Oracle

    k = np.arange(n)
    off = [d for d in (1, 13, 170) if d < n]
    i = np.concatenate([k] + [k[:-d] for d in off] + [k[d:] for d in off])
    j = np.concatenate([k] + [k[d:] for d in off] + [k[:-d] for d in off])
    v = np.full(len(i), -1.0)
    v[:n] = np.bincount(i[n:], minlength=n) + 0.05
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    col, val = j[o].astype(np.int32), v[o]
    b = np.random.default_rng(n).standard_normal(n)
    s, h = ast_solver.OctreeSmoke3(24, 2), Oracle(8, 2, reduce_mode=1)
    x, st = s.solve(rp, col, val, b)
    xo, ito = h.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    r = b.copy()
    np.subtract.at(r, np.repeat(k, np.diff(rp)), val * xm[col])
    assert sm.converged == 1 and np.abs(r).max() <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
    s.close()
    h.close()
