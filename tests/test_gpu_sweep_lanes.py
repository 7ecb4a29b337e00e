"""Items of the barrier-free sweeps whose spare lanes repeat a row, where no wait for an entry stands
between a lane's read of the row's value and another's write of it: rows without entries (all of a
diagonal system, and the last rows of a forest of pairs in the backward sweep), in items of 1 to 32
rows.  FP64 solutions equal the oracle's bit for bit, the same every time; the mixed form solves a
diagonal system to its FP64 stopping test."""
import numpy as np
import pytest

from fixtures import csr, residual

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 65, 2047, 4097, 16 * 32 * 9 + 16])
def test_rows_without_entries_in_part_filled_items(n, pairs):
    import ast_solver
    from oracle.oracle import Oracle

    k = np.arange(n)
    couples = np.stack([k[0 : n // 2 * 2 : 2], k[1 : n // 2 * 2 : 2]], 1) if pairs else []
    rp, col, val = csr(n, couples, 1.0 + k / n)
    b = np.random.default_rng(n).standard_normal(n)
    s, o = ast_solver.OctreeSmoke3(24, 2), Oracle(8, 2, reduce_mode=1)
    xo, ito = o.solve(rp, col, val, b)
    for _ in range(4):
        x, st = s.solve(rp, col, val, b)
        assert st.converged == 1 and st.iterations == ito
        np.testing.assert_array_equal(x, xo)
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    assert sm.converged == 1 and residual(rp, col, val, xm, b) <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
    s.close()
    o.close()
