"""The barrier-free sweeps at the size where one CTA gives way to a cluster (2,100 rows), one row more or
less, alone and in batches: FP64 solutions and iteration counts equal the oracle's bit for bit, so the
tolerance is zero; the mixed form meets the FP64 stopping test."""
import numpy as np
import pytest

from fixtures import csr, residual

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2099, 2100, 2101])
def test_one_cta_or_a_cluster(n):
    import ast_solver
    from oracle.oracle import Oracle

    k = np.arange(n)
    rp, col, val = csr(n, np.concatenate([np.stack([k[:-d], k[d:]], 1) for d in (1, 13, 170)]), 0.05)
    b = np.random.default_rng(n).standard_normal(n)
    s, o = ast_solver.OctreeSmoke3(16, 2), Oracle(8, 2, reduce_mode=1)
    xo, ito = o.solve(rp, col, val, b)
    x, st = s.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    np.testing.assert_array_equal(s.solve_batch(rp, col, val, np.stack([b] * 26))[0], np.stack([xo] * 26))
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    assert sm.converged == 1 and residual(rp, col, val, xm, b) <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
    s.close()
    o.close()
