"""Every form of the sweeps (ASTG_SWEEP) solves the same systems to the same bits, the one without
clusters (its matrix product too) among them: in the library's order against the oracle's, at sizes of
one chunk of 2048 rows, a ragged last chunk, and more chunks than one cluster kernel takes."""
import numpy as np
import pytest

from fixtures import csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["async", "dsmem", "cluster", "syncfree"])
def test_forms_agree_with_the_oracle(mode, monkeypatch):
    import ast_solver
    from oracle.oracle import Oracle

    monkeypatch.setenv("ASTG_SWEEP", mode)
    s, o = ast_solver.OctreeSmoke3(24, 2), Oracle(8, 2, reduce_mode=1)
    for n in (1, 33, 2048, 2049, 5000, 8 * 2048 + 777):
        k = np.arange(n)
        off = [np.stack([k[:-d], k[d:]], 1) for d in (1, 17, 300) if d < n] or [np.zeros((0, 2), int)]
        rp, col, val = csr(n, np.concatenate(off), 0.1)
        b = np.random.default_rng(n).standard_normal(n)
        x, st = s.solve(rp, col, val, b)
        xo, ito = o.solve(rp, col, val, b)
        assert st.converged == 1 and st.iterations == ito
        np.testing.assert_array_equal(x, xo)
    s.close()
    o.close()


@pytest.mark.parametrize("mode", ["async", "syncfree"])
def test_reference_order_is_the_same_in_both_products(mode, monkeypatch):
    import ast_solver

    n = 4100
    k = np.arange(n)
    rp, col, val = csr(n, np.concatenate([np.stack([k[:-d], k[d:]], 1) for d in (1, 17, 300)]), 0.1)
    b = np.random.default_rng(n).standard_normal(n)
    out = []
    for m in ("dsmem", mode):
        monkeypatch.setenv("ASTG_SWEEP", m)
        s = ast_solver.OctreeSmoke3(16, 2)
        s.set_reduction_order("reference")
        out.append(s.solve(rp, col, val, b)[0])
        s.close()
    np.testing.assert_array_equal(out[0], out[1])
