"""The barrier-free MIC(0) sweeps (k_precond_async) on systems at the edges of their schedule: items
of 32 rows (one row more or less), quads of four entries (rows of 0 to 29 lower entries), one CTA or
a cluster, one or three row blocks per CTA, and a chain with more items than their arrays hold (the
level-synchronous form takes over).  FP64 solutions and iteration counts equal the oracle's bit for
bit (the same operations in the same order); the mixed form meets the FP64 stopping test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def csr(n, pairs, diag):
    """Symmetric CSR with off-diagonals -1 at `pairs` and a dominant diagonal."""
    i = np.concatenate([pairs[:, 0], pairs[:, 1], np.arange(n)])
    j = np.concatenate([pairs[:, 1], pairs[:, 0], np.arange(n)])
    v = np.concatenate([-np.ones(2 * len(pairs)), np.full(n, -1.0)])
    deg = np.bincount(i[: 2 * len(pairs)], minlength=n)
    v[2 * len(pairs):] = deg + diag
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))])
    return rp.astype(np.int32), j[o].astype(np.int32), v[o]


def band(n, reach):
    k = np.arange(n)
    return np.concatenate([np.stack([k[:-d], k[d:]], 1) for d in range(1, reach + 1) if d < n] or [np.zeros((0, 2), int)])


def box(nx, ny, nz):
    k = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    return np.concatenate([np.stack([a.ravel(), b.ravel()], 1) for a, b in
                           ((k[:, :, :-1], k[:, :, 1:]), (k[:, :-1], k[:, 1:]), (k[:-1], k[1:]))])


CASES = {
    "one row": (1, band(1, 1)),
    "independent rows": (33, np.zeros((0, 2), int)),
    "31 rows": (31, band(31, 3)),
    "dense 30": (30, band(30, 29)),
    "ragged band": (4095, np.unique(np.concatenate([band(4095, 2), np.stack([np.arange(0, 4000, 7), np.arange(0, 4000, 7) + 61], 1)]), axis=0)),
    "one CTA's last size": (4096, box(16, 16, 16)),
    "first cluster size": (4097, np.concatenate([box(16, 16, 16), [[0, 4096], [4000, 4096]]])),
    "rows of 13 entries": (6000, np.unique(np.concatenate([band(6000, 6), np.stack([np.arange(5900), np.arange(5900) + 97], 1)]), axis=0)),
    "last size of one block per CTA": (46 * 46 * 47, box(46, 46, 47)),
    "first size of three blocks per CTA": (46 * 47 * 47, box(46, 47, 47)),
    "more items than the arrays hold": (40000, band(40000, 1)),
}


@pytest.fixture(scope="module")
def handles():
    import ast_solver
    from oracle.oracle import Oracle

    s, o = ast_solver.OctreeSmoke3(48, 2), Oracle(8, 2, reduce_mode=1)
    yield s, o
    s.close()
    o.close()


@pytest.mark.parametrize("name", CASES)
def test_sweeps_on_edge_systems(name, handles):
    s, o = handles
    n, pairs = CASES[name]
    rp, col, val = csr(n, np.asarray(pairs, dtype=np.int64).reshape(-1, 2), 0.05)
    b = np.random.default_rng(n).standard_normal(n)
    x, st = s.solve(rp, col, val, b)
    xo, ito = o.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    r = b.copy()
    np.subtract.at(r, np.repeat(np.arange(n), np.diff(rp)), val * xm[col])
    assert sm.converged == 1 and np.abs(r).max() <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
