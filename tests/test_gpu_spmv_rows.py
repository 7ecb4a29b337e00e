"""The PCG's matrix product, dot products and folds at the edges of their split (256-row CTAs in
clusters of eight, 2048-row chunks, entry quads, eight entries before the remainder): FP64 solutions
and iteration counts equal the oracle's bit for bit, so the tolerance is zero; the mixed form meets
the FP64 stopping test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 32, 255, 256, 257, 2047, 2048, 2049, 4100, 18433]


def system(n, rng):
    """Symmetric, diagonally dominant; rows of 1 to 31 entries, some warps with short rows alone."""
    room = np.full(n, 1)
    long_rows = rng.random(n) < 0.05
    room[long_rows] = rng.integers(5, 31, long_rows.sum())
    room[: n // 2 : 3] += 4
    cols = [set() for _ in range(n)]
    for i in range(n):
        for j in rng.integers(max(0, i - 300), min(n, i + 300), 2 * room[i]):
            if j != i and len(cols[i]) < min(room[i], 31) and len(cols[j]) < 31:
                cols[i].add(int(j))
                cols[int(j)].add(i)
    rp, col, val = [0], [], []
    for i in range(n):
        for j in sorted(cols[i] | {i}):
            col.append(j)
            val.append(len(cols[i]) + 0.1 if j == i else -1.0)
        rp.append(len(col))
    return np.array(rp, np.int32), np.array(col, np.int32), np.array(val)


@pytest.mark.parametrize("n", SIZES)
def test_solutions_at_the_edges_of_the_row_split(n):
    import ast_solver
    from oracle.oracle import Oracle

    rng = np.random.default_rng(n)
    rp, col, val = system(n, rng)
    assert np.diff(rp).max() <= 32
    b = rng.standard_normal(n)
    s, o = ast_solver.OctreeSmoke3(24, 2), Oracle(8, 2, reduce_mode=1)
    x, st = s.solve(rp, col, val, b)
    xo, ito = o.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito
    np.testing.assert_array_equal(x, xo)
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    r = b.copy()
    np.subtract.at(r, np.repeat(np.arange(n), np.diff(rp)), val * xm[col])
    assert sm.converged == 1 and np.abs(r).max() <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
    s.close()
    o.close()
