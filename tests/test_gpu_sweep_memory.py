"""What the barrier-free sweeps' records take.  They are held per row, so a handle's memory follows its
row capacity, and a matrix of narrow levels (a chain: one row a level) runs in the form it was asked
for like any other."""
import numpy as np
import pytest

from fixtures import csr, residual

pytestmark = pytest.mark.gpu


def used(make):
    import torch

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = make()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0], s


def test_handles_take_memory_by_their_rows():
    """4 KB a row (matrix rows of 32 entries at 68 bytes in their several forms, the records, vectors and
    fields: about 3.4 KB) and 24 MB whatever the size."""
    import ast_solver

    def grid():
        s = ast_solver.ASTSolver2(resolution=[192, 384], dx=1.0 / 192, name="memory")
        s.initialize()
        return s

    ast_solver.OctreeSmoke3(8, 2).close()  # the context and the library's own first use
    for make, rows in ((lambda: ast_solver.OctreeSmoke3(8, 3), None), (lambda: ast_solver.OctreeSmoke3(22, 2), None),
                       (grid, 192 * 384 + 193 * 385)):
        b, s = used(make)
        if rows is None:
            rows = 2 * int(s.get("level_sizes")[:, 0].sum()) + len(s.get("half_tilts"))
        s.close()
        assert b <= 4096 * rows + 24e6, f"{b / 1e6:.1f} MB for {rows} rows"


@pytest.mark.parametrize("n", [4097, 33000, 40000])
def test_a_chain_keeps_the_precision_asked_for(n):
    import ast_solver
    from oracle.oracle import Oracle

    k = np.arange(n)
    rp, col, val = csr(n, np.stack([k[:-1], k[1:]], 1), 0.05)
    b = np.random.default_rng(n).standard_normal(n)
    s, o = ast_solver.OctreeSmoke3(48, 2), Oracle(8, 2, reduce_mode=1)
    x, st = s.solve(rp, col, val, b)
    xo, ito = o.solve(rp, col, val, b)
    assert st.converged == 1 and st.iterations == ito and st.outer == 0
    np.testing.assert_array_equal(x, xo)
    xm, sm = s.solve(rp, col, val, b, precision="mixed")
    assert sm.converged == 1 and sm.outer > 0 and residual(rp, col, val, xm, b) <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
    s.close()
    o.close()


def ladder(levels, width=32, reach=31):
    """Levels of `width` rows: rows 1.. each on its namesake of the level before, row 0 on `reach` of
    them.  Every item of 32 rows (forward) then holds one row of 31 entries and 31 of one."""
    at = np.arange(1, levels)[:, None] * width
    k = np.arange(1, width)[None, :]
    same = np.stack([(at - width + k).ravel(), (at + k).ravel()], 1)
    far = np.stack([(at - width + k[:, :reach]).ravel(), np.broadcast_to(at, (levels - 1, reach)).ravel()], 1)
    return np.unique(np.concatenate([same, far]), axis=0)


@pytest.mark.parametrize("share", [0.1, 0.5, 0.95])
def test_items_of_rows_of_very_different_lengths(share):
    """Seven quads after the first for each row of the forward sweep, where a handle starts with room for
    four per row of its capacity: the largest share takes more (and the next solve finds it)."""
    import ast_solver
    from oracle.oracle import Oracle

    s, o = ast_solver.OctreeSmoke3(16, 2), Oracle(8, 2, reduce_mode=1)
    capacity = 2 * int(s.get("level_sizes")[:, 0].sum()) + len(s.get("half_tilts"))
    levels = int(share * capacity) // 32
    n = 32 * levels
    rp, col, val = csr(n, ladder(levels), 0.05)
    assert np.diff(rp).max() == 32
    b = np.random.default_rng(n).standard_normal(n)
    xo, ito = o.solve(rp, col, val, b)
    for _ in range(2):
        xm, sm = s.solve(rp, col, val, b, precision="mixed")
        assert sm.converged == 1 and sm.outer > 0
        assert residual(rp, col, val, xm, b) <= 1e-6 * np.abs(b).max() * (1 + 1e-6)
        x, st = s.solve(rp, col, val, b)
        assert st.converged == 1 and st.iterations == ito
        np.testing.assert_array_equal(x, xo)
    X = s.solve_batch(rp, col, val, np.stack([b, 2 * b, b]))[0]
    np.testing.assert_array_equal(X[0], xo)
    np.testing.assert_array_equal(X[2], xo)
    s.update(0.01)  # the handle's own systems after the caller's
    p = ast_solver.OctreeSmoke3(16, 2)
    p.update(0.01)
    np.testing.assert_array_equal(s.get("p"), p.get("p"))
    for h in (s, p, o):
        h.close()
