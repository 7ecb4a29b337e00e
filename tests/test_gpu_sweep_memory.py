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
