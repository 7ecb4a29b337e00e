"""The wavefront sweeps of the uniform 2-D solver (one warp per 32 columns, boundary results handed
from warp to warp) at the edges of their split: one column pair, a warp less / exactly / more than
full, several warps with a ragged last one, the widest grid the sweeps take, and one just wider and
one just taller, which take the generic sweeps.  Whole frames against the 2-D oracle, whose
arithmetic is the same in the same order: the tolerance is zero."""
import numpy as np
import pytest

import ast_solver
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [(2, 5), (7, 2), (31, 40), (32, 33), (33, 17), (64, 31), (65, 70), (96, 2), (157, 40), (512, 24), (513, 12), (2, 25400)]


@pytest.mark.parametrize("nx,ny", SIZES)
def test_frames_at_the_edges_of_the_column_split(nx, ny):
    g = ast_solver.ASTSolver2(resolution=[nx, ny], dx=1.0 / nx, adaptive_dofs=True, name="test")
    g.initialize()
    o = orc.Oracle2D(nx, ny, adaptive=True, reduce_mode=1)
    rng = np.random.default_rng(1000 * nx + ny)
    for f in ("mac_x", "mac_y"):  # a divergent start, so that the projection has work at every size
        v = 0.01 * rng.standard_normal(g.get(f).size)
        if ny > 1000:  # the tallest: only across the channel's first rows (along it the CG needs thousands)
            v[30 if f == "mac_x" else 0 :] = 0
        g.set(f, v)
        o.set(f, v)
    for frame in range(2 if ny < 1000 else 1):
        for st in ("source", "project", "advect")[ny > 1000 :]:
            g.stage(st, 0.02)
            o.stage(st, 0.02)
        assert g.last_stats()["pcg_iterations"] == o.info()["pcg_iters"]
        for f in ("p", "mac_x", "mac_y", "tilt_open", "density_cell"):
            np.testing.assert_array_equal(g.get(f), o.get(f), err_msg=f"frame {frame + 1} {f}")
