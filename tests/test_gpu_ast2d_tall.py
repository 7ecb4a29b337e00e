"""The wavefront sweeps of the uniform 2-D solver on tall grids: the last height whose boundary results
fit a CTA's shared memory and the first whose do not (they go through global memory), at two warps of
columns, more warps, and grids of one warp, which hand nothing on, far above it.  A projection with open
tilts, against the generic sweeps, whose arithmetic is the same in the same order: the tolerance is
zero.  (Against the oracle these sizes take minutes; the generic sweeps are tested against it.)"""
import numpy as np
import pytest

import ast_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(33, 18592), (33, 18593), (64, 18600), (70, 19001), (100, 20000), (2, 60000), (32, 18593)])
def test_tall_grids_equal_the_generic_sweeps(nx, ny, monkeypatch):
    rng = np.random.default_rng(nx + ny)
    flow = {"mac_x": 0.01 * rng.standard_normal((nx + 1) * ny), "mac_y": 0.01 * rng.standard_normal(nx * (ny + 1))}
    tilts = np.zeros((ny + 1, nx + 1), np.uint8)
    tilts[1:-1, 1:-1] = rng.random((ny - 1, nx - 1)) < 0.05
    out = []
    for wave in ("1", "0"):
        monkeypatch.setenv("ASTG_WAVE", wave)
        g = ast_solver.ASTSolver2(resolution=[nx, ny], dx=1.0 / nx, adaptive_dofs=True, name="test")
        g.initialize()
        g.set_solver_parameters(max_iter=5)  # the sweeps of a few iterations
        for f, v in flow.items():
            g.set(f, v)
        g.set("tilt_open", tilts)
        g.stage("project", 0.02)
        st = g.last_stats()
        out.append((g.get("p"), st["pcg_residual"], st["unknowns"]))
        g.close()
    assert out[0][2] == nx * ny + tilts.sum() and np.abs(out[0][0]).max() > 0
    assert out[0][1:] == out[1][1:]
    np.testing.assert_array_equal(out[0][0], out[1][0])
