"""Half tilts that a caller marks open or not closed (astg_set "tilt_open" / "tilt_flags" take any marks)
are visited as open tilts and as half tilts, in that order: the buoyancy of both adds up, and the
advected half tilt stands.  Both stages against the oracle, whose loops run one after the other, bit
for bit, the same on every repetition."""
import numpy as np
import pytest

from fixtures import FIELDS

pytestmark = pytest.mark.gpu
DT = 0.01
TF_CLOSED, TF_HALF = 2, 32


@pytest.mark.parametrize("stage", [1, 5])
@pytest.mark.parametrize("size", [(8, 3), (16, 2)])
def test_half_tilts_marked_open(size, stage):
    import ast_solver
    from oracle.oracle import Oracle

    s, o = ast_solver.OctreeSmoke3(*size), Oracle(*size, reduce_mode=1, tilt_adaptivity=False)
    s.set_tilt_adaptivity(False)
    for _ in range(2):
        s.update(DT)
    for i in range(stage):
        s.stage(i, DT)
    state = {q + f: s.get(q + f) for f in FIELDS for q in ("", "t_")}
    marks = s.get("tilt_open")
    half = (state["tilt_flags"][:, 0] & TF_HALF) != 0
    assert half.sum() == len(s.get("half_tilts"))
    some = half & (np.cumsum(half) % 3 != 0)  # two of three
    marks[some] |= 1
    state["tilt_open"] = marks
    for q in ("", "t_"):
        state[q + "tilt_flags"][some, 0] &= ~TF_CLOSED
    for f, v in state.items():
        o.set(f, v)
    o.stage(stage, DT)
    for _ in range(3):
        for f, v in state.items():
            s.set(f, v)
        s.stage(stage, DT)
        for f in ("mac", "tilt_vel", "density_oct", "density_tilt", "heat_tilt"):
            np.testing.assert_array_equal(s.get(f), o.get(f), err_msg=f)
    s.close()
    o.close()
