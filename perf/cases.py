"""The work a user of this library has it do, as cases that can be timed and whose outputs can be
compared: octree smoke steps (FP64 and mixed, adaptive and frozen topology, obstacle and CFL
sub-steps), pressure solves of systems the caller holds (one right-hand side, many, the caller's own
matrix), the advection stage, a differentiated window of steps, extrapolation, and the uniform 2-D
solver.  Every case goes through ast_solver's public entry points.

Ranges: octrees of 8 to 64 coarsest cells per axis and 2 to 4 levels (finest at most 256 per axis),
caller's matrices of 1,000 to 9,000 rows, 1 to 20 right-hand sides, windows of 2 to 8 steps, 2-D
grids of 24 x 32 to 192 x 384 cells.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ast-grid_gb300"))
import ast_solver  # noqa: E402

DT = 0.01
DT_2D = 0.02500000037252903  # 0.025f, the time step of the 2-D smoke scene
SCALARS = ["density_oct", "density_tilt", "heat_oct", "heat_tilt"]
VELOCITY = ["mac", "tilt_vel"]
DUAL = ["dual_oct", "dual_tilt"]
FIELDS_2D = ["density_cell", "heat_cell", "density_vert", "heat_vert", "mac_x", "mac_y", "tilt_vel", "tilt_open"]


def listed():
    return [
        # the simulation the library exists for: the 256^3-equivalent plume, topology adapting, one
        # frame after the other with the fields read back on the device
        {"name": "step_256_fp64", "kind": "step", "coarsest": 64, "levels": 3, "precision": "fp64", "frozen": False,
         "collider": False, "cfl": False},
        # the same simulation by a user who asked for the faster mixed-precision projection
        {"name": "step_256_mixed", "kind": "step", "coarsest": 64, "levels": 3, "precision": "mixed", "frozen": False,
         "collider": False, "cfl": False},
        # the smallest grid anyone runs (interactive, unit tests): launches and latencies
        {"name": "step_32_fp64", "kind": "step", "coarsest": 8, "levels": 3, "precision": "fp64", "frozen": True,
         "collider": False, "cfl": False},
        # an ordinary run on a size that is no power of two: the stock sphere obstacle and CFL sub-steps
        {"name": "step_obstacle_44", "kind": "step", "coarsest": 22, "levels": 2, "precision": "fp64", "frozen": True,
         "collider": True, "cfl": True},
        # a pressure system the caller holds on the host, solved once (PCGSolver::solve)
        {"name": "solve_256", "kind": "solve", "coarsest": 64, "levels": 3, "precision": "fp64", "nrhs": 1},
        # many right-hand sides of one matrix, side by side
        {"name": "solve_batch_128", "kind": "solve", "coarsest": 32, "levels": 3, "precision": "fp64", "nrhs": 20},
        # the caller's own matrix: a Poisson problem on an odd box with solid cells left out
        {"name": "solve_box_6k", "kind": "box", "nx": 23, "ny": 17, "nz": 19, "precision": "fp64"},
        # the advection stage by itself on the largest grid (solver loops that call the stages)
        {"name": "advect_256", "kind": "advect", "coarsest": 64, "levels": 3},
        # a differentiated window in an optimisation loop: forward and backward through autograd
        {"name": "window_64", "kind": "window", "coarsest": 32, "levels": 2, "steps": 6, "every": 0,
         "precision": "fp64"},
        # extrapolation of a field out of a level set on the largest grid
        {"name": "extrapolate_256", "kind": "extrapolate", "coarsest": 64, "levels": 3, "reach": 6.0},
        # the uniform 2-D solver at its example's size
        {"name": "frame2d_192x384", "kind": "frame2d", "nx": 192, "ny": 384, "adaptive": True},
        # a small odd 2-D grid
        {"name": "frame2d_45x83", "kind": "frame2d", "nx": 45, "ny": 83, "adaptive": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "solve", "box", "advect", "window", "extrapolate", "frame2d"])
    if kind == "box":
        while True:
            nx, ny, nz = (_log_int(rng, 7, 40) for _ in range(3))
            if 1000 <= nx * ny * nz <= 9000:
                return {"kind": "box", "nx": nx, "ny": ny, "nz": nz, "precision": rng.choice(["fp64", "mixed"])}
    if kind == "frame2d":
        nx = _log_int(rng, 24, 160)
        return {"kind": "frame2d", "nx": nx, "ny": max(32, min(384, int(nx * (1 + rng.random())))),
                "adaptive": rng.random() < 0.7}
    if kind == "window":
        return {"kind": "window", "coarsest": _log_int(rng, 8, 32), "levels": 2, "steps": rng.randint(2, 6),
                "every": rng.choice([0, 2]), "precision": rng.choice(["fp64", "mixed"])}
    levels = rng.choice([2, 3, 3, 4])
    c = _log_int(rng, 8, min(63, 256 >> (levels - 1)))
    if kind == "step":
        return {"kind": "step", "coarsest": c, "levels": levels, "precision": rng.choice(["fp64", "mixed"]),
                "frozen": True, "collider": rng.random() < 0.3, "cfl": rng.random() < 0.3}
    if kind == "solve":
        return {"kind": "solve", "coarsest": c, "levels": levels, "precision": rng.choice(["fp64", "mixed"]),
                "nrhs": 1 if c > 40 else rng.choice([1, 3, 8, 20])}
    if kind == "extrapolate":
        return {"kind": "extrapolate", "coarsest": c, "levels": levels, "reach": round(2.0 + 5.0 * rng.random(), 2)}
    return {"kind": "advect", "coarsest": c, "levels": levels}


# ---------------------------------------------------------------- what a program has in hand


def _plume(case, seed, steps=3):
    """A running simulation: the scene with its own curl noise, after a few frames."""
    s = ast_solver.OctreeSmoke3(case["coarsest"], case["levels"], seed=seed + 1,
                                precision=case.get("precision", "fp64"))
    if case.get("collider"):
        s.set_collider_sphere()
    for _ in range(steps):
        s.update(DT)
    return s


def _load(s, state):
    for k, v in state.items():
        s.set_tensor(k, v)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        s = _plume(case, seed)
        s.useFixedTimeStep = not case["cfl"]
        if not case["frozen"]:
            return {"case": case, "s": s, "x": None}
        s.set_tilt_adaptivity(False)
        return {"case": case, "s": s, "x": {k: s.get_tensor(k) for k in SCALARS + VELOCITY}}
    if kind == "solve":
        s = _plume(case, 0, 2)  # one system; the right-hand sides are the seed's
        rp, col, val, b = (s.get(k) for k in ("A_rowptr", "A_col", "A_val", "b"))
        r = np.random.default_rng(seed)
        B = np.stack([b + 0.1 * np.abs(b).max() * r.standard_normal(len(b)) for _ in range(case["nrhs"])])
        return {"case": case, "s": s, "A": (rp, col, val), "B": B}
    if kind == "box":
        A, b = _box(case, seed)
        # a handle whose capacity holds the caller's system (it solves, it does not step)
        return {"case": case, "s": ast_solver.OctreeSmoke3(24, 2), "A": A, "B": b[None, :]}
    if kind == "advect":
        s = _plume(case, seed)
        s.set_tilt_adaptivity(False)
        for i in range(5):
            s.stage(i, DT)
        return {"case": case, "s": s, "x": {k: s.get_tensor(k) for k in SCALARS + VELOCITY + DUAL}}
    if kind == "window":
        s = _plume(case, seed, 4)
        s.set_tilt_adaptivity(False)
        x = {k: s.get_tensor(k) for k in SCALARS}
        one = torch.ones(s.slots, dtype=torch.float64, device="cuda")
        p = [s.get_tensor("mac"), s.get_tensor("tilt_vel"), one, one.clone()]
        z = s.get("slot_coords")
        lev = np.repeat(np.arange(case["levels"]), s.get("level_sizes")[:, 2])
        pos = (z[:, :3] + 0.5) * ((1.0 / s.size(2)) * 2.0 ** lev)[:, None]
        goal = np.exp(-((pos - np.array([0.5, 0.5, 0.2])) ** 2).sum(1) / (2 * 0.1 ** 2))
        return {"case": case, "s": s, "x": x, "p": p, "goal": torch.tensor(goal, device="cuda")}
    if kind == "extrapolate":
        s = _plume(case, seed, 2)
        res = case["coarsest"] << (case["levels"] - 1)
        r = np.random.default_rng(seed)
        c, rad = np.array([0.5, 0.5, 0.15]) + 0.01 * r.standard_normal(3), 0.08 + 0.01 * r.random()
        x = (np.arange(res) + 0.5) / res
        sdf = np.sqrt((x[None, None, :] - c[0]) ** 2 + (x[None, :, None] - c[1]) ** 2
                      + (x[:, None, None] - c[2]) ** 2) - rad
        return {"case": case, "s": s, "sdf": sdf, "x": {k: s.get_tensor(k) for k in SCALARS[:2]}}
    if kind == "frame2d":
        nx, ny = case["nx"], case["ny"]
        s = ast_solver.ASTSolver2(resolution=[nx, ny], dx=1.0 / nx, adaptive_dofs=case["adaptive"], name="frames")
        s.initialize()
        for _ in range(4):
            s.update(DT_2D)
        x = {k: s.get(k) for k in FIELDS_2D}
        r = np.random.default_rng(seed)
        for k in ("mac_x", "mac_y"):  # another flow for another seed
            x[k] = x[k] * (1 + 1e-2 * r.standard_normal(x[k].shape))
        return {"case": case, "s": s, "x": x}
    raise ValueError(kind)


def run(state):
    case, s, kind = state["case"], state["s"], state["case"]["kind"]
    if kind == "step":
        if state["x"] is not None:
            _load(s, state["x"])
        s.update(0.03 if case["cfl"] else DT)
        return {k: s.get_tensor(k) for k in SCALARS + VELOCITY}
    if kind in ("solve", "box"):
        rp, col, val = state["A"]
        if len(state["B"]) == 1:
            return s.solve(rp, col, val, state["B"][0], precision=case["precision"])[0]
        return s.solve_batch(rp, col, val, state["B"], precision=case["precision"])[0]
    if kind == "advect":
        _load(s, state["x"])
        s.stage(5, DT)
        return {k: s.get_tensor(k) for k in SCALARS + VELOCITY}
    if kind == "window":
        _load(s, state["x"])
        p = [t.detach().requires_grad_() for t in state["p"]]
        d = ast_solver.OctreeSmokeFunction.apply(s, case["steps"], DT, case["every"], *p)
        ((d - state["goal"]) ** 2).sum().backward()
        return {"density": d.detach(), "grads": [t.grad for t in p]}
    if kind == "extrapolate":
        _load(s, state["x"])
        s.extrapolate("density", state["sdf"], 0.0, case["reach"])
        return {k: s.get_tensor(k) for k in SCALARS[:2]}
    for k, v in state["x"].items():
        s.set(k, v)
    s.update(DT_2D)
    return {"density": s.getDensity(), "mac_x": s.get("mac_x"), "mac_y": s.get("mac_y")}


# ---------------------------------------------------------------- bytes and operations


def _cells(case):
    """Unknowns of the scene's octree: the coarsest grid, and the refined region around the source
    (a ball of about 0.06 + 2 cells per level)."""
    n = case["coarsest"] ** 3
    for k in range(1, case["levels"]):
        res = case["coarsest"] << k
        n += 0.875 * 4.19 * (0.06 + 4.0 / res) ** 3 * res ** 3
    return n


def work(case):
    """Bytes: the fields or the system read once and the results written once; operations: one
    residual of the system (what a solver cannot do without) or the interpolation of each unknown."""
    kind = case["kind"]
    if kind == "step":
        n = _cells(case)
        return {"bytes": 240.0 * n, "flops": 600.0 * n}
    if kind == "solve":
        n = _cells(case)
        return {"bytes": 12 * 8.0 * n + 16.0 * n * case["nrhs"], "flops": 32.0 * n * case["nrhs"]}
    if kind == "box":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 12 * 7.0 * n + 16.0 * n, "flops": 28.0 * n}
    if kind == "advect":
        n = _cells(case)
        return {"bytes": 288.0 * n, "flops": 500.0 * n}
    if kind == "window":
        n = _cells(case)
        return {"bytes": 480.0 * n * case["steps"], "flops": 1800.0 * n * case["steps"]}
    if kind == "extrapolate":
        res = case["coarsest"] << (case["levels"] - 1)
        return {"bytes": 8.0 * res ** 3 + 32.0 * _cells(case), "flops": 30.0 * _cells(case)}
    n = case["nx"] * case["ny"]
    return {"bytes": 160.0 * n, "flops": 400.0 * n}


# ---------------------------------------------------------------- the caller's own matrix


def _box(case, seed):
    """Poisson's equation on a box of nx x ny x nz cells, a tenth of them solid and left out, open
    at the top: CSR rows sorted by column, and a right-hand side of seeded noise."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    fluid = np.random.default_rng(nx + 100 * ny + 10000 * nz).random((nz, ny, nx)) > 0.1
    index = np.full((nz + 2, ny + 2, nx + 2), -1, dtype=np.int64)
    n = int(fluid.sum())
    index[1:-1, 1:-1, 1:-1][fluid] = np.arange(n)
    zyx = np.argwhere(fluid) + 1
    near = [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1), (0, 1, 0), (1, 0, 0)]
    cols = np.stack([index[tuple((zyx + np.array(o)).T)] for o in near], axis=1)
    diag = (cols >= 0).sum(1) + (zyx[:, 0] == nz) + 1e-3
    six = np.concatenate([cols[:, :3], np.arange(n)[:, None], cols[:, 3:]], axis=1)
    val = np.concatenate([-np.ones((n, 3)), diag[:, None], -np.ones((n, 3))], axis=1)
    keep = six >= 0
    rowptr = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return (rowptr, six[keep].astype(np.int32), val[keep]), np.random.default_rng(seed).standard_normal(n)


def exact(case, seed):
    """The caller's own system solved directly in 64 bits; the octree and 2-D cases have no value
    that a few lines of torch give."""
    if case["kind"] != "box":
        return None
    (rp, col, val), b = _box(case, seed)
    n = len(b)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.zeros((n, n), dtype=torch.float64, device=dev)
    rows = np.repeat(np.arange(n), np.diff(rp))
    A[torch.tensor(rows, device=dev), torch.tensor(col.astype(np.int64), device=dev)] = torch.tensor(val, device=dev)
    return torch.linalg.solve(A, torch.tensor(b, device=dev)).cpu().numpy()
