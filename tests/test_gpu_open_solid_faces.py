"""Faces left open beside solid cells: nothing in a grid's description closes them
(faces_from_blocked does, the C ABI does not), and the reference steps such a grid
with the solid cell's density and pressure on one side of the face. FP64 against
the oracle, at the bars of the other parity tests: 1e-12 relative L2 for a stage,
1e-9 per step."""
import numpy as np
import pytest

from oracle.oraclepy import OracleSolver
from photon_gb300 import casegen
from photon_gb300.solver import Solver

from gpu_util import STATE, rel_l2

pytestmark = pytest.mark.gpu


def open_faces(solid, value):
    """A closed room with a burner and solid cells all of whose faces are open by `value`."""
    c = casegen.tiny_room(9, 8, 8, 0.2, 40e3)
    shape = (c.nz, c.ny, c.nx)
    blocked = c.blocked.reshape(shape)
    if solid == "block":
        blocked[3:5, 2:4, 5:7] = 1
    else:
        blocked[np.random.default_rng(4).random(shape) < 0.1] = 1
        blocked[0] = 0
    for f, a, n in (("fx", "ax", (c.nz, c.ny, c.nx + 1)), ("fy", "ay", (c.nz, c.ny + 1, c.nx)), ("fz", "az", (c.nz + 1, c.ny, c.nx))):
        axis = {"x": 2, "y": 1, "z": 0}[f[1]]
        lo, hi = np.moveaxis(blocked, axis, 0)[:-1], np.moveaxis(blocked, axis, 0)[1:]
        beside = (lo | hi) != 0
        for name in (f, a):
            inner = np.moveaxis(getattr(c, name).reshape(n), axis, 0)[1:-1]
            inner[beside] = value
    return c


CASES = [("block", 1.0), ("scattered", 1.0), ("block", 0.5)]


@pytest.mark.parametrize("solid,value", CASES)
def test_steps_from_rest(solid, value):
    c = open_faces(solid, value)
    o, g = OracleSolver(c), Solver(c)
    for s in range(4):
        dto, dtg = o.step(0.02), g.step(0.02)
        assert abs(dtg - dto) <= 1e-12 * dto, (s, dtg, dto)
        bad = {f: rel_l2(g.get(f), o.get(f)) for f in STATE}
        assert all(e <= 1e-9 for e in bad.values()), (s, bad)


@pytest.mark.parametrize("solid,value", CASES)
@pytest.mark.parametrize("stage", ["heat", "momentum", "advect"])
def test_stage(stage, solid, value):
    c = open_faces(solid, value)
    o, g = OracleSolver(c), Solver(c)
    for _ in range(4):
        o.step(0.02)
    for f in STATE:
        g.set(f, o.get(f))
    sc = o.scalars()
    g.set_scalars(sc["time"], sc["maxVel"], sc["maxNu"], sc["maxDiv"])
    o.stage(stage, 0.013)
    g.stage(stage, 0.013)
    bad = {f: rel_l2(g.get(f), o.get(f)) for f in STATE}
    assert all(e <= 1e-12 for e in bad.values()), bad
