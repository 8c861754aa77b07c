"""Closed zones large enough that a team of several CTAs solves them: the zone means that
each iteration removes (mixed) and the crack faces' network, which the small sealed
rooms of the other tests leave to one CTA. FP64 against the oracle within 1e-9 per
step; both paths with one CTA and with all of them, bit for bit."""
import numpy as np
import pytest

from oracle.oraclepy import OracleSolver
from photon_gb300 import _lib, casegen
from photon_gb300.solver import Solver

from gpu_util import STATE, rel_l2

pytestmark = pytest.mark.gpu


def sealed():
    return casegen.tiny_room(36, 24, 24, 0.1, 60e3, doorway=False)


def two_leaky_rooms():
    """Two sealed rooms with crack faces between them and to the outside."""
    c = casegen.tiny_room(40, 26, 22, 0.1, 60e3, doorway=False)
    shape = (c.nz, c.ny, c.nx + 1)
    fx, lx, ax = c.fx.reshape(shape), c.lx.reshape(shape), c.ax.reshape(shape)
    for where, share in (((slice(1, 6), slice(3, 9), 0), 0.01), ((slice(None), slice(None), 17), 0.02)):
        fx[where], lx[where], ax[where] = share, 1, 0
    return c


CASES = {"sealed": sealed, "leaky": two_leaky_rooms}


@pytest.mark.parametrize("name", list(CASES))
def test_steps_match_oracle(name):
    c = CASES[name]()
    o, g = OracleSolver(c), Solver(c)
    for s in range(6):
        dto, dtg = o.step(0.02), g.step(0.02)
        assert abs(dtg - dto) <= 1e-12 * dto
        bad = {f: rel_l2(g.get(f), o.get(f)) for f in STATE}
        assert all(e <= 1e-9 for e in bad.values()), (s, bad)
    assert g.stats()["pressure_iters"] == o.scalars()["pressureIters"]


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["fp64", "mixed"])
def test_one_cta_or_many(name, precision, monkeypatch):
    c = CASES[name]()
    c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    many = Solver(c, precision)
    monkeypatch.setenv("PHX_PERSIST_CTAS", "1")
    one = Solver(c, precision)
    for g in (many, one):
        g.run(6, 0.02)
    assert many.stats()["pressure_rel_residual"] <= 1e-8
    for f in STATE:
        assert np.array_equal(many.get(f), one.get(f)), f
