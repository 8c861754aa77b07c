"""Waits of the pressure solve's team: one that runs out ends the kernel with an error
the host reads, and a coarsest level that one thread solves (more than 4,096 unknowns,
src/sim/pressure_mg.cpp:258-266) is waited for as long as its sweeps take."""
import numpy as np
import pytest

from oracle.oraclepy import OracleSolver
from photon_gb300 import _lib, casegen
from photon_gb300.solver import Solver

from gpu_util import STATE, rel_l2

BOTH = pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["fp64", "mixed"])


def chimneys(n=70, height=4):
    """n x n columns closed to one another, open at the top: no level joins two of them."""
    c = casegen.from_blocked("chimneys_%d" % n, np.zeros((height, n, n), np.uint8), 0.1)
    for f in ("fx", "fy", "ax", "ay"):
        getattr(c, f)[:] = 0
    c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    return c


def test_chimneys_have_a_serial_coarsest_level():
    o = OracleSolver(chimneys())
    o.step(1e-3)
    assert o.mg()[-1]["n"] > 4096


@pytest.mark.gpu
@BOTH
def test_serial_coarsest_level_is_waited_for(precision, monkeypatch):
    """Waits of a millisecond, sweeps of some eighty."""
    monkeypatch.setenv("PHX_TEAM_WAIT_CYCLES", "2000000")
    c = chimneys()
    g = Solver(c, precision)
    rng = np.random.default_rng(2)
    r = rng.standard_normal(c.N)
    o = OracleSolver(c)
    o.stage("zones")
    o.step(1e-3)
    z = g.precondition(r)
    assert rel_l2(z, o.precondition(r)) <= (1e-12 if precision == _lib.PREC_FP64 else 1e-5)
    g.set("w", rng.standard_normal(len(g.get("w"))) * (c.fz > 0))
    g.stage("project", 0.01)
    assert g.stats()["pressure_rel_residual"] <= 1e-8


@pytest.mark.gpu
@BOTH
def test_a_wait_that_runs_out_is_an_error(precision, monkeypatch):
    def house():
        return casegen.house(40, 32, 24, 0.2, 5)
    before = Solver(house(), precision)
    monkeypatch.setenv("PHX_TEAM_WAIT_CYCLES", "0")
    g = Solver(house(), precision)
    monkeypatch.delenv("PHX_TEAM_WAIT_CYCLES")
    for _ in range(2):   # reported once per step that failed, then cleared
        with pytest.raises(_lib.PhxError) as e:
            g.step(0.02)
        assert e.value.code == _lib.PHX_ERR_TIMEOUT
        g.sync()
    after = Solver(house(), precision)
    for s in (before, after):
        s.run(3, 0.02)
    for f in STATE:
        assert np.array_equal(before.get(f), after.get(f)), f
