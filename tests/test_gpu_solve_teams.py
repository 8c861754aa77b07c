"""The cooperative pressure solve (photon_gb300/csrc/solve.cuh) at the sizes where
its division of the work changes: grids of one to three cells per axis, odd and
even rows, a block count at and past each tile shape (512 and 4,096 groups of
eight 2x2x2 blocks), blocks split by solid cells, and faces that are only partly
open (cells that read the coefficient arrays).

FP64: one V-cycle against the oracle within 1e-12 relative L2, the bar of the
other parity tests. Mixed: the solve's FP64 residual meets the stop and its
pressure is the FP64 path's converged one within 1e-5, the path's bar per step.
The number of CTAs must not change a bit of either."""
import ctypes

import numpy as np
import pytest

from oracle.oraclepy import OracleSolver
from photon_gb300 import _lib, casegen
from photon_gb300.solver import Batch, Solver, make_grid

from gpu_util import STATE, rel_l2


def grid(dims, solid=0.0, partial=0.0, seed=0):
    """Gas in a box open at its sides and top; a share of solid cells and of faces half open."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    blocked = (rng.random((nz, ny, nx)) < solid).astype(np.uint8)
    blocked[0, 0, 0] = 0
    c = casegen.from_blocked("grid_%dx%dx%d" % dims, blocked, 0.1)
    for f, a in (("fx", "ax"), ("fy", "ay"), ("fz", "az")):
        open_ = getattr(c, f)
        half = (rng.random(open_.size) < partial) & (open_ > 0)
        open_[half] = 0.5
        getattr(c, a)[half] = 0.5
    c.profile.tol = 0.0
    c.profile.rel_tol = 1e-8
    return c


GRIDS = [((1, 1, 1), 0, 0), ((2, 1, 1), 0, 0), ((1, 3, 2), 0, 0), ((3, 3, 3), 0, 0), ((5, 2, 7), 0.2, 0.1),
         ((16, 16, 2), 0, 0), ((17, 5, 3), 0.3, 0.2), ((18, 16, 4), 0.1, 0), ((33, 9, 8), 0.2, 0.1),
         ((32, 32, 32), 0, 0), ((33, 32, 32), 0.1, 0.05), ((34, 32, 32), 0, 0), ((64, 64, 64), 0, 0), ((65, 64, 64), 0.05, 0.01)]
IDS = ["%dx%dx%d" % g[0] for g in GRIDS]


@pytest.mark.gpu
@pytest.mark.parametrize("dims,solid,partial", GRIDS, ids=IDS)
def test_vcycle_matches_oracle(dims, solid, partial):
    c = grid(dims, solid, partial)
    o, g = OracleSolver(c), Solver(c)
    o.stage("zones")
    o.step(1e-3)
    r = np.random.default_rng(1).standard_normal(c.N) * (1 - c.blocked)
    assert rel_l2(g.precondition(r), o.precondition(r)) <= 1e-12


def project(c, precision, rel_tol):
    c.profile.rel_tol = rel_tol
    g = Solver(c, precision)
    rng = np.random.default_rng(2)
    for f in "uvw":
        g.set(f, rng.standard_normal(len(g.get(f))) * (getattr(c, "f" + "xyz"["uvw".index(f)]) > 0))
    g.stage("project", 0.01)
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("dims,solid,partial", GRIDS, ids=IDS)
def test_mixed_solve_meets_the_stop(dims, solid, partial):
    m = project(grid(dims, solid, partial), _lib.PREC_MIXED, 1e-8)
    assert m.stats()["pressure_rel_residual"] <= 1e-8
    d = project(grid(dims, solid, partial), _lib.PREC_FP64, 1e-12)
    assert rel_l2(m.get("p"), d.get("p")) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", [1, 2, 7])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_teams_do_not_change_the_result(precision, ctas, monkeypatch):
    cs = [casegen.house(40, 32, 24, 0.2, 5), casegen.tiny_room(13, 11, 9, 0.2), casegen.tiny_room(10, 8, 8, 0.2, doorway=False)]
    for c in cs:
        c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    whole = [Solver(c, precision) for c in cs]
    for g in whole:
        g.run(4, 0.02)
    monkeypatch.setenv("PHX_PERSIST_CTAS", str(ctas))
    few, batch = Solver(cs[0], precision), Batch(cs, precision)
    few.run(4, 0.02)
    batch.run(4, 0.02)
    for f in STATE:
        assert np.array_equal(few.get(f), whole[0].get(f)), f
        for s, g in enumerate(whole):
            assert np.array_equal(batch.get(s, f), g.get(f)), (s, f)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_a_large_batch_equals_its_scenarios_alone(precision):
    """24 scenarios: the FP32 solve runs two CTAs per SM instead of one."""
    shapes = [(13, 11, 9), (10, 8, 8), (9, 7, 5), (16, 12, 8), (21, 10, 9), (33, 12, 10), (12, 12, 12), (40, 9, 7)]
    cs = [casegen.tiny_room(*d, 0.2) for d in shapes]
    for c in cs:
        c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    batch = Batch([cs[q % len(cs)] for q in range(24)], precision)
    batch.run(3, 0.02)
    for s, c in enumerate(cs):
        alone = Solver(c, precision)
        alone.run(3, 0.02)
        for f in STATE:
            for q in range(s, 24, len(cs)):
                assert np.array_equal(batch.get(q, f), alone.get(f)), (q, f)


@pytest.mark.parametrize("precision,widest", [(_lib.PREC_FP64, 410), (_lib.PREC_MIXED, 776)])
def test_rows_past_the_widest_are_refused(precision, widest):
    """Rejected on the host, before any device call."""
    g, keep = make_grid(grid((widest + 1, 2, 2)))
    h = ctypes.c_void_p()
    assert _lib.load().phx_create(ctypes.byref(g), precision, ctypes.byref(h)) == _lib.PHX_ERR_UNSUPPORTED
