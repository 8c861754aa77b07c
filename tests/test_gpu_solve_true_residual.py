"""The FP64 solve's residual is a recurrence, and so is its q = A d: at stops down to the
rounding floor the pressure's own residual b - A p, formed in extended precision from
the fields, must be what the solve reports. Each iteration rounds p and r once and A's
rows sum to at most 12, so the two differ by at most iterations x 12 u max|p| / max|b|."""
import numpy as np
import pytest

from photon_gb300 import casegen
from photon_gb300.solver import Solver

pytestmark = pytest.mark.gpu

L = np.longdouble


def system(c, before, dt):
    """b, the operator and its diagonal over the fields before the projection
    (src/sim/gasphase.cpp:528-549)."""
    nx, ny, nz = c.nx, c.ny, c.nz
    shape = dict(x=(nz, ny, nx + 1), y=(nz, ny + 1, nx), z=(nz + 1, ny, nx))
    f, a, v = ({k: np.asarray(src(k), L).reshape(shape[k]) for k in "xyz"}
               for src in (lambda k: getattr(c, "f" + k), lambda k: getattr(c, "a" + k), lambda k: before["uvw"["xyz".index(k)]]))
    F = {k: f[k] * v[k] for k in "xyz"}
    div = (F["x"][:, :, 1:] - F["x"][:, :, :-1] + F["y"][:, 1:] - F["y"][:, :-1] + F["z"][1:] - F["z"][:-1]) / L(c.dx)
    b = (np.asarray(before["S"], L).reshape(nz, ny, nx) - div) * (L(c.dx) * L(c.dx) / L(dt))

    def head(u, inward):   # Bernoulli head of an inflow
        return np.where(inward * u > 0, L(-0.5) * u * u, L(0))
    b[:, :, 0] += a["x"][:, :, 0] * head(v["x"][:, :, 0], 1)
    b[:, :, -1] += a["x"][:, :, -1] * head(v["x"][:, :, -1], -1)
    b[:, 0] += a["y"][:, 0] * head(v["y"][:, 0], 1)
    b[:, -1] += a["y"][:, -1] * head(v["y"][:, -1], -1)
    b[-1] += a["z"][-1] * head(v["z"][-1], -1)
    dg = a["x"][:, :, 1:] + a["x"][:, :, :-1] + a["y"][:, 1:] + a["y"][:, :-1] + a["z"][1:] + a["z"][:-1]
    live = (c.blocked.reshape(nz, ny, nx) == 0) & (dg > 0)

    def apply(p):
        P = np.pad(np.asarray(p, L).reshape(nz, ny, nx), 1)
        return (dg * P[1:-1, 1:-1, 1:-1] - a["x"][:, :, :-1] * P[1:-1, 1:-1, :-2] - a["x"][:, :, 1:] * P[1:-1, 1:-1, 2:]
                - a["y"][:, :-1] * P[1:-1, :-2, 1:-1] - a["y"][:, 1:] * P[1:-1, 2:, 1:-1]
                - a["z"][:-1] * P[:-2, 1:-1, 1:-1] - a["z"][1:] * P[2:, 1:-1, 1:-1])
    return np.where(live, b, 0), lambda p: np.where(live, apply(p), 0)


def building(kind):
    if kind == "room":
        return casegen.tiny_room(36, 24, 24, 0.1)
    c = casegen.house(40, 32, 24, 0.2, 5)
    if kind == "partial":
        rng = np.random.default_rng(3)
        for f, a in (("fx", "ax"), ("fy", "ay"), ("fz", "az")):
            half = (rng.random(getattr(c, f).size) < 0.05) & (getattr(c, f) > 0)
            getattr(c, f)[half] = getattr(c, a)[half] = 0.5
    return c


@pytest.mark.parametrize("stop", [1e-8, 1e-12, 0.0])
@pytest.mark.parametrize("kind", ["room", "house", "partial"])
def test_reported_residual_is_the_pressures(kind, stop):
    c = building(kind)
    c.profile.tol, c.profile.rel_tol, c.profile.maxIters = 0.0, stop, 100
    g = Solver(c)
    rng = np.random.default_rng(7)
    for f in "uvw":
        v = rng.standard_normal(len(g.get(f))) * (getattr(c, "f" + "xyz"["uvw".index(f)]) > 0)
        g.set(f, v)
    g.set("S", 0.1 * rng.standard_normal(c.N) * (c.blocked == 0))
    before = {f: g.get(f) for f in ("u", "v", "w", "S")}
    g.stage("project", 0.01)
    b, apply = system(c, before, 0.01)
    p, scale = g.get("p"), np.abs(b).max()
    true = float(np.abs(b - apply(p)).max() / scale)
    st = g.stats()
    assert st["pressure_rel_residual"] <= stop or st["pressure_iters"] == 100
    gap = float(st["pressure_iters"] * 12 * 2.0 ** -53 * np.abs(p).max() / scale)
    assert abs(true - st["pressure_rel_residual"]) <= gap, (true, st["pressure_rel_residual"], gap)
