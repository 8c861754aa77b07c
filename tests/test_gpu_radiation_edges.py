"""The radiation trace where its kernels' shapes can go wrong, against the oracle's
FP64 trace: element counts around a CTA's 128 and a warp's 32, a cell count that
is no multiple of four (flags are set by words), walls on the domain's own
boundary faces, origins outside the grid, spheres, and soot from clear air to
opaque cells (absorption on both sides of the 1e-3 switch and past the cutoff of
the exponential).

Tolerances: an element sums 32 rays of at most some 50 cells, a cell's gain as
many terms; FP64 rounding (1.1e-16 each, band differences cancelling to a
hundredth of their terms) stays below 1e-12 of the norm, FP32 (6e-8) below 1e-4."""
import numpy as np
import pytest

from oracle import oraclepy
from photon_gb300 import _lib, casegen
from photon_gb300.solver import Solver

from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


def scene(n_el, seed):
    nx, ny, nz, dx = 13, 11, 7, 0.25
    rng = np.random.default_rng(seed)
    blocked = (rng.random((nz, ny, nx)) < 0.08).astype(np.uint8)
    c = casegen.from_blocked("rad_edges", blocked, dx, (0.5, -1.0, 0.0))
    n = nx * ny * nz
    gas = {"T": 293.15 + 900.0 * rng.random(n), "Ys": 10.0 ** rng.uniform(-9, -1, n), "Yc": 0.1 * rng.random(n),
           "Yw": 0.1 * rng.random(n), "hrr": np.where(rng.random(n) < 0.1, 5e5, 0.0), "Pb": np.full(n, 101325.0)}
    gas = {f: gas[f] for f in oraclepy.RAD_GAS_FIELDS}
    faces = [(nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1)]
    wl = []
    for axis, m in enumerate(faces):
        for f in rng.choice(m, m // 6, replace=False):
            wl.append((axis, f, 293.15 + 300 * rng.random(), 293.15 + 300 * rng.random()))
    el = np.zeros((n_el, 11))
    size = np.array([nx, ny, nz]) * dx
    el[:, 0:3] = np.array([0.5, -1.0, 0.0]) + size * rng.uniform(-0.05, 1.05, (n_el, 3))
    nrm = rng.normal(size=(n_el, 3))
    el[:, 3:6] = nrm / np.linalg.norm(nrm, axis=1)[:, None]
    axis_aligned = rng.random(n_el) < 0.5
    el[axis_aligned, 3:6] = np.eye(3)[rng.integers(0, 3, axis_aligned.sum())]
    el[:, 6] = dx * dx
    el[:, 7] = rng.uniform(0.3, 1.0, n_el)
    el[:, 8] = 293.15 + 700 * rng.random(n_el)
    el[:, 9] = rng.random(n_el) < 0.2
    el[:, 10] = el[:, 9]
    return c, gas, el, np.array(wl, float), 293.15 + 200 * rng.random(n)


@pytest.mark.parametrize("n_el", [1, 31, 33, 127, 128, 129, 400])
@pytest.mark.parametrize("precision,tol", [(_lib.PREC_FP64, 1e-12), (_lib.PREC_MIXED, 1e-4)])
def test_trace_at_the_edges_of_its_kernels(n_el, precision, tol):
    c, gas, el, wl, solid = scene(n_el, 40 + n_el)
    g = Solver(c, precision)
    for f, a in gas.items():
        g.set(f, a)
    ab, gain = g.rad_trace(el, wl, solid)
    oab, ogain = oraclepy.rad_trace((c.nx, c.ny, c.nz), (c.dx, c.ox, c.oy, c.oz), c.blocked, gas, el, wl, solid)
    assert rel_l2(ab, oab) <= tol
    assert rel_l2(gain, ogain) <= tol


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_records_and_rows_are_the_same_elements(precision):
    """Elements as an (n, 11) array and as phx_rad_elem records: the same bits."""
    c, gas, el, wl, solid = scene(130, 7)
    g = Solver(c, precision)
    for f, a in gas.items():
        g.set(f, a)
    ab1, _ = g.rad_trace(el, wl, solid)
    ab2, _ = g.rad_trace(_lib.rad_elements(el), _lib.rad_walls(wl), solid)
    np.testing.assert_array_equal(ab1, ab2)
