"""The volume march steps over bricks of cells that cannot change a pixel. A heat
release of 11,050 W/m3 everywhere marks every brick, and drives a flame by 0.0099,
below the shader's threshold of 0.01: where no cell is above 1000 K (heat adds to the
drive) it adds nothing. So a sparse scene with and without it must give the same
image, bit for bit -- on grids whose sides are and are not multiples of a brick's
four cells, with smoke and glowing soot in single cells next to brick sides, far from the origin, from outside and inside the box, with and
without the slice, and with steps from a fraction of a cell to several cells."""
import numpy as np
import pytest

from photon_gb300 import _lib, casegen, render
from photon_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("dims,origin,inside,slice_z,step", [
    ((13, 11, 7), (0.0, 0.0, 0.0), False, None, 0.3),
    ((16, 8, 8), (0.0, 0.0, 0.0), False, 0.9, 0.3),
    ((13, 11, 7), (3000.0, -2000.0, 0.0), False, 0.7, 0.3),
    ((21, 10, 9), (-5.0, 1.0, 0.0), True, None, 0.05),
    ((21, 10, 9), (-5.0, 1.0, 0.0), True, 1.1, 1.7),
])
def test_skipped_bricks_change_nothing(precision, dims, origin, inside, slice_z, step):
    nx, ny, nz = dims
    dx, n = 0.25, nx * ny * nz
    rng = np.random.default_rng(nx * ny + nz)
    c = casegen.from_blocked("bricks", np.zeros((nz, ny, nx), np.uint8), dx, origin)
    thick = rng.random(n) < 0.04
    soot = np.where(thick, 10.0 ** rng.uniform(-6, -2, n), 0.0)
    T = np.where(rng.random(n) < 0.01, 900.0, 293.15)
    g = Solver(c, precision)
    for f, a in (("T", T), ("Ys", soot), ("Ya", 0.3 * soot), ("Pb", np.full(n, 101325.0))):
        g.set(f, a)
    size = np.array(dims) * dx
    at = np.array(origin)
    eye = at + size * (0.45 if inside else np.array([-0.8, -1.1, 1.3]))
    p = render.camera(c, tuple(eye), tuple(at + size * np.array([0.6, 0.5, 0.4])), 97, 61, time=2.0, slice_z=slice_z,
                      lights=[(at[0], at[1], 1.0, 2.0)])
    p.step = step * dx
    images = []
    for q in (0.0, 11050.0):
        g.set("hrr", np.full(n, q))
        images.append(g.vol_render(p))
    np.testing.assert_array_equal(images[0], images[1])
    assert np.ptp(images[0]) > 0.05
