"""A trace of more elements than are traced at a time (524,288): every element has the
bits it has in a smaller trace, the cells gain the same power (FP64: a cell's FP32
sum of some hundred thousand rays has no bound worth testing), and the scratch on
the device stays bounded."""
import numpy as np
import pytest
import torch

from photon_gb300 import _lib
from photon_gb300.solver import Solver

from gpu_util import rel_l2
from test_gpu_radiation_edges import scene

pytestmark = pytest.mark.gpu
PORTION = 1 << 19


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n_el", [PORTION, PORTION + 1, 3 * PORTION - 77])
def test_portions(n_el, precision):
    c, gas, el, wl, solid = scene(997, 5)
    many = np.tile(el, (n_el // len(el) + 1, 1))[:n_el]
    g = Solver(c, precision)
    for f, a in gas.items():
        g.set(f, a)
    one, gain = g.rad_trace(el, wl, solid)
    free = torch.cuda.mem_get_info()[0]
    ab, total = g.rad_trace(many, wl, solid)
    used = free - torch.cuda.mem_get_info()[0]
    np.testing.assert_array_equal(ab, np.tile(one, n_el // len(el) + 1)[:n_el])
    whole, rest = divmod(n_el, len(el))
    part = g.rad_trace(el[:rest], wl, solid)[1]
    if precision == _lib.PREC_FP64:
        assert rel_l2(total, whole * gain + part) <= 1e-12
    # an element's inputs and result, its rays for a portion's elements, some buffers
    assert used <= 100 * n_el + (800 if precision == _lib.PREC_MIXED else 1500) * PORTION + (32 << 20)
