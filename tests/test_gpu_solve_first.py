"""The first solve of a building that joins a running batch, new or restored from a
checkpoint: its longest, whose team must not be sized by a count of iterations it has
not made yet."""
import ctypes

import pytest

from photon_gb300 import _lib, casegen
from photon_gb300.solver import STAT_KEYS, Batch

pytestmark = pytest.mark.gpu


def stop(c):
    c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    return c


def first_step_ms(precision, restored):
    """A 72x52x44 house joins 40 running rooms: time of the step it joins in."""
    b = Batch([stop(casegen.tiny_room(36, 24, 24, 0.1)) for _ in range(40)], precision)
    b.run(4, 0.02)
    s = b.add(stop(casegen.house(72, 52, 44, 0.2, 1)))
    if restored:
        st = _lib.PhxStats()
        for k in STAT_KEYS:
            v = b.stats(s)[k]
            setattr(st, k, 12.5 if k == "time" else v)
        assert b.L.phx_batch_set_stats(b.h, s, ctypes.byref(st)) == 0
        assert b.stats(s)["time"] == 12.5
    ms = b.time_steps(1, 0.02)[0]
    b.close()
    return ms


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["fp64", "mixed"])
def test_restored_joins_as_fast_as_new(precision):
    new = min(first_step_ms(precision, False) for _ in range(3))
    restored = min(first_step_ms(precision, True) for _ in range(3))
    assert restored < 2.0 * new, (restored, new)
