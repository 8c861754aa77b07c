"""Batches whose scenarios are more than the solve's CTAs, or a few large ones among
very many small ones: small scenarios share CTAs by turns, large ones keep a team.
Neither changes a bit of a scenario, and a large building does not wait with a
few CTAs for a solve it could spread over the GPU."""
import numpy as np
import pytest

from photon_gb300 import _lib, casegen
from photon_gb300.solver import Batch, Solver

from gpu_util import STATE

pytestmark = pytest.mark.gpu

BOTH = pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["fp64", "mixed"])


def stop(c):
    c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    return c


def closet():
    return stop(casegen.tiny_room(13, 11, 9, 0.2))


def house():
    return stop(casegen.house(72, 52, 44, 0.2, 1))


@BOTH
@pytest.mark.parametrize("ctas", [3, 8, 40, 64])
def test_sharing_does_not_change_the_result(precision, ctas, monkeypatch):
    kinds = [stop(casegen.house(40, 32, 24, 0.2, 5)), closet(), stop(casegen.tiny_room(7, 6, 5, 0.2)),
             stop(casegen.tiny_room(10, 8, 8, 0.2, doorway=False))]
    order = [1, 2, 3] * 10 + [0] + [2, 1, 3] * 10
    alone = [Solver(c, precision) for c in kinds]
    for g in alone:
        g.run(4, 0.02)
    monkeypatch.setenv("PHX_PERSIST_CTAS", str(ctas))
    batch = Batch([kinds[k] for k in order], precision)
    batch.run(4, 0.02)
    for s, k in enumerate(order):
        for f in STATE:
            assert np.array_equal(batch.get(s, f), alone[k].get(f)), (s, f)


def device_ms(cases, precision):
    b = Batch(cases, precision)
    b.run(6, 0.02)
    ms = min(b.time_steps(3, 0.02)[0] / 3 for _ in range(3))
    b.close()
    return ms


@pytest.mark.parametrize("precision,closets", [(_lib.PREC_FP64, 280), (_lib.PREC_FP64, 140), (_lib.PREC_MIXED, 300), (_lib.PREC_MIXED, 500)],
                         ids=["fp64-280", "fp64-140", "mixed-300", "mixed-500"])
def test_a_large_building_keeps_its_ctas(precision, closets):
    """A step takes no more than twice what the large building and the small ones take by themselves."""
    small = [closet() for _ in range(closets)]
    apart = device_ms([house()], precision) + device_ms(small, precision)
    assert device_ms([house()] + small, precision) < 2.0 * apart
