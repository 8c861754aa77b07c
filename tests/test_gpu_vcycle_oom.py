"""The V-cycle tuner on a GPU whose memory is taken: it reports that it cannot allocate,
and leaves the context as it was -- its hierarchy, its fields and the steps that
follow are those of a context that was never tuned."""
import numpy as np
import pytest
import torch

from photon_gb300 import _lib, casegen
from photon_gb300.solver import Batch

from gpu_util import STATE

pytestmark = pytest.mark.gpu


def test_failed_tuning_changes_nothing(monkeypatch):
    monkeypatch.setenv("PHX_COARSE_SWEEPS", "2")
    c = casegen.house(144, 104, 88, 0.1, 1)
    c.profile.tol, c.profile.rel_tol = 0.0, 1e-8
    b, twin = Batch([c], _lib.PREC_MIXED), Batch([c], _lib.PREC_MIXED)
    for x in (b, twin):
        x.run(3, 0.02)
    # from too little for the copy of the state up to just too little for a second hierarchy
    seen = []
    for leave in range(int(0.5 * b.device_bytes()), b.device_bytes(), 32 << 20):
        taken = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
        try:
            with pytest.raises(_lib.PhxError) as e:
                b.tune_vcycle(1, 0.02)
        finally:
            del taken
            torch.cuda.empty_cache()
        seen.append(str(e.value))
        for f in STATE:
            assert np.array_equal(b.get(0, f), twin.get(0, f)), (f, seen)
        for x in (b, twin):
            x.run(1, 0.02)
        if "multigrid levels" in seen[-1]:
            break
    assert "multigrid levels" in seen[-1], seen
    assert b.mg_levels(0) == twin.mg_levels(0)
    for x in (b, twin):
        x.run(2, 0.02)
    for f in STATE:
        assert np.array_equal(b.get(0, f), twin.get(0, f)), f
