"""A schedule that the particle batch refuses leaves it as it was."""
import numpy as np
import pytest

from conftest import seeded_m
from test_gpu_teams import _particle

pytestmark = pytest.mark.gpu


def test_refused_schedule_changes_nothing():
    from nmag import _lib
    from nmag.batch import ParticleBatch
    parts = [_particle(b) for b in ((3, 3, 3), (4, 3, 2))]
    ms = [seeded_m(m.n_nodes, base=(0.2, 1.0, 0.3), seed=k, noise=0.2) for k, (m, _) in enumerate(parts)]
    steps = []
    for refused in (False, True):
        b = ParticleBatch([p for _, p in parts], n_stages=3, h_max=0.3, rtol=1e-7, atol=1e-7, cg_rtol=1e-10)
        b.set_m(ms)
        if refused:
            with pytest.raises(_lib.NmagGpuError):
                b.set_schedule(1024, 1e12)       # more threads than the kernel's registers allow
        b.run(20)
        st = b.state()
        steps.append((st["steps"].tolist(), st["t"].tolist()))
        b.close()
    assert steps[0] == steps[1]
    assert max(steps[0][0]) > 0
