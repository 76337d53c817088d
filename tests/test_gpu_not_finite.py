"""A state on the device that is not a number: the direct solver's evaluation is
an error that says so, and leaves no trace in a later one."""
import numpy as np
import pytest

from conftest import permalloy, seeded_m
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_direct_solves(cube, bad):
    import torch
    from nmag import _lib
    eng = make_engine(cube, permalloy(0.1))
    m = seeded_m(len(cube.points), seed=5, noise=0.4)
    eng.set_m(m)
    eng.ts_init()
    good = eng.eval_fields()
    worse = m.copy()
    worse[700, 1] = bad
    d = torch.tensor(worse.reshape(-1), dtype=torch.float64, device="cuda")
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    with pytest.raises(_lib.NmagGpuError, match="non-finite"):
        eng.rhs_device(d.data_ptr(), out.data_ptr())
    again = eng.eval_fields()
    for key in good:
        assert np.array_equal(good[key], again[key]), key
    eng.close()
