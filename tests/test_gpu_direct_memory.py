"""What the direct Poisson solver's factors hold on the device.  A handle whose
solves are in mixed precision keeps the FP32 factors alone, until a gradient's
FP64 adjoint asks for the FP64 ones too."""
import numpy as np
import pytest

from conftest import permalloy, seeded_m
from test_gpu_parity import rel_err
from test_gpu_wires import _engine

pytestmark = pytest.mark.gpu


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _taken(msh, mixed):
    """Bytes that the factors of a handle take, beside the integrator's."""
    import torch
    eng = _engine(msh, mixed, 1e-9)
    eng.set_m(np.tile([1.0, 0.0, 0.0], (msh.n_nodes, 1)))
    eng.eval_fields()
    before = _free(torch)
    eng.ts_init()
    counts = np.array(eng.cg_iterations())
    eng.eval_fields()
    assert (np.array(eng.cg_iterations()) - counts <= 11).all()
    taken = before - _free(torch)
    eng.close()
    return taken


def test_mixed_precision_keeps_fp32_factors_alone():
    from nmag import mesh
    msh = mesh.box_mesh(25, 25, 25, 2.0)       # 1.7e7 factor entries: 138 MB in FP64
    full, half = _taken(msh, False), _taken(msh, True)
    print("FP64 handle %.1f MB, mixed %.1f" % (full / 1e6, half / 1e6))
    assert full > 138e6
    assert half < full - 0.4 * 138e6


def test_gradient_on_a_mixed_handle(cube):
    """The forward pass on FP32 factors, the adjoint on FP64 ones: the forward
    states are those of the handle before the FP64 factors were asked for."""
    import torch
    eng = _engine(cube, True, 1e-9)
    m = seeded_m(len(cube.points), seed=3, noise=0.2)
    eng.set_m(m)
    eng.ts_init()
    a = eng.eval_fields()
    d0 = torch.tensor(m.reshape(-1), dtype=torch.float64, device="cuda")
    d1, g1 = torch.empty_like(d0), torch.ones_like(d0)
    g0 = torch.empty_like(d0)
    torch.cuda.synchronize()
    eng.rk4_forward(d0.data_ptr(), 1e-3, 2, 1, 0, 0, 0, d1.data_ptr(), 0)
    eng.rk4_adjoint(g1.data_ptr(), 0, g0.data_ptr(), 0, 0, 0, 0)
    b = eng.eval_fields()
    assert np.isfinite(g0.cpu().numpy()).all()
    # (one state, the same factors and FP64 residuals to 1e-9 on either side)
    assert rel_err(b["H_demag"], a["H_demag"]) < 1e-6
    eng.close()
