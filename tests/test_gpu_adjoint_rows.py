"""The adjoint's matrix kernels in both forms (rows by four lanes up to 8,192
nodes, a row per thread above), and the transposed BEM product's partial sums
down to one slab: against central differences along seeded directions, at the
1e-5 and h = 1e-6 that the cube's gradient is held to."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import permalloy, seeded_m  # noqa: E402
from test_gpu_adjoint import _params, _run  # noqa: E402
from test_gpu_parity import make_engine  # noqa: E402

pytestmark = pytest.mark.gpu


# boundary nodes: 12 (one slab), 60, and 2,322 of 8,820
@pytest.mark.parametrize("box", [(2, 1, 1), (4, 3, 2), (20, 20, 19)])
def test_gradient_matches_finite_differences(box):
    from nmag import mesh
    msh = mesh.box_mesh(*box, 2.0, 2.1, 1.9)
    mat = permalloy(0.5)
    eng = make_engine(msh, mat, tol=1e-12)
    c = mat.coefficients("nmag")
    N, T = len(msh.points), len(msh.simplices)
    m0 = seeded_m(N, seed=0, noise=0.2)
    Ms_T, K1_T, pulses = _params(T, 3)
    eng.set_h_ext(np.zeros(3))
    args = (6, 4, 2)
    _, _, g_Ms, g_K1, g_P, _ = _run(eng, c, m0, Ms_T, K1_T, pulses, *args)
    rng, h = np.random.default_rng(11), 1e-6
    for _ in range(2):
        dM, dK = Ms_T * rng.standard_normal(T), 0.05 * rng.standard_normal(T)
        dP = np.abs(pulses).mean() * rng.standard_normal(pulses.shape)
        lp, lm = (_run(eng, c, m0, Ms_T + q * dM, K1_T + q * dK, pulses + q * dP, *args, grad=False)[0]
                  for q in (h, -h))
        ad = g_Ms @ dM + g_K1 @ dK + (g_P * dP).sum()
        assert abs((lp - lm) / (2 * h) - ad) <= 1e-5 * max(abs(ad), 1e-30)
    eng.close()
