"""The integrator's fused Newton and Gram-Schmidt kernels: Krylov spaces of one
vector up to more than the 32 that one launch takes, against the oracle's BDF
(same family, own steps).  m(t) at rtol = atol = 1e-6
agrees to the 1e-4 that the trajectories are held to."""
import numpy as np
import pytest

import oracle
from conftest import permalloy, seeded_m
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


def _run(msh, m0, krylov_max, t_end, level=0, mat=None, tol=1e-6):
    eng = make_engine(msh, mat or permalloy(0.5))
    eng.set_jacobian(level)
    eng.set_h_ext(np.zeros(3))
    eng.set_m(m0)
    eng.ts_init(rtol=tol, atol=tol, max_order=2, krylov_max=krylov_max)
    most, seen, t = 0.0, (0, 0), 0.0
    while t < t_end:
        t, st = eng.ts_advance(t_end, max_steps=1)
        dn, dl = st["nni"] - seen[0], st["nli"] - seen[1]
        seen = (st["nni"], st["nli"])
        most = max(most, dl / max(dn, 1))
    m = eng.get_m()
    eng.close()
    return m, most, st


@pytest.mark.parametrize("krylov_max", [1, 2, 3, 33, 300])
def test_krylov_limits(small_box, krylov_max):
    m0 = seeded_m(len(small_box.points), base=(1.0, 0.5, 0.2), seed=2, noise=0.3)
    m, _, _ = _run(small_box, m0, krylov_max, 20.0)
    mat = permalloy(0.5)
    s = oracle.OracleSim(oracle.OracleMesh(small_box.points, small_box.simplices), mat.coefficients("nmag"),
                         nbc=(1e-12, 1e-50, 20000), dbc=(1e-12, 1e-50, 20000))
    s.set_h_ext(np.zeros(3))
    s.ts_init(m0, rtol=1e-6, atol=1e-6, max_order=2, krylov_max=300)
    _, ref = s.ts_advance(20.0)
    assert np.abs(m.reshape(-1, 3) - np.asarray(ref).reshape(-1, 3)).max() <= 1e-4


def test_more_than_32_vectors():
    """A long bar's domain wall at a loose tolerance: long steps, and an exchange
    over 400 cells that the block preconditioner does not see.  Vectors that lost
    their orthogonality past the 32nd would leave the solves at the limit, and
    Newton's iterations failing: one failure in a thousand steps is usual."""
    import nmag
    from nmag import SI, mesh
    mat = nmag.MagMaterial("A", Ms=SI(8.6e5, "A/m"), exchange_coupling=SI(1.3e-10, "J/m"), llg_damping=1.0)
    bar = mesh.box_mesh(400, 1, 1, 1.0, 1.0, 1.0)
    th = bar.points[:, 0] / 400.0 * 0.9 * np.pi
    m0 = np.stack([np.cos(th), np.sin(th), 0.05 + 0.0 * th], axis=1)
    m0 /= np.linalg.norm(m0, axis=1)[:, None]
    m, most, st = _run(bar, m0, 300, 1500.0, 1, mat, 1e-3)
    print("most Krylov vectors in a solve: %g, failures %d in %d steps" % (most, st["ncfn"], st["nst"]))
    assert 32 < most < 200
    assert st["ncfn"] <= 0.05 * st["nst"]
    assert np.abs(np.linalg.norm(m.reshape(-1, 3), axis=1) - 1.0).max() <= 0.05
