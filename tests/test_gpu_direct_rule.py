"""When a handle gets the direct Poisson solver's factors: once its CG solves are
worth 3/4 of what the factors cost (both estimated from iteration counts and
the mesh, nd_solve.cu), at once where an integration or enough RK4 steps are
certain.  The fields are the same on either side: 1e-9 of the oracle's, the
bound of the other field comparisons at a Poisson tolerance of 1e-12."""
import numpy as np
import pytest

from conftest import permalloy, seeded_m
from test_gpu_direct_solver import BOXES, _mesh, _oracle_fields
from test_gpu_parity import make_engine, rel_err

pytestmark = pytest.mark.gpu
PASSES = 11   # a direct solve takes no more; the CG on these meshes takes more


def _worth(eng, msh):
    """The two sides of the rule: seconds of a CG iteration, and 3/4 of the factors'."""
    N, inner = msh.n_nodes, msh.n_nodes - eng.nb
    cost = 1e-3 + 2.5e-6 * min(N, 2000) + 2e-6 * (N - 0.95 * eng.nb) + 1e-11 * inner ** 2
    return 8e-6 + 2.6e-8 * N ** 0.5, 0.75 * cost


@pytest.mark.parametrize("tol", [1e-5, 1e-12])
@pytest.mark.parametrize("box", [(10, 10, 10), (40, 30, 2)])
def test_evaluations_alone(box, tol):
    from nmag import mesh
    msh = mesh.box_mesh(*box, 2.0, 2.1, 1.9)
    eng = make_engine(msh, permalloy(0.1), tol=tol)
    iteration, limit = _worth(eng, msh)
    counts = [0]
    for k in range(60):
        eng.set_m(seeded_m(msh.n_nodes, seed=k, noise=0.5))
        eng.eval_fields()
        counts.append(sum(eng.cg_iterations()))
        if counts[-1] - counts[-2] <= 2 * PASSES and eng.cg_iterations()[0]:
            break
    first = len(counts) - 2                        # evaluations before the one that had the factors
    assert 3 <= first < 59
    assert counts[first] * iteration >= limit
    assert first == 3 or counts[first - 1] * iteration < limit
    eng.close()


def _passes(eng):
    before = np.array(eng.cg_iterations())
    eng.eval_fields()
    return np.array(eng.cg_iterations()) - before


def test_integrations_and_rk4(cube):
    import torch
    m = seeded_m(len(cube.points), seed=1, noise=0.5)
    eng = make_engine(cube, permalloy(0.1))
    eng.set_m(m)
    assert (_passes(eng) > PASSES).all()
    eng.ts_init()
    assert (_passes(eng) <= PASSES).all()
    eng.close()
    eng = make_engine(cube, permalloy(0.1))
    d = torch.tensor(m.reshape(-1), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    eng.set_m(m)
    eng.rk4_device(d.data_ptr(), 1e-3, 1)           # four evaluations are not worth them here
    assert eng.cg_iterations()[0] > 4 * PASSES
    eng.rk4_device(d.data_ptr(), 1e-3, 20)
    assert (_passes(eng) <= PASSES).all()
    eng.close()


@pytest.mark.parametrize("name", list(BOXES) + ["pinched"])
def test_factors_at_once(name):
    msh, mat = _mesh(name), permalloy(0.1)
    m = seeded_m(msh.n_nodes, seed=0, noise=0.5)
    (d, hd), = _oracle_fields(msh, mat, [m])
    eng = make_engine(msh, mat, tol=1e-12)
    eng.set_m(m)
    eng.ts_init()
    before = np.array(eng.cg_iterations())
    f = eng.eval_fields()
    assert (np.array(eng.cg_iterations()) - before <= PASSES).all()
    assert rel_err(f["dmdt"], d) < 1e-9
    assert rel_err(f["H_demag"], hd.reshape(-1, 3)) < 1e-9
    eng.close()
