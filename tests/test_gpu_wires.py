"""Direct Poisson solves of long wires, magnetised along their axis: the
condition number is the square of the length in elements, so an FP64 answer's
residual does not come below 1.5e-12 (500 cells) to 2e-10 (12,000) of the
charges.  What the CG accepts, the factors answer too, or leave to it.

Tolerance: the CG's answer and the factors' each have a residual of at most
2e-10 |b|, so the fields differ by at most 2 |r| / sqrt(lambda V) with lambda =
2 (pi / 2 L)^2 the smallest eigenvalue and V = 2 a node's volume (cells of 2 x 2
x 2): 2e-6 to 3e-6 of |b| / |H| ~ 3 at 12,000 cells, hence 1e-5.  The
mixed-precision CG measures the residual itself and refuses 1e-12 on these
wires: it and the FP32 factors answer to 1e-9 (6e-6 at 3,000 cells)."""
import numpy as np
import pytest

from conftest import permalloy

pytestmark = pytest.mark.gpu


def _engine(msh, mixed, tol):
    from nmag import _lib
    c = permalloy(0.1).coefficients("nmag")
    mt = _lib.Material()
    mt.Ms, mt.exch_coeff, mt.C1, mt.C2, mt.C3 = c["Ms"], c["exch_coeff"], c["C1"], c["C2"], c["C3"]
    op = _lib.Options()
    op.do_demag, op.cg_precision = 1, int(mixed)
    op.nbc_rtol = op.dbc_rtol = tol
    op.nbc_atol = op.dbc_atol = 1e-50
    op.nbc_maxits = op.dbc_maxits = 20000
    return _lib.Engine(msh.points, msh.simplices, mt, op)


@pytest.mark.parametrize("cells,mixed", [(500, False), (500, True), (3000, False), (3000, True), (12000, False)])
def test_uniformly_magnetised(cells, mixed):
    from nmag import mesh
    msh = mesh.box_mesh(cells, 1, 1, 2.0, 2.0, 2.0)
    eng = _engine(msh, mixed, 1e-9 if mixed else 1e-12)
    m = np.zeros((msh.n_nodes, 3))
    m[:, 0] = 1.0
    eng.set_m(m)
    first = eng.eval_fields()["H_demag"].copy()
    cg = eng.cg_iterations()[0]
    assert cg > 20                      # a new handle's evaluations take the CG
    eng.ts_init()                       # integrations factor
    before = eng.cg_iterations()[0]
    H = eng.eval_fields()["H_demag"]
    passes = eng.cg_iterations()[0] - before
    print("%d cells: CG %d iterations, factors %d passes" % (cells, cg, passes))
    assert passes <= 11 or mixed        # (FP32 factors of a long wire: left to the CG)
    assert np.abs(H - first).max() <= 1e-5 * np.abs(first).max()
    eng.close()


def test_mixed_precision_near_rounding():
    """At 1e-13 the FP32 factors still answer (the setup's smooth probe, whose
    rounding lies higher, does not turn them away)."""
    from nmag import mesh
    msh = mesh.box_mesh(25, 19, 7, 2.5, 2.4, 1.9)
    eng = _engine(msh, True, 1e-13)
    eng.set_m(np.tile([1.0, 0.0, 0.0], (msh.n_nodes, 1)))
    eng.ts_init()
    before = eng.cg_iterations()
    eng.eval_fields()
    assert (np.subtract(eng.cg_iterations(), before) <= 11).all()
    eng.close()


def test_mixed_precision_refuses_a_tolerance_below_rounding():
    """As the mixed-precision CG does, before and after the factors."""
    from nmag import _lib, mesh
    eng = _engine(mesh.box_mesh(25, 19, 7, 2.5, 2.4, 1.9), True, 1e-17)
    eng.set_m(np.tile([1.0, 0.0, 0.0], (26 * 20 * 8, 1)))
    with pytest.raises(_lib.NmagGpuError):
        eng.eval_fields()
    with pytest.raises(_lib.NmagGpuError):
        eng.ts_init()
    eng.close()
