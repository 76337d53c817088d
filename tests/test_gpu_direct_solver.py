"""The direct Poisson solver (csrc/nd_solve.cu) against the oracle's fields.

A handle's first evaluations use the CG, later ones the factors; both answer
to the same tolerance (1e-12), so the fields of one state agree with the
oracle's (Poisson solves at 1e-13) to 1e-9 relative, the bound of the other
field comparisons.  Meshes: one front (few nodes, one block), several tree
levels, no interior node, an interior that falls into parts, a bar; ensembles
of 1, 2, 3 and 8 members in FP64 and with FP32 factors; a mesh of two parts,
whose Neumann system stays with the CG."""
import numpy as np
import pytest

import oracle
from conftest import permalloy, seeded_m
from test_gpu_parity import make_engine, rel_err

pytestmark = pytest.mark.gpu

BOXES = {"one_front": (4, 3, 2), "one_cell": (1, 1, 1), "no_interior": (23, 17, 1), "bar": (61, 2, 2),
         "levels": (25, 19, 7), "plate": (60, 33, 2)}


def _mesh(name):
    from nmag import mesh
    if name == "pinched":   # two blocks that share an edge: the interior nodes fall into two parts
        a, b = mesh.box_mesh(4, 4, 4, 2.0), mesh.box_mesh(4, 4, 4, 2.0, origin=(8.0, 8.0, 0.0))
        pts = np.concatenate([a.points, b.points])
        uniq, inv = np.unique(np.round(pts, 6), axis=0, return_inverse=True)
        sim = np.concatenate([a.simplices, b.simplices + a.n_nodes])
        return mesh.Mesh(uniq, inv.reshape(-1)[sim].astype(np.int32))
    if name == "two_parts":
        a, b = mesh.box_mesh(4, 3, 3, 2.0), mesh.box_mesh(4, 3, 3, 2.0, origin=(20.0, 0.0, 0.0))
        return mesh.Mesh(np.concatenate([a.points, b.points]), np.concatenate([a.simplices, b.simplices + a.n_nodes]))
    return mesh.box_mesh(*BOXES[name], 2.5, 2.4, 1.9)


def _oracle_fields(msh, mat, states):
    om = oracle.OracleMesh(msh.points, msh.simplices)
    out = []
    for m in states:
        s = oracle.OracleSim(om, mat.coefficients("nmag"), nbc=(1e-13, 1e-50, 50000), dbc=(1e-13, 1e-50, 50000))
        d = s.rhs(m).reshape(-1, 3)
        out.append((d, s.field("H_demag").copy()))
    return out


@pytest.mark.parametrize("name", list(BOXES) + ["pinched", "two_parts"])
def test_fields_before_and_after_the_factors(name):
    msh, mat = _mesh(name), permalloy(0.1)
    states = [seeded_m(msh.n_nodes, seed=s, noise=0.5) for s in range(2)]
    ref = _oracle_fields(msh, mat, states)
    eng = make_engine(msh, mat, tol=1e-12)
    for k in range(8):
        eng.set_m(states[k % 2])
        f = eng.eval_fields()
        d, hd = ref[k % 2]
        assert rel_err(f["dmdt"], d) < 1e-9
        assert rel_err(f["H_demag"], hd.reshape(-1, 3)) < 1e-9


@pytest.mark.parametrize("members,mixed", [(1, True), (2, False), (3, True), (8, False), (8, True), (9, True)])
def test_members(members, mixed):
    from nmag import _lib
    msh, mat = _mesh("levels"), permalloy(0.1)
    states = [seeded_m(msh.n_nodes, seed=s, noise=0.5) for s in range(members)]
    ref = _oracle_fields(msh, mat, states[:3] + states[-1:])
    c = mat.coefficients("nmag")
    mt = _lib.Material()
    mt.Ms, mt.exch_coeff, mt.C1, mt.C2, mt.C3 = c["Ms"], c["exch_coeff"], c["C1"], c["C2"], c["C3"]
    op = _lib.Options()
    op.do_demag, op.n_members, op.cg_precision = 1, members if members > 1 else 0, int(mixed)
    op.nbc_rtol = op.dbc_rtol = 1e-12
    op.nbc_atol = op.dbc_atol = 1e-50
    op.nbc_maxits = op.dbc_maxits = 20000
    eng = _lib.Engine(msh.points, msh.simplices, mt, op)
    eng.set_m(np.stack(states) if members > 1 else states[0])
    for _ in range(5):
        f = eng.eval_fields()
    for k, (d, hd) in zip([0, 1, 2, members - 1][:len(ref)] if members > 2 else range(members), ref):
        got = f["dmdt"][k] if members > 1 else f["dmdt"]
        assert rel_err(got, d) < 1e-9


def test_tolerance_below_rounding():
    """The FP64 CG's recurrence meets any tolerance; so does a factor's answer once its residual is rounding."""
    msh, mat = _mesh("levels"), permalloy(0.1)
    m = seeded_m(msh.n_nodes, noise=0.5)
    (d, _), = _oracle_fields(msh, mat, [m])
    eng = make_engine(msh, mat, tol=1e-17)
    eng.set_m(m)
    for _ in range(5):
        f = eng.eval_fields()
    assert rel_err(f["dmdt"], d) < 1e-9
