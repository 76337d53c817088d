"""The direct Poisson solver where its other tests do not go: meshes that are
neither structured, nor aligned with the axes, nor at the origin; several
materials; two handles used by two threads.  Fields against the oracles at the
1e-9 of the other field comparisons (Poisson tolerance 1e-12)."""
import threading

import numpy as np
import pytest

from conftest import permalloy, seeded_m
from test_gpu_direct_solver import _oracle_fields
from test_gpu_parity import make_engine, rel_err

pytestmark = pytest.mark.gpu


def _direct(eng, m):
    """Fields of m from direct solves."""
    eng.set_m(m)
    eng.ts_init()
    before = np.array(eng.cg_iterations())
    f = eng.eval_fields()
    assert (np.array(eng.cg_iterations()) - before <= 11).all()
    return f


def _turned(box, seed, offset):
    """A box whose nodes are displaced by up to a fifth of a cell, turned by 40 degrees about two axes, moved."""
    from nmag import mesh
    b = mesh.box_mesh(*box, 2.0, 2.1, 1.9)
    p = b.points + 0.38 * np.random.default_rng(seed).uniform(-1, 1, b.points.shape)
    c, s = np.cos(0.7), np.sin(0.7)
    turn = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]]) @ np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
    return mesh.Mesh(p @ turn.T + np.asarray(offset), b.simplices)


@pytest.mark.parametrize("box,offset", [((12, 11, 9), (0.0, 0.0, 0.0)), ((40, 21, 2), (300.0, -200.0, 100.0)),
                                        ((18, 15, 14), (-1000.0, 0.0, 50.0))])
def test_unstructured_meshes(box, offset):
    msh, mat = _turned(box, 3, offset), permalloy(0.1)
    m = seeded_m(msh.n_nodes, seed=0, noise=0.5)
    (d, hd), = _oracle_fields(msh, mat, [m])
    eng = make_engine(msh, mat, tol=1e-12)
    f = _direct(eng, m)
    assert rel_err(f["dmdt"], d) < 1e-9
    assert rel_err(f["H_demag"], hd.reshape(-1, 3)) < 1e-9
    eng.close()


def test_several_materials():
    from multimat import MultiOracle
    from nmag import _lib
    from nmag.sites import SiteLayer
    from test_gpu_multimat import engine, halves, materials
    msh, (py, co) = halves(), materials()
    eng = engine(msh, [[0], [1]], [py, co])
    L = SiteLayer(msh, [["Py"], ["Co"]])
    mo = MultiOracle(msh.points, msh.simplices, L, {"Py": py.coefficients("nmag"), "Co": co.coefficients("nmag")})
    h = np.array([0.02, -0.01, 0.03])
    mo.set_h_ext(h)
    eng.set_h_ext(h)
    m = seeded_m(L.n_sites, base=(0.3, 1.0, -0.2), seed=71, noise=0.4)
    d = mo.rhs(m)
    for _ in range(2):                # before and after the factors
        eng.set_m(m)
        f = eng.eval_fields()
        assert rel_err(f["H_demag"], mo.fields["H_demag"][L.site_node]) < 1e-9
        assert rel_err(f["phi"], mo.fields["phi"][L.site_node]) < 1e-9
        assert rel_err(f["dmdt"], d) < 1e-9
        eng.ts_init()
    eng.close()


def test_two_handles_on_two_threads(cube):
    meshes = [cube, _turned((14, 9, 8), 5, (0.0, 0.0, 0.0))]
    states = [[seeded_m(len(q.points), seed=s, noise=0.5) for s in range(12)] for q in meshes]
    engines = [make_engine(q, permalloy(0.1)) for q in meshes]
    for e, ms in zip(engines, states):
        _direct(e, ms[0])

    def run(e, ms, out):
        for m in ms:
            e.set_m(m)
            f = e.eval_fields()
            out.append((f["H_demag"].copy(), f["dmdt"].copy()))

    alone = [[], []]
    for k in range(2):
        run(engines[k], states[k], alone[k])
    both = [[], []]
    threads = [threading.Thread(target=run, args=(engines[k], states[k], both[k])) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(both[k]) == len(alone[k])
        for a, b in zip(alone[k], both[k]):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        engines[k].close()
