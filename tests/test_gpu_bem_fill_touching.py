"""Two parts that touch with unlike cells, so that nodes of the one lie on edges
of the other: the reference's formula is not a number there, and the matrix says
so in the same entries (a finite value would be taken for one).  The others:
1e-12 of the largest entry, as the other comparisons of that matrix."""
import numpy as np
import pytest

import oracle
from conftest import permalloy
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


def _touching():
    from nmag import mesh
    a = mesh.box_mesh(2, 2, 2, 2.0)
    b = mesh.box_mesh(4, 4, 3, 1.0, origin=(0.0, 0.0, 4.0))
    return mesh.Mesh(np.concatenate([a.points, b.points]), np.concatenate([a.simplices, b.simplices + a.n_nodes]))


@pytest.mark.parametrize("bem_precision", [0, 1])
def test_entries_that_are_not_numbers(bem_precision):
    msh = _touching()
    om = oracle.OracleMesh(msh.points, msh.simplices)
    eng = make_engine(msh, permalloy(0.5), bem_precision=bem_precision)
    B, ref = eng.bem(), om.bem
    assert 0 < np.isnan(ref).sum() < ref.size / 10
    assert np.array_equal(np.isfinite(B), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert np.abs(B - ref)[ok].max() <= 1e-12 * np.abs(ref[ok]).max()
    eng.close()
