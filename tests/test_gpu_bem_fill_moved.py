"""The boundary matrix of a turned mesh far from the origin against the oracle's
fill of the same coordinates: the 1e-12 of the largest entry that the matrix is
held to at the origin, since every term is of differences of coordinates."""
import numpy as np
import pytest

import oracle
from conftest import permalloy
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bem_precision", [0, 1])
@pytest.mark.parametrize("offset", [(0.0, -1e3, 0.0), (1e4, 0.0, -1e4), (3e5, -2e5, 1e5)])
def test_matrix_matches_oracle(offset, bem_precision):
    from nmag import mesh
    msh = mesh.box_mesh(9, 8, 5, 2.0, 2.1, 1.9)
    c, s = np.cos(0.7), np.sin(0.7)
    turn = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]]) @ np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
    pts = msh.points @ turn.T + np.asarray(offset)
    om = oracle.OracleMesh(pts, msh.simplices)
    eng = make_engine(mesh.Mesh(pts, msh.simplices), permalloy(0.5), bem_precision=bem_precision)
    B, ref = eng.bem(), om.bem
    print("largest difference %.2e of the largest entry" % (np.abs(B - ref).max() / np.abs(ref).max()))
    assert np.abs(B - ref).max() <= 1e-12 * np.abs(ref).max()
    eng.close()
