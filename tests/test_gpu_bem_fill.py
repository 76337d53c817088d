"""The boundary matrix's fill (csrc/bem_kernels.cu) against the oracle's, bit
for bit the reference's formula: 1e-12 of the largest entry, as the other
comparisons of that matrix, with the shared series (FP64 handles) and in the
reference's operation order (handles that round the matrix).  Meshes: fewer
observers than a warp, a chunk's remainder, edges near and far on either side
of the series' bound, interior faces between boundary nodes."""
import numpy as np
import pytest

import oracle
from conftest import permalloy
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bem_precision", [0, 1])
@pytest.mark.parametrize("box,h", [((1, 1, 1), (2.0, 2.0, 2.0)), ((3, 1, 1), (2.0, 1.5, 1.0)),
                                   ((31, 1, 1), (3.0, 1.0, 0.5)), ((17, 13, 2), (2.0, 2.5, 1.5)),
                                   ((9, 8, 7), (2.0, 2.1, 1.9))])
def test_matrix_matches_oracle(box, h, bem_precision):
    from nmag import mesh
    msh = mesh.box_mesh(*box, *h)
    om = oracle.OracleMesh(msh.points, msh.simplices)
    eng = make_engine(msh, permalloy(0.5), bem_precision=bem_precision)
    B, ref = eng.bem(), om.bem
    assert np.abs(B - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.abs(B.sum(1) + 1.0).max() < 1e-9
