"""Fields posted through pinned memory (up to 2^20 values) and copied (more):
the same evaluation on either side of the line, and in one evaluation alone.
Poisson tolerance 1e-12 on 60 and 245 nodes (condition ~1e2): 1e-9 of the largest value."""
import numpy as np
import pytest

from conftest import permalloy, seeded_m
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 251, 252])   # 17 x 245 x B values: 1,045,415 and 1,049,580 at the line
def test_fields_posted_and_copied(small_box, B):
    from nmag import mesh
    from test_gpu_ensemble import make_ensemble
    small_box = small_box if B < 3 else mesh.box_mesh(6, 6, 4, 2.0, 2.5, 1.5)
    mat, N = permalloy(0.5), len(small_box.points)
    states = [seeded_m(N, base=(1.0, 0.2 * b, -0.3), seed=b, noise=0.3) for b in range(3)]
    ms = np.stack([states[b % 3] for b in range(B)])
    ens, _ = make_ensemble(small_box, mat, B)
    one = make_engine(small_box, mat)
    ens.set_h_ext(np.zeros(3))
    one.set_h_ext(np.zeros(3))
    ens.set_m(ms if B > 1 else ms[0])
    f = ens.eval_fields()
    for b in sorted({0, min(1, B - 1), B - 1}):
        one.set_m(ms[b])
        g = one.eval_fields()
        for key in g:
            x = f[key][b] if B > 1 else f[key]
            assert np.abs(x - g[key]).max() <= 1e-9 * max(np.abs(g[key]).max(), 1.0), (key, b)
        a, e = ens.member_averages(b, energies=True)
        a1, e1 = one.averages(energies=True)
        assert np.allclose(a, a1, rtol=0, atol=1e-12) and np.allclose(e, e1, rtol=1e-9, atol=1e-9 * np.abs(e1).max())
    ens.close()
    one.close()
