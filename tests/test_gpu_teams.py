"""Particles shared by a cluster of CTAs (csrc/batch.cu, team_cg) against the
same particles run by one CTA each, and against the oracle.

A particle belongs to a team when it costs more than an even share of the
batch on the SMs, so a particle alone does and one of 160 copies does not; the
team adds up every sum in the single CTA's order, so the two give the same
bits (states, times and step counts of adaptive steps).  Sizes: the smallest a
team takes (512 nodes), one past a block of rows, a remainder, a plate without
interior nodes."""
import numpy as np
import pytest

from conftest import seeded_m
from test_gpu_batch import _oracle_rhs

pytestmark = pytest.mark.gpu

BOXES = [(7, 7, 7), (8, 7, 7), (11, 10, 9), (24, 24, 1)]


def _particle(box):
    import nmag
    from nmag import SI, mesh
    msh = mesh.box_mesh(*box, 2.0, 2.1, 1.9)
    mat = nmag.MagMaterial("p", Ms=SI(9e5, "A/m"), exchange_coupling=SI(1.3e-11, "J/m"), llg_damping=0.1,
                           llg_gamma_G=SI(2.211e5, "m/A s"),
                           anisotropy=nmag.uniaxial_anisotropy(axis=[0.6, 0.0, 0.8], K1=SI(2e5, "J/m^3")))
    return msh, (msh.points, msh.simplices, mat.coefficients("nmag"), np.array([0.0, 0.6, 0.8]))


@pytest.mark.parametrize("box", BOXES)
def test_team_equals_one_block_bit_for_bit(box):
    from nmag.batch import ParticleBatch
    msh, part = _particle(box)
    m = seeded_m(msh.n_nodes, base=(0.2, 1.0, 0.3), seed=7, noise=0.2)
    got = []
    for copies in (1, 160):
        b = ParticleBatch([part] * copies, n_stages=3, h_max=0.3, rtol=1e-7, atol=1e-7, cg_rtol=1e-10)
        b.set_m([m] * copies)
        f, H = b.eval()
        b.run(3)
        st = b.state()
        got.append((f[0], H[0], b.get_m()[0], st["t"][0], st["steps"][0], st["rhs"][0], st["max_dmdt"][0]))
        b.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    assert got[0][4] > 0


def test_teams_and_single_blocks_against_the_oracle():
    from nmag.batch import ParticleBatch
    parts = [_particle(b) for b in ((3, 3, 3), (11, 10, 9), (2, 3, 4), (9, 9, 8))]
    b = ParticleBatch([p for _, p in parts], n_stages=5, h_max=0.3, cg_rtol=1e-12)
    ms = [seeded_m(m.n_nodes, base=(1.0, 0.5, -0.3), seed=40 + k, noise=0.4) for k, (m, _) in enumerate(parts)]
    b.set_m(ms)
    f, _ = b.eval()
    for (msh, p), m, g in zip(parts, ms, f):
        _, ref = _oracle_rhs(msh, p[2], 0.3 * p[3] / np.linalg.norm(p[3]), m)
        assert np.abs(g - ref).max() <= 1e-5 * np.abs(ref).max()   # FP32 BEM blocks, as test_gpu_batch
    b.close()
