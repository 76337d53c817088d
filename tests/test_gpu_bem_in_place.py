"""nmg_bem_apply where the answers overwrite the vectors, on boundaries of
several waves of blocks (2,402 to 4,706 nodes: below the line where a product
of one vector has a block per row) and above it (4,898): the same numbers as
from vectors and answers apart, which are compared with the matrix.  Each
vector's product is the same sums in either case but for the single ones, whose
sums are of the same terms in another order: 2 n eps |B||x| with n columns."""
import numpy as np
import pytest

from conftest import permalloy
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module", params=[(20, 20, 20), (26, 26, 26), (28, 28, 28), (32, 24, 30)])
def engine(request):
    from nmag import mesh
    eng = make_engine(mesh.box_mesh(*request.param, 2.0, 2.1, 1.9), permalloy(0.5))
    yield eng
    eng.close()


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (9, 0), (11, 0), (1, 5), (4, 1), (5, -1), (3, 700)])
def test_overlapping(engine, n, shift):
    """shift: the answers' distance from the vectors, in values (1 to 5: within
    a vector; a vector's answer then lies on part of the next vector, which is
    read after it was written, as one product after the other does)."""
    import torch
    nb, pad = engine.nb, 1000
    B = engine.bem()
    buf = np.random.default_rng(n).standard_normal(n * nb + 2 * pad)
    d = torch.tensor(buf, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    x0 = d.data_ptr() + 8 * pad
    engine.bem_apply_device(x0, x0 + 8 * shift, n)
    got = d.cpu().numpy()
    ref = buf.copy()
    tol = np.zeros_like(buf)
    absB = np.abs(B)
    for k in range(n):
        x, e = ref[pad + k * nb:pad + (k + 1) * nb].copy(), tol[pad + k * nb:pad + (k + 1) * nb].copy()
        o = slice(pad + shift + k * nb, pad + shift + (k + 1) * nb)
        ref[o] = B @ x
        tol[o] = absB @ (e + 2 * nb * EPS * np.abs(x))
    assert (np.abs(got - ref) <= tol).all()
