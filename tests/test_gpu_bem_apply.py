"""nmg_bem_apply for several vectors: passes of up to eight over the matrix in
the FP64 and the compensated form, against the matrix itself in numpy FP64.

Counts on either side of the passes' sizes.  FP64: sums of n terms in another
order, n eps |B||x| bounds their difference (n = 602: 1.4e-13); compensated:
2^-44 per term on top, 602 x 5.7e-14 = 3.5e-11 of max |B||x|; FP32 and split
BF16 (one product per vector, unchanged): 1e-5."""
import numpy as np
import pytest

from conftest import permalloy
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu
BOUND = {0: 1.4e-13, 1: 1e-5, 2: 3.5e-11, 3: 1e-5}


@pytest.fixture(scope="module")
def engines(cube):
    return {f: make_engine(cube, permalloy(0.5), bem_precision=f) for f in BOUND}


@pytest.mark.parametrize("form", list(BOUND))
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 13, 16, 21])
def test_products_of_several_vectors(engines, form, n):
    import torch
    eng = engines[form]
    B = engines[0].bem()
    x = 100.0 * np.random.default_rng(n).standard_normal((n, eng.nb))
    dx = torch.tensor(x, dtype=torch.float64, device="cuda")
    dy = torch.full((n + 1, eng.nb), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    eng.bem_apply_device(dx.data_ptr(), dy.data_ptr(), n)
    y = dy.cpu().numpy()
    scale = (np.abs(B) @ np.abs(x).T).max()
    assert np.abs(y[:n] - x @ B.T).max() <= BOUND[form] * scale
    assert (y[n] == 7.0).all()   # nothing past the last vector


def test_in_place(engines):
    import torch
    for form in (0, 2):
        eng = engines[form]
        x = np.random.default_rng(1).standard_normal((11, eng.nb))
        d = torch.tensor(x, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        eng.bem_apply_device(d.data_ptr(), d.data_ptr(), 11)
        B = engines[0].bem()
        assert np.abs(d.cpu().numpy() - x @ B.T).max() <= BOUND[form] * (np.abs(B) @ np.abs(x).T).max()
