"""The tensor-core product's sum over its splits of 1,024 boundary nodes.  A
vector that is zero outside one split's nodes gives that split's FP32 sum as it
is, so the sum over the splits can be checked by itself: no further from the
exact sum of these than FP64 additions, (splits - 1) 2^-53 of their sizes.  The
splits' vectors are of falling sizes, so that the sums need all of FP64's bits."""
import math

import numpy as np
import pytest

from conftest import permalloy
from test_gpu_bem_tc import _apply
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(20, 20, 20), (50, 50, 50)])   # 2,402 and 15,002 nodes: 3 and 15 splits
def test_sum_over_splits(box):
    from nmag import mesh
    eng = make_engine(mesh.box_mesh(*box, 2.0, 2.1, 1.9), permalloy(0.5), bem_precision=3)
    nb = eng.nb
    splits = -(-nb // 1024)
    rng = np.random.default_rng(4)
    X = rng.standard_normal((3, nb)) * 10.0 ** rng.uniform(-3, 3, size=(3, nb))
    X *= 0.6 ** np.arange(3)[:, None] * 2.0 ** (-(3 + 3 * np.arange(3)[:, None]) * (np.arange(nb) // 1024))
    Y = _apply(eng, X)
    parts = np.zeros((splits, 3, nb))
    for k in range(splits):
        Z = np.zeros_like(X)
        Z[:, 1024 * k:1024 * (k + 1)] = X[:, 1024 * k:1024 * (k + 1)]
        parts[k] = _apply(eng, Z)
    eng.close()
    assert np.array_equal(parts, parts.astype(np.float32))
    worst = 0.0
    for n in range(3):
        for r in range(nb):
            p = parts[:, n, r]
            worst = max(worst, abs(math.fsum(list(p) + [-Y[n, r]])) / np.abs(p).sum())
    print("%d splits: %.2f x 2^-53 of the terms" % (splits, worst * 2.0 ** 53))
    assert worst <= (splits - 1) * 2.0 ** -53
