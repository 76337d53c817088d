"""The tensor-core product when a CTA walks several tiles (accumulators in turn,
the load ring running on), for each tile width, ragged counts and a split K,
and with values that are not finite.  Tolerance: the 2e-6 of max |B||x| that
the six-term split with FP32 sums of a thousand terms is held to."""
import numpy as np
import pytest

from conftest import permalloy
from test_gpu_bem_tc import TOL_PRODUCT, _apply, _check
from test_gpu_parity import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [4095, 4097, 8961])   # 5 x R / 128 tiles of one split: 1 to 3 per CTA
def test_many_vectors(cube, R):
    eng = make_engine(cube, permalloy(0.5), bem_precision=3)
    X = np.random.default_rng(R).standard_normal((R, eng.nb))
    assert _check(eng.bem(), X, _apply(eng, X)) <= TOL_PRODUCT
    eng.close()


def test_tile_widths_on_the_film_give_the_same_bits():
    """3,465 tiles per 32, 64 or 128 vectors: 23 per CTA, 21 splits.  Every
    output is the same sums in the same order, whatever the tile width; the
    narrowest form's products of this mesh are compared with FP64 elsewhere."""
    from nmag import mesh
    eng = make_engine(mesh.film_mesh(), permalloy(0.02), bem_precision=3)
    X = np.random.default_rng(3).standard_normal((129, eng.nb))
    Y = np.concatenate([_apply(eng, X[n:n + 8]) for n in range(0, 129, 8)])
    for R in (17, 33, 64, 128, 129):
        assert np.array_equal(_apply(eng, X[:R]), Y[:R]), R
    eng.close()


def test_not_finite(cube):
    eng = make_engine(cube, permalloy(0.5), bem_precision=3)
    X = np.random.default_rng(1).standard_normal((40, eng.nb))
    bad = X.copy()
    bad[7, 11], bad[20, 3] = np.inf, np.nan
    Y, Z = _apply(eng, X), _apply(eng, bad)
    assert not np.isfinite(Z[[7, 20]]).any()
    rest = np.delete(np.arange(40), [7, 20])
    assert np.array_equal(Z[rest], Y[rest])
    eng.close()
