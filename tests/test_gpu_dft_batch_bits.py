"""A DFT problem's products have the same bits in any batch: more problems than
a tile of 64 change neither the split of K nor its order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, n", [(100, 256), (3002, 1024), (2000, 4096), (64, 900), (9001, 400)])
def test_products_do_not_depend_on_the_batch(gpulib, m, n):
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, n))
    X, R = rng.standard_normal((130, n)), rng.standard_normal((130, m))
    for b in (2, 64, 65):
        at = rng.choice(130, b, replace=False)
        np.testing.assert_array_equal(gpulib.dft_apply(A, X)[at], gpulib.dft_apply(A, X[at]))
        np.testing.assert_array_equal(gpulib.dft_apply(A, R, transpose=True)[at],
                                      gpulib.dft_apply(A, R[at], transpose=True))
