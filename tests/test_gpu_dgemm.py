"""The FP64 matrix products of the DFT operator and of the leave-one-out error
(dgemm_mma.cuh) at the edges of their tiles: one row more or less than a tile
of 64, odd leading dimensions (8-byte copies), column blocks of 1, 2, 4 and 8,
more than 64 problems, K ranges that end inside a step of 16; against numpy.
The products are FP64 sums of at most 1031 terms of size 1: 1e-13 relative."""
import numpy as np
import pytest

from conftest import rel
from oracle import looe_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, n, b", [(63, 65, 2), (64, 64, 8), (65, 129, 9), (130, 17, 17), (257, 1031, 33),
                                     (1030, 66, 64), (201, 200, 65), (2, 15, 130)])
def test_products_match_numpy(gpulib, m, n, b):
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, n))
    X, R = rng.standard_normal((b, n)), rng.standard_normal((b, m))
    assert rel(gpulib.dft_apply(A, X), X @ A.T) < 1e-13
    assert rel(gpulib.dft_apply(A, R, transpose=True), R @ A) < 1e-13


@pytest.mark.parametrize("m, ns", [(301, 1), (300, 64), (301, 65), (1001, 128), (1000, 129), (2049, 333)])
def test_looe_tile_edges_match_oracle(gpulib, m, ns):
    """Panels of one column, full and one more; odd and even M."""
    rng = np.random.default_rng(ns)
    nx = 24
    A = rng.normal(size=(m, nx * nx)) / np.sqrt(m)
    x = np.zeros(nx * nx)
    x[rng.choice(nx * nx, ns, replace=False)] = 1 + rng.random(ns)
    y = A @ x + 0.01 * rng.normal(size=m)
    mean, std, pos = gpulib.dft_looe(y, A, x[None], nx, lambda_tsv=[0.3])
    st, wm, ws = O.looe(y, A, x, nx, 0.3)
    assert st == 1 and pos[0]
    assert abs(mean[0] - wm) <= 1e-9 * abs(wm) and abs(std[0] - ws) <= 1e-9 * abs(ws)


@pytest.mark.parametrize("b", [1, 2, 9])
def test_looe_of_a_batch_is_that_of_its_solutions(gpulib, b):
    """More solutions than streams, each with its own support (columns of A in
    runs with gaps of 1 to 5, the first and the last one; one solution empty,
    one not positive definite between good ones): same bits as alone."""
    rng = np.random.default_rng(b)
    nx, m = 16, 400
    n = nx * nx
    A = rng.normal(size=(m, n)) / np.sqrt(m)
    A[:, 7] = 0.0  # a column of zeros: singular without lambda_tsv
    X = np.zeros((b, n))
    for k in range(b):
        at = np.cumsum(rng.integers(1, 7, size=n // 4))
        X[k, at[at < n]] = 1 + rng.random((at < n).sum())
        X[k, 7] = 1.0 if k == 3 else 0.0
    X[0, [0, n - 1]] = 2.0
    if b > 4:
        X[4] = 0.0
    y = A @ X[0] + 0.01 * rng.normal(size=m)
    lam = np.where(np.arange(b) == 3, 0.0, 0.1 * (1 + np.arange(b)))
    mean, std, pos = gpulib.dft_looe(y, A, X, nx, lambda_tsv=lam)
    for k in range(b):
        one = gpulib.dft_looe(y, A, X[k:k + 1], nx, lambda_tsv=lam[k:k + 1])
        assert (mean[k], std[k], pos[k]) == (one[0][0], one[1][0], one[2][0])
        assert pos[k] == (k != 3)
        if k not in (3, 4):
            _, wm, ws = O.looe(y, A, X[k], nx, lam[k])
            assert abs(mean[k] - wm) <= 1e-9 * abs(wm) and abs(std[k] - ws) <= 1e-9 * abs(ws)
