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
