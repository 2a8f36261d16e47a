"""The FGP prox over the shapes its kernels divide differently: images smaller
than a cluster, slabs whose last CTAs are short or empty, one and two rows a
thread, rows wider than a CTA's threads (the kernel with all arrays in shared
memory or in global memory); against the oracle (FP64: 1e-12, the contract of
the operators; FP32: 2e-5).  A problem's solve has the same bits alone and in
a batch that takes another kernel."""
import numpy as np
import pytest

from conftest import rel
from oracle import mfista_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", [(2, 2), (3, 40), (5, 200), (33, 97), (64, 17), (64, 64), (100, 100), (128, 128),
                                    (256, 33), (500, 40), (1000, 3), (1200, 20), (700, 300)])
@pytest.mark.parametrize("nonneg", [0, 1])
def test_prox_matches_oracle(gpulib, nx, ny, nonneg):
    rng = np.random.default_rng(nx + ny)
    b = 3 * rng.standard_normal(nx * ny)
    box = (rng.random(nx * ny) < 0.9).astype(np.float32) if nx % 2 else None
    iters = 7 if nx * ny > 50000 else 25
    want = O.fgp(nx, ny, b, 0.0 if nonneg else 0.2, 0.7, iters, nonneg, box)
    assert rel(gpulib.fgp_prox(b, nx, ny, 0.2, 0.7, iters, nonneg, cl_box=box), want) < 1e-12
    assert rel(gpulib.fgp_prox(b, nx, ny, 0.2, 0.7, iters, nonneg, cl_box=box, precision=gpulib.FP32), want) < 2e-5


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_size_leaves_bits(gpulib, precision):
    prec = gpulib.FP64 if precision == "fp64" else gpulib.FP32
    n = 48
    rng = np.random.default_rng(3)
    a, b = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    F = np.fft.fft2(np.maximum(rng.standard_normal((n, n)), 0)).ravel()
    data = (a.ravel(), b.ravel(), F.real.copy(), F.imag.copy(), np.full(n * n, 3.0), n, n)
    probs = [dict(lambda_l1=0.01, lambda_tv=0.02 * (k + 1), cinit=1.0, maxiter=6, nonneg_flag=1) for k in range(150)]
    X, _ = gpulib.fft_batch(*data, probs, 0.0, precision=prec, fgp_iter=12)
    for k in (0, 77, 149):
        x, _ = gpulib.fft_batch(*data, [probs[k]], 0.0, precision=prec, fgp_iter=12)
        assert np.linalg.norm(x) > 0 and np.array_equal(x[0], X[k])
