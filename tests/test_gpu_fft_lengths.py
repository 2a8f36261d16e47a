"""The FFT passes at lengths that reach every radix and every arrangement of
their stages: powers of two from one to three stages, lengths without a radix
that reads or writes global memory directly, the primes 7, 11 and 13, a single
stage; against numpy's transforms through the operators that use them.
Contract of the operators: 1e-12 relative in FP64, 2e-5 in FP32."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

LENGTHS = [12, 13, 14, 16, 18, 22, 26, 27, 32, 36, 49, 54, 64, 66, 78, 90, 96, 98, 100, 121, 128, 144, 169, 192, 200, 256]


@pytest.mark.parametrize("nx", LENGTHS)
def test_nufft_passes(gpulib, nx):
    """At the centre of the uv plane the operators reduce to sums the exact
    Fourier sum gives; rows of length nx, columns of length 2 nx."""
    rng = np.random.default_rng(nx)
    m = 40
    lim = np.pi * max(1, nx - 13) / nx  # within the gridding's range
    u, v = rng.uniform(-lim, lim, m), rng.uniform(-lim, lim, m)
    x = rng.standard_normal((nx, nx))
    k = np.arange(nx) - nx // 2
    ex, ey = np.exp(1j * np.outer(u, k)), np.exp(1j * np.outer(v, k))
    want = np.einsum("ki,ij,kj->k", ex, x, ey)
    fr, fi = gpulib.nufft_forward(u, v, nx, nx, x.ravel())
    gr, gi = gpulib.nufft_forward(u, v, nx, nx, x.ravel(), precision=gpulib.FP32)
    r = rng.standard_normal(m) + 1j * rng.standard_normal(m)
    back = gpulib.nufft_adjoint(u, v, nx, nx, r.real, r.imag)
    # adjointness holds to rounding whatever the gridding's own error (1e-11)
    lhs, rhs = float(np.sum(fr * r.real + fi * r.imag)), float(x.ravel() @ back)
    assert abs(lhs - rhs) <= 1e-12 * np.linalg.norm(fr + 1j * fi) * np.linalg.norm(r)
    assert rel(gr + 1j * gi, fr + 1j * fi) < 2e-5
    if nx % 2 == 0:  # the reference centres odd images half a pixel off
        assert rel(fr + 1j * fi, want) < 1e-9


@pytest.mark.parametrize("nx, ny", [(2, 2), (3, 4), (5, 6), (7, 10), (16, 16), (22, 26), (27, 54), (64, 32), (100, 96),
                                    (128, 128), (169, 338), (256, 512)])
def test_gridded_passes(gpulib, nx, ny):
    """One step from zero with step size 1 / cinit: the image is the threshold
    of the gradient, the inverse transform of the data."""
    rng = np.random.default_rng(nx * ny)
    a, b = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    F = np.fft.fft2(rng.standard_normal((nx, ny)))
    noise = np.full(nx * ny, 2.0)
    probs = [dict(lambda_l1=0.0, cinit=100.0, maxiter=1, nonneg_flag=0)]
    y = F.ravel()
    x, r = gpulib.fft_batch(a.ravel(), b.ravel(), y.real.copy(), y.imag.copy(), noise, nx, ny, probs, 0.0)
    grad = np.fft.ifft2(F / 4).real * np.sqrt(nx * ny) / 2  # mask y / noise, c2r, 1 / (2 sqrt N)
    assert rel(x[0].reshape(nx, ny), grad / 100.0) < 1e-12
    res = F / 2 - np.fft.fft2(grad / 100.0) / np.sqrt(nx * ny) / 2
    chi2 = 0.5 * np.sum(np.abs(res) ** 2)
    assert abs(r[0]["sq_error"] - chi2) <= 1e-12 * chi2
