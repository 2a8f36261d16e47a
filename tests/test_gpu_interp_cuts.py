"""FP64 interpolation with up to 128 points to a CTA and several problems
sharing it (k_nufft_interp_mma with eight units of 16 points, windows double
buffered over the CTA's problems): 60 spots of 200 points each in a tile of its
own, an odd number of problems.  Bits as for each problem alone, whose CTAs have
32 or 64 points and one problem; the tap-by-tap kernels to 1e-10 after three
steps (operators agree to 1e-12)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [45, 63])
def test_full_ctas_of_several_problems(gpulib, monkeypatch, b):
    rng = np.random.default_rng(b)
    nx = 100
    a, c = np.meshgrid(16 * np.arange(-5, 5) + 13.0, 16 * np.arange(-3, 3) + 13.0)
    at = np.stack([a.ravel(), c.ravel()], 1)[:, None] + rng.uniform(0, 12, (60, 200, 2))
    first = np.round(at).astype(int) - 11
    tiles = np.unique(first.reshape(-1, 2) // 16, axis=0, return_counts=True)[1]
    assert len(tiles) == 60 and tiles.min() == 200  # two CTAs of 128 and 72 points each
    assert 4 * len(tiles) * b >= 8000               # enough of them for CTAs of 128 points
    u, v = (np.pi * at.reshape(-1, 2) / nx).T.copy()
    data = (u, v, rng.standard_normal(u.size), rng.standard_normal(u.size), np.full(u.size, 2.0))
    probs = [dict(lambda_l1=0.02 * (k + 1), lambda_tsv=0.01, cinit=1e8, maxiter=3, nonneg_flag=0) for k in range(b)]
    run = lambda p: gpulib.nufft_batch(*data, nx, nx, p, 0.0)[0]
    x = run(probs)
    for k in (0, b // 2, b - 1):
        assert np.linalg.norm(x[k]) > 0
        np.testing.assert_array_equal(run([probs[k]])[0], x[k])
    monkeypatch.setenv("MFISTA_INTERP_TC", "0")
    monkeypatch.setenv("MFISTA_SPREAD_TC", "0")
    y = run(probs)
    for k in range(b):
        assert rel(x[k], y[k]) < 1e-10
