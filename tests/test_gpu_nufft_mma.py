"""Interpolation and spreading on the FP64 matrix instruction
(k_nufft_interp_mma, k_nufft_spread_mma) against the tap-by-tap kernels.

Both sum the same products in FP64 in another order, so the operators agree
as the operators of this library must with the oracle (1e-12 relative L2).
The geometries reach the edges of the kernels: windows cut by the Nyquist
rows and columns, points whose taps are dropped or mirrored, columns that are
direct and mirrored in one window, tiles of one point, of 8, 9, 16, 17 and of
more points than a CTA takes, lists longer than a segment, grids whose sides
are no multiple of a tile; frames of uneven size, one of a single point."""
import os

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _taps(fn):
    """fn() with the tap-by-tap kernels."""
    old = {n: os.environ.get(n) for n in ("MFISTA_INTERP_TC", "MFISTA_SPREAD_TC")}
    os.environ.update({n: "0" for n in old})
    try:
        return fn()
    finally:
        for n, v in old.items():
            if v is None:
                del os.environ[n]
            else:
                os.environ[n] = v


def _points(name):
    """(u, v, nx) in radians per pixel; grid position = u nx / pi."""
    rng = np.random.default_rng(len(name))
    at = lambda k, nx: np.pi * np.asarray(k, float) / nx
    if name == "one":
        return at([3.3], 12), at([-2.2], 12), 12
    if name == "edges":
        nx = 32
        e = np.array([31, 31.4, -31.9, -32, 0, 0.4, -0.4, 20, 21, -12, 11, 12])
        a, b = np.meshgrid(e, e)
        return at(a.ravel(), nx), at(b.ravel(), nx), nx
    if name == "fold":
        return at(rng.uniform(-40, 40, 300), 54), at(rng.uniform(-1, 1, 300), 54), 54
    if name == "dense":
        n = [1, 8, 9, 16, 17, 130, 700]  # points at one spot each
        u = np.concatenate([rng.uniform(6 * i, 6 * i + 0.9, m) for i, m in enumerate(n)])
        v = np.concatenate([rng.uniform(-9 * i, -9 * i + 0.9, m) for i, m in enumerate(n)])
        return at(u, 100), at(v, 100), 100
    return at(rng.uniform(-190, 190, 5001), 250), at(rng.uniform(-190, 190, 5001), 250), 250


@pytest.mark.parametrize("name", ["one", "edges", "fold", "dense", "uniform"])
def test_operators_match_tap_by_tap(gpulib, name):
    u, v, nx = _points(name)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(nx * nx)
    a, b = rng.standard_normal(u.size), rng.standard_normal(u.size)
    fwd = lambda: np.array(gpulib.nufft_forward(u, v, nx, nx, x))
    adj = lambda: gpulib.nufft_adjoint(u, v, nx, nx, a, b)
    assert rel(fwd(), _taps(fwd)) < TOL
    assert rel(adj(), _taps(adj)) < TOL


@pytest.mark.parametrize("b", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("shared", [True, False])
def test_batches_match_tap_by_tap(gpulib, shared, b):
    """Chunks of 1, 2, 4 and 8 problems per CTA, and frames with their own points."""
    u, v, nx = _points("dense")
    rng = np.random.default_rng(2)
    data = (u, v, rng.standard_normal(u.size), rng.standard_normal(u.size), np.full(u.size, 2.0))
    off = None if shared else np.concatenate([[0, 1], np.linspace(40, u.size, b)])[:b + 1].astype(np.int32)
    probs = [dict(lambda_l1=0.02 * (k + 1), lambda_tsv=0.01, cinit=1e7, maxiter=4, nonneg_flag=0) for k in range(b)]
    run = lambda: gpulib.nufft_batch(*data, nx, nx, probs, 0.0, pt_off=off)[0]
    x, y = run(), _taps(run)
    assert np.linalg.norm(x) > 0
    assert rel(x, y) < 1e-10  # four steps of operators that agree to 1e-12


@pytest.mark.parametrize("name,b", [("dense", 24), ("uniform", 20)])
def test_cut_of_points_keeps_bits(gpulib, name, b):
    """One problem alone (32 or 64 points per interpolation CTA) and in a batch
    large enough for the next size (64 or 128) and several chunks: same bits."""
    u, v, nx = _points(name)
    rng = np.random.default_rng(3)
    data = (u, v, rng.standard_normal(u.size), rng.standard_normal(u.size), np.full(u.size, 2.0))
    probs = [dict(lambda_l1=0.02 * (k + 1), lambda_tsv=0.01, cinit=1e7, maxiter=3, nonneg_flag=0) for k in range(b)]
    x = gpulib.nufft_batch(*data, nx, nx, probs, 0.0)[0]
    for k in (0, b - 1):
        alone = gpulib.nufft_batch(*data, nx, nx, [probs[k]], 0.0)[0]
        assert np.linalg.norm(x[k]) > 0
        np.testing.assert_array_equal(alone[0], x[k])
