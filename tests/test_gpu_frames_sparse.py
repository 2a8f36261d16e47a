"""Problems with points of their own and few of them to a tile, against the
tap-by-tap kernels.  Spots of 1 to 150 points, points at the edges of the grid
(dropped and mirrored taps), frames of one point; few frames, and enough of
them that interpolation takes the smaller CTAs of many tiles, of two and of
four warps (and cuts a frame of 2000 points in one place into more).  Operators
agree to 1e-12, so four steps agree to 1e-10; the FP32 form to its 2e-5.  A
frame has the same bits alone and among others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(nx, more):
    rng = np.random.default_rng(nx)
    e = np.array([nx - 1, nx - 0.6, 0.1 - nx, -nx, 0, 0.4, -0.4, nx - 12, 13 - nx, -12, 11, 12])
    a, b = np.meshgrid(e, e)
    spots = [(rng.uniform(-nx / 2, nx / 2 - 1, 2), k) for k in (1, 7, 8, 9, 17, 150)]
    spot = np.concatenate([c + rng.uniform(0, 0.4, (k, 2)) for c, k in spots])
    lim = nx - 13
    parts = [np.stack([a.ravel(), b.ravel()], 1), spot, rng.uniform(-lim, lim, (1, 2)), rng.uniform(-lim, lim, (333, 2)),
             np.concatenate([spot, rng.uniform(-lim, lim, (90, 2))]), rng.uniform(-3, 3, (2000, 2))]
    parts += [rng.uniform(-lim, lim, (40, 2)) for _ in range(more)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.int32)
    at = np.pi * np.concatenate(parts) / nx
    vis = rng.standard_normal((2, len(at)))
    return (at[:, 0].copy(), at[:, 1].copy(), vis[0], vis[1], np.full(len(at), 2.0)), off


@pytest.mark.parametrize("nx, more", [(16, 0), (54, 0), (128, 0), (54, 40), (128, 30), (20, 170)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sparse_frames(gpulib, monkeypatch, nx, more, precision):
    prec = gpulib.FP64 if precision == "fp64" else gpulib.FP32
    data, off = _frames(nx, more)
    B = len(off) - 1
    probs = [dict(lambda_l1=0.02 * (k + 1), lambda_tsv=0.01, cinit=1e7, maxiter=4, nonneg_flag=0) for k in range(B)]
    run = lambda d, o, p: gpulib.nufft_batch(*d, nx, nx, p, 0.0, pt_off=o, precision=prec)[0]
    x = run(data, off, probs)
    for k in range(min(B, 8)):
        s = slice(off[k], off[k + 1])
        alone = run(tuple(d[s] for d in data), np.array([0, off[k + 1] - off[k]], np.int32), [probs[k]])
        assert np.linalg.norm(x[k]) > 0
        np.testing.assert_array_equal(alone[0], x[k])
    monkeypatch.setenv("MFISTA_INTERP_TC", "0")
    monkeypatch.setenv("MFISTA_SPREAD_TC", "0")
    y = run(data, off, probs)
    for k in range(B):
        assert np.linalg.norm(x[k] - y[k]) <= (1e-10 if precision == "fp64" else 2e-5) * np.linalg.norm(y[k])
