"""The leave-one-out error with many active pixels: more of them than a launch
has rows of CTAs, and a Hessian held once.

With fewer visibilities than pixels, H = A^T A + lambda D (D the curvature of
the TSV term) and the leverages follow from an M x M system alone
(Woodbury): with G = A D^-1 A^T / lambda, A H^-1 A^T = (I + G)^-1 G."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nx, active, m, seed):
    rng = np.random.default_rng(seed)
    n = nx * nx
    A = rng.normal(size=(m, n)) / np.sqrt(m)
    x = np.zeros(n)
    S = np.sort(rng.choice(n, active, replace=False))
    x[S] = 1 + rng.random(active)
    return A, x, S, A @ x + rng.normal(size=m)


def _expected(A, x, S, y, nx, lam):
    inner = lambda k: (k > 0) & (k < nx - 1)
    D = lam * (4.0 + 2 * inner(S % nx) + 2 * inner(S // nx))
    G = (A[:, S] / D) @ A[:, S].T
    d = np.diag(np.linalg.solve(np.eye(len(y)) + G, G))
    s = 0.5 * ((y - A @ x) / (1 - d)) ** 2
    return s.mean(), s.std(ddof=1)


@pytest.mark.parametrize("nx, active", [(257, 65537)])
def test_more_active_pixels_than_grid_rows(gpulib, nx, active):
    """The sums of the factorisation are of FP64 terms of size 1 at most, the
    matrix is lambda D plus a matrix of rank m: 1e-9, as the other sizes."""
    A, x, S, y = _case(nx, active, 16, 1)
    mean, std, pos = gpulib.dft_looe(y, A, x[None], nx, lambda_tsv=[2.0])
    wm, ws = _expected(A, x, S, y, nx, 2.0)
    assert pos[0]
    assert abs(mean[0] - wm) <= 1e-9 * wm and abs(std[0] - ws) <= 1e-9 * ws


def test_hessian_is_held_once(gpulib):
    """8281 active pixels, 0.55 GB of Hessian (its product is not split at this
    size): a call's largest device memory, read while it runs."""
    import torch
    nx = 91
    A, x, S, y = _case(nx, nx * nx, 6, 2)
    call = lambda: gpulib.dft_looe(y, A, x[None], nx, lambda_tsv=[2.0])
    mean, std, pos = call()
    wm, ws = _expected(A, x, S, y, nx, 2.0)
    assert pos[0] and abs(mean[0] - wm) <= 1e-9 * wm and abs(std[0] - ws) <= 1e-9 * ws
    torch.cuda.synchronize()
    before, least, done = torch.cuda.mem_get_info()[0], [], threading.Event()

    def watch():
        while not done.is_set():
            least.append(torch.cuda.mem_get_info()[0])

    w = threading.Thread(target=watch)
    w.start()
    for _ in range(3):
        call()
    done.set()
    w.join()
    hessian = 8 * len(S) ** 2
    used = before - min(least)
    assert hessian <= used < 1.5 * hessian
