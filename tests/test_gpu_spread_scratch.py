"""Spreading on the FP64 matrix instruction with more points than its scratch
has partial tiles: lists cut into longer segments, staged in several rounds.
The operators agree with the tap-by-tap kernels to 1e-12 (the contract of the
operators), a problem has the same bits alone and in a batch, and the plan's
memory is what its points and grids need."""
import os

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _points(m, nx):
    rng = np.random.default_rng(m)
    lim = np.pi * (nx - 13) / nx
    return rng.uniform(-lim, lim, m), rng.uniform(-lim, lim, m), rng


@pytest.mark.parametrize("m, nx", [(400000, 64), (120000, 20)])
def test_long_lists_match_tap_by_tap(gpulib, monkeypatch, m, nx):
    u, v, rng = _points(m, nx)
    a, b = rng.standard_normal(m), rng.standard_normal(m)
    got = gpulib.nufft_adjoint(u, v, nx, nx, a, b)
    monkeypatch.setenv("MFISTA_SPREAD_TC", "0")
    assert rel(got, gpulib.nufft_adjoint(u, v, nx, nx, a, b)) < 1e-12


def test_memory_and_bits_of_a_batch(gpulib, monkeypatch):
    """Beyond what the tap-by-tap spreading holds: list entries (4 bytes, about
    11 a point) and 8 MB of scratch a problem."""
    import torch
    m, nx, B = 400000, 64, 16
    u, v, rng = _points(m, nx)
    data = (u, v, rng.standard_normal(m), rng.standard_normal(m), np.full(m, 2.0))
    probs = [dict(lambda_l1=0.1 * (k + 1), lambda_tsv=0.01, cinit=1e9, maxiter=2, nonneg_flag=0) for k in range(B)]

    def make():
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        plan = gpulib.Plan(*data, nx, nx, B)
        return plan, before - torch.cuda.mem_get_info()[0]

    make()[0].close()  # the library's own start
    with monkeypatch.context() as mp:
        mp.setenv("MFISTA_SPREAD_TC", "0")
        plan, taps = make()
        plan.close()
    plan, used = make()
    assert used - taps < 48 * m + 8.5e6 * B
    plan.set_problems(probs, 0.0)
    plan.run()
    X, _ = plan.fetch()
    plan.close()
    for k in (0, B - 1):
        alone = gpulib.nufft_batch(*data, nx, nx, [probs[k]], 0.0)[0]
        assert np.linalg.norm(X[k]) > 0
        np.testing.assert_array_equal(alone[0], X[k])
