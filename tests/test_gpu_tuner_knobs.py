"""The autotuner and the launch shapes by the kernels that a plan runs: with
the matrix-product kernels the interpolation and spreading shapes decide
nothing and stay as they were set; the tap-by-tap kernels (selected by the
environment) regroup their sums with them, which moves results by rounding
only (the bounds of test_gpu_tuner.py)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _plan(si, c0, B=4, precision=None):
    lam1 = float(c0["lam1"])
    plan = si.Plan(c0["u"], c0["v"], c0["vis_r"], c0["vis_i"], c0["vis_std"], 64, 64, B,
                   precision=si.FP64 if precision is None else precision)
    return plan, [dict(lambda_l1=lam1 * s, lambda_tsv=lam1 * 1e-3 * s, cinit=float(c0["cinit"]), maxiter=150,
                       nonneg_flag=1) for s in np.geomspace(0.2, 5.0, B)]


def _solve(plan, probs):
    plan.set_problems(probs, 1e-5)
    plan.run()
    return plan.fetch()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_tuner_leaves_shapes_without_effect(gpulib, c0, precision):
    plan, probs = _plan(gpulib, c0, precision=gpulib.FP64 if precision == "fp64" else gpulib.FP32)
    plan.set_problems(probs, 1e-5)
    for ppw, cl in [(4, 2), (2, 16), (16, 1)]:
        plan.set_shapes(interp_ppw=ppw, spread_cluster=cl)
        shapes, ms = plan.tune(reps=2)
        assert (shapes["interp_ppw"], shapes["spread_cluster"]) == (ppw, cl)
        assert all(v > 0 for v in ms.values())
    plan.close()


def test_tap_kernel_shapes_move_results_by_rounding_only(gpulib, c0, monkeypatch):
    monkeypatch.setenv("MFISTA_INTERP_TC", "0")
    monkeypatch.setenv("MFISTA_SPREAD_TC", "0")
    plan, probs = _plan(gpulib, c0)
    X0, R0 = _solve(plan, probs)
    moved = 0
    for ppw, cl in [(1, 1), (4, 2), (16, 4)]:
        plan.set_shapes(interp_ppw=ppw, spread_cluster=cl)
        X, R = _solve(plan, probs)
        moved += not np.array_equal(X, X0)
        for b in range(len(R)):
            assert R[b]["ITER"] == R0[b]["ITER"]
            assert rel(X[b], X0[b]) < 1e-10
            assert abs(R[b]["finalcost"] - R0[b]["finalcost"]) <= 1e-12 * R0[b]["finalcost"]
    assert moved  # the shapes reach the kernels
    plan.close()
