"""Requests whose full workspace bound exceeds a server's budget, but which fit in less device memory,
are admitted and give the same results."""
from __future__ import annotations

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import _lib, synthetic
from cuscan_gb300.serving import FitServer


def bound(n, d, min_samples, precision):
    return cg.load().cuscan_fit_workspace_bytes(n, d, min_samples, precision)


# (n, d): plain fits in spatial order, screens of wide rows, tile lists
CASES = [(10_007, 101, _lib.PRECISION_PLAIN, "fp32"),
         (3001, 200, _lib.PRECISION_BF16_REFINED, "bf16_refined"),
         (16_500, 40, _lib.PRECISION_FP16_REFINED, "fp16_refined")]


@pytest.mark.parametrize("n,d,code,name", CASES)
def test_admitted_below_the_full_bound(n, d, code, name):
    with FitServer(slots=1, budget_bytes=bound(n, d, 5, code) - 1, simulated_us_per_kpoint=1.0) as srv:
        rid = srv.submit(np.zeros((n, d), np.float32), min_cluster_size=5, min_samples=5,
                         precision=name)
        info = srv.wait(rid, 5.0)
        assert info["status"] == _lib.OK
        assert info["workspace_bound_bytes"] < bound(n, d, 5, code)


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,code,name", CASES)
def test_lean_fits_equal_full_ones(n, d, code, name):
    x = synthetic.gaussian_mixture(n, d, 9, seed=n)
    results = []
    for budget in (bound(n, d, 5, code) - 1, 4 * bound(n, d, 5, code)):
        with FitServer(slots=1, budget_bytes=budget) as srv:
            results.append(srv.result(srv.submit(x, min_cluster_size=20, min_samples=5,
                                                 precision=name), timeout=60.0))
    lean, full = results
    np.testing.assert_array_equal(lean["labels"], full["labels"])
    np.testing.assert_array_equal(lean["probabilities"], full["probabilities"])


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,k", [(2048, 8, 5), (10_007, 101, 33), (16_500, 40, 10), (20_011, 32, 50),
                                   (9001, 200, 15)])
@pytest.mark.parametrize("code", [_lib.PRECISION_PLAIN, _lib.PRECISION_BF16_REFINED])
def test_the_bound_holds_for_every_route(n, d, k, code):
    ctx = cg.Context(0)
    ctx.fit_core(synthetic.gaussian_mixture(n, d, 9, seed=n), k, code)
    assert cg.load().cuscan_ctx_reserved_bytes(ctx.handle) <= bound(n, d, k, code)


@pytest.mark.gpu
def test_lean_predictions_equal_full_ones():
    n, d, m = 20_000, 64, 2001
    x = synthetic.gaussian_mixture(n + m, d, 10, seed=3)
    model = cg.HDBSCAN(min_cluster_size=50, min_samples=5, precision="fp16_refined").fit(x[:n])
    predictor = model.to_predictor()
    full = cg.load().cuscan_predict_workspace_bytes(predictor._predictor.handle, m)
    results = []
    for budget in (full - 1, 4 * full):
        with FitServer(slots=1, budget_bytes=budget) as srv:
            results.append(srv.result(srv.submit_predict(predictor, x[n:]), timeout=60.0))
    lean, full = results
    for name in ("labels", "strengths", "connecting_points"):
        np.testing.assert_array_equal(lean[name], full[name])
