"""The rule that searches prediction batches in spatial order: which predictors and batches it takes,
the results against the oracle on both sides of its lines, and no loss against the plain search
where the rows' cells do not lie apart."""
from __future__ import annotations

import time

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import synthetic
from oracle import oracle as O
from tests.test_gpu_first_calls import searches_spatially

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def mixture(n, d, clusters, std, seed):
    """Clusters whose centres are spread over [0, 20]^d."""
    rng = np.random.default_rng(seed)
    centres = 20.0 * rng.random((clusters, d))
    return (centres[rng.integers(0, clusters, n)] + std * rng.normal(size=(n, d))).astype(np.float32)


def fitted(n, d, clusters, std, ms, m, seed=1):
    x = mixture(n + m, d, clusters, std, seed)
    x[n // 2:n // 2 + 50] = x[:50]  # ties between rows with different ids
    x[n:n + min(m, 20)] = x[:min(m, 20)]
    x[n::9] += 25.0                 # queries far from every cluster
    model = cg.HDBSCAN(min_cluster_size=200, min_samples=ms, precision="fp16_refined").fit(x[:n])
    assert model.labels_.max() >= 1
    return model, model.to_predictor(), x


@pytest.mark.parametrize("n,d,clusters,std,m,spatial", [
    (65_536, 16, 40, 1.0, 4096, True), (65_535, 16, 40, 1.0, 4096, False),  # every cell
    (65_600, 24, 40, 1.0, 2048, True), (65_600, 24, 40, 1.0, 2047, False),  # far apart: 8 of a cell
    (70_001, 13, 4, 0.4, 4096, True), (70_001, 13, 4, 0.4, 4095, False),    # apart: 16 of a cell
    (70_001, 40, 3, 4.0, 4096, False),                                      # overlapping
    (66_000, 8, 40, 0.5, 4096, False),                                      # little work
])
@pytest.mark.parametrize("ms", [5, 25])
def test_batches_on_both_sides_of_the_rule_equal_the_oracle(n, d, clusters, std, m, spatial, ms):
    model, predictor, x = fitted(n, d, clusters, std, ms, m)
    assert searches_spatially(predictor._predictor, m) == spatial
    got = predictor.approximate_predict(x[n:], True)
    exp = O.approximate_predict(model.condensed_tree_, model.labels_, np.arange(n), ms, x[:n], x[n:],
                                cores=predictor._predictor.cores())
    for a, b in zip(got, exp):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("m", [256, 512, 2048])
def test_overlapping_rows_cost_no_more_than_the_same_work_in_small_batches(m):
    # a batch in one call takes less than the same queries in pieces of 255, which are searched
    # plainly and pay a call each
    n, d = 100_000, 64
    _, predictor, x = fitted(n, d, 3, 4.0, 5, m)

    def fastest(size):
        times = []
        for _ in range(7):
            t = time.perf_counter()
            for a in range(n, n + m, size):
                predictor.approximate_predict(x[a:min(a + size, n + m)])
            times.append(time.perf_counter() - t)
        return min(times)

    fastest(m)
    assert fastest(m) < fastest(255)


def test_requests_run_at_the_first_level_whose_bound_fits():
    """Spatial search, split plain search, plain search in one part: equal results, smaller bounds."""
    from cuscan_gb300 import _lib
    from cuscan_gb300.serving import FitServer

    n, d, m = 66_000, 16, 4096
    _, predictor, x = fitted(n, d, 40, 1.0, 5, m)
    full = cg.load().cuscan_predict_workspace_bytes(predictor._predictor.handle, m)
    k = 10
    split = 4 * m * d + 8 * m * k + 8 * k * min(512 * 152 + m, m * 258) + (1 << 20)
    one_part = 4 * m * d + 8 * m * k + (1 << 20)
    results = []
    for budget, bound in ((full, full), (full - 1, split), (split, split), (split - 1, one_part),
                          (one_part, one_part), (one_part - 1, None)):
        with FitServer(slots=1, budget_bytes=budget) as srv:
            rid = srv.submit_predict(predictor, x[n:])
            info = srv.wait(rid, 60.0)
            if bound is None:
                assert info["status"] == _lib.MEMORY
                continue
            assert info["status"] == _lib.OK and info["workspace_bound_bytes"] == bound
            results.append(srv.result(rid, timeout=60.0))
    for other in results[1:]:
        for name in ("labels", "strengths", "connecting_points"):
            np.testing.assert_array_equal(other[name], results[0][name])


@pytest.mark.parametrize("slots,m,spatial", [(2, 600, True), (2, 511, False), (1, 600, False)])
def test_slots_that_share_the_device_search_smaller_batches_in_spatial_order(slots, m, spatial):
    from cuscan_gb300 import _lib
    from cuscan_gb300.serving import FitServer

    n, d = 70_000, 64
    _, predictor, x = fitted(n, d, 40, 1.0, 5, m)
    assert not searches_spatially(predictor._predictor, m)
    alone = predictor.approximate_predict(x[n:], True)
    plain = cg.load().cuscan_predict_workspace_bytes(predictor._predictor.handle, m)
    with FitServer(slots=slots, budget_bytes=8 << 30) as srv:
        rid = srv.submit_predict(predictor, x[n:])
        info = srv.wait(rid, 60.0)
        got = srv.result(rid, timeout=60.0)
    assert info["status"] == _lib.OK and (info["workspace_bound_bytes"] > plain) == spatial
    for name, value in zip(("labels", "strengths", "connecting_points"), alone):
        np.testing.assert_array_equal(got[name], value)
