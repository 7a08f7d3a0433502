"""Budgets that admitted a request before the fit's faster routes (spatial order, lists of tiles, screens
of wide rows) took memory of their own still admit it: (rows, features, min_samples, precision,
the bound then)."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib
from cuscan_gb300.serving import FitServer

BOUNDS = [
    (2048, 16, 5, "bf16_refined", 16033104),
    (5000, 128, 10, "bf16_refined", 41302504),
    (5000, 2, 32, "fp16_refined", 51611624),
    (9001, 32, 5, "bf16_refined", 57568188),
    (16384, 64, 5, "fp16_refined", 105358376),
    (20000, 200, 15, "bf16_refined", 49364220),
    (50000, 128, 5, "fp16_refined", 338616680),
    (9000, 32, 100, "bf16_refined", 81056624),
    (65536, 64, 10, "bf16_refined", 417107432),
    (100000, 64, 10, "fp32", 88107796),
    (2500, 256, 32, "bf16_refined", 27657680),
]


@pytest.mark.parametrize("n,d,k,precision,bound", BOUNDS)
def test_budgets_of_earlier_bounds_admit_the_request(n, d, k, precision, bound):
    with FitServer(slots=1, budget_bytes=bound, simulated_us_per_kpoint=0.01) as srv:
        rid = srv.submit(np.zeros((n, d), np.float32), min_cluster_size=5, min_samples=k,
                         precision=precision)
        info = srv.wait(rid, 5.0)
        assert info["status"] == _lib.OK
        assert info["workspace_bound_bytes"] <= bound
