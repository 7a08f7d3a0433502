"""Exact neighbours of rows with many equal distances (duplicates, overflow): the oracle's rows, and
no more time than rows without ties need, but for a factor that covers the first tiles of every list."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib
from oracle import oracle as O
from tests.test_gpu_fit import assert_fit_equal
from tests.test_gpu_ops import bits, gpu_knn

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def tied_rows(kind, n, d):
    rng = np.random.default_rng(n + d)
    if kind == "equal":
        return np.repeat(rng.normal(size=(1, d)), n, 0).astype(np.float32)
    if kind == "overflow":  # every squared distance is infinite
        return (1e25 * rng.normal(size=(n, d))).astype(np.float32)
    if kind == "binary":
        return rng.integers(0, 2, size=(n, d)).astype(np.float32)
    x = np.repeat(rng.normal(size=(1, d)), n, 0)  # ties at a distance above zero
    x[::2] += 1.0
    return x.astype(np.float32)


@pytest.mark.parametrize("kind", ["equal", "overflow", "binary", "two_places"])
@pytest.mark.parametrize("n,d,k", [(129, 3, 1), (700, 9, 8), (1500, 16, 33), (1999, 5, 100)])
@pytest.mark.parametrize("exclude_self,squared", [(True, True), (False, False)])
def test_tied_neighbours_equal_the_oracle(gpu_ctx, kind, n, d, k, exclude_self, squared):
    x = tied_rows(kind, n, d)
    ids, ds = gpu_knn(gpu_ctx, x, x.copy(), k, exclude_self, 0, squared)
    eids, eds = O.exact_neighbors(x, x, k, exclude_self=exclude_self, squared=squared)
    np.testing.assert_array_equal(ids, eids)
    np.testing.assert_array_equal(bits(ds), bits(eds))


@pytest.mark.parametrize("kind", ["equal", "two_places"])
def test_tied_plain_fits_in_spatial_order_equal_the_oracle(gpu_ctx, kind):
    x = tied_rows(kind, 7001, 210)  # n^2 d >= 1e10
    assert_fit_equal(gpu_ctx.fit_core(x, 6, _lib.PRECISION_PLAIN), O.fit_core(x, 6))


@pytest.mark.parametrize("kind", ["equal", "overflow"])
@pytest.mark.parametrize("k", [8, 60])
@pytest.mark.parametrize("squared", [True, False])
def test_ties_cost_no_list_insertions(gpu_ctx, kind, k, squared):
    n, d = 10_000, 16
    ids = torch.empty((n, k), dtype=torch.int32, device="cuda")
    ds = torch.empty((n, k), dtype=torch.float32, device="cuda")
    legacy_stream = 1  # the events' stream

    def fastest(rows):
        q = torch.from_numpy(rows).cuda()
        r = q.clone()
        times = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            gpu_ctx.exact_knn(q.data_ptr(), n, r.data_ptr(), n, d, k, False, 0, squared,
                              ids.data_ptr(), ds.data_ptr(), legacy_stream)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    plain = fastest(np.random.default_rng(1).normal(size=(n, d)).astype(np.float32))
    assert fastest(tied_rows(kind, n, d)) < 4 * plain
