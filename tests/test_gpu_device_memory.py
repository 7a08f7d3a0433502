"""Device memory that calls hold: what a call takes is kept in the context's workspace, counted and
given back with it."""
from __future__ import annotations

from contextlib import contextmanager

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_first_calls import searches_spatially
from tests.test_gpu_fit import assert_fit_equal
from tests.test_gpu_ops import bits

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@contextmanager
def little_memory(left):
    """All but about `left` bytes of the device taken."""
    torch.cuda.empty_cache()
    filler = torch.empty(free_bytes() - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def test_repeated_packs_with_wide_lists_hold_no_more_memory():
    ctx = _lib.Context(0)
    fits = [(synthetic.gaussian_mixture(n, 32, 5, seed=n), k, _lib.PRECISION_PLAIN)
            for n, k in ((2000, 50), (2047, 100), (700, 33), (900, 5))]
    ctx.fit_core_packed(fits)
    free, reserved = free_bytes(), ctx.reserved_bytes()
    for _ in range(50):
        ctx.fit_core_packed(fits)
    assert free_bytes() == free
    assert ctx.reserved_bytes() == reserved


def test_packs_count_every_launch_of_wide_lists():
    ctx = _lib.Context(0)
    fits = [(synthetic.gaussian_mixture(n, 32, 5, seed=n), 50, _lib.PRECISION_PLAIN)
            for n in (2000, 900)]
    ctx.fit_core_packed(fits)
    before = _lib.launch_count()
    ctx.fit_core_packed(fits)
    assert _lib.launch_count() - before == ctx.packed_launch_stats()["launches"]


@pytest.mark.parametrize("squared", [True, False])
def test_exact_knn_of_wide_lists_runs_without_room_for_partial_lists(squared):
    m, n, d, k = 3000, 60_000, 16, 200
    x = synthetic.gaussian_mixture(m + n, d, 9, seed=1)
    q, r = torch.from_numpy(x[:m]).cuda(), torch.from_numpy(x[m:]).cuda()
    ids = torch.empty((m, k), dtype=torch.int32, device="cuda")
    ds = torch.empty((m, k), dtype=torch.float32, device="cuda")

    def run(ctx):
        ids.fill_(-1)
        torch.cuda.synchronize()
        ctx.exact_knn(q.data_ptr(), m, r.data_ptr(), n, d, k, False, 0, squared, ids.data_ptr(),
                      ds.data_ptr())
        torch.cuda.synchronize()
        return ids.cpu().numpy(), ds.cpu().numpy()

    left = 24 << 20
    ctx = _lib.Context(0)
    ids0, ds0 = run(ctx)
    assert ctx.reserved_bytes() > left  # the lists of the parts
    ctx.close()
    with little_memory(left):
        ids1, ds1 = run(_lib.Context(0))
    np.testing.assert_array_equal(ids1, ids0)
    np.testing.assert_array_equal(bits(ds1), bits(ds0))


def test_plain_fits_with_wide_lists_run_without_room_for_partial_lists():
    x = synthetic.gaussian_mixture(5003, 64, 9, seed=2)
    left = 32 << 20
    warm = _lib.Context(0)
    warm.fit_core(x, 250, _lib.PRECISION_PLAIN)
    assert warm.reserved_bytes() > left
    warm.close()
    ctx = _lib.Context(0)
    with little_memory(left):
        got = ctx.fit_core(x, 250, _lib.PRECISION_PLAIN)
    assert_fit_equal(got, O.fit_core(x, 250))


def spatial_model(n, d, m):
    x = synthetic.gaussian_mixture(n + m, d, 10, seed=5)
    x[n // 2:n // 2 + 50] = x[:50]  # ties between rows with different ids
    x[n:n + min(m, 20)] = x[:min(m, 20)]
    return cg.HDBSCAN(min_cluster_size=50, min_samples=5, precision="fp16_refined").fit(x[:n]), x


def test_predictors_leave_no_workspace_and_copy_their_rows_only_with_ample_room():
    n, d, m = 100_000, 64, 4096
    model, x = spatial_model(n, d, m)
    arrays, meta = model.to_predictor()._predictor.export_state()
    np.testing.assert_array_equal(arrays["geometry"].reshape(n, d), x[:n])
    rows = 4 * n * d
    results = []
    for left, copies in ((None, 2), (6 * rows, 1)):
        # on a context that has run nothing, whose workspace stays empty
        ctx = _lib.Context(0)

        def restore():
            free = free_bytes()
            predictor = cg.prediction.Predictor.from_state(arrays, meta, ctx)
            # (ids, bounds and up to 2 MiB of rounding per allocation beside the rows)
            assert copies * rows <= free - free_bytes() < (copies + 0.5) * rows
            assert searches_spatially(predictor, m) == (copies == 2)
            assert ctx.reserved_bytes() == 0
            results.append(predictor.predict(x[n:]))

        if left is None:
            restore()
        else:
            with little_memory(left):
                restore()
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)




@pytest.mark.parametrize("n,d,k,precision,left", [
    # in spatial order 400 MB; the plain sweeps take 113 MB in blocks of 2 MiB. (With 300 to 320 MiB
    # the order, the balls and the partial lists fit, but not the rounds' arrays beside them.)
    (600_000, 2, 5, _lib.PRECISION_PLAIN, 200 << 20), (600_000, 2, 5, _lib.PRECISION_PLAIN, 310 << 20),
    (600_000, 2, 5, _lib.PRECISION_PLAIN, 320 << 20),
    # screens of wide rows 155 MB, the exact sweeps 40 MB
    (20_000, 200, 15, _lib.PRECISION_BF16_REFINED, 60 << 20),
])
def test_fits_run_where_only_the_plain_sweeps_fit(n, d, k, precision, left):
    x = synthetic.gaussian_mixture(n, d, 30, seed=7)
    warm = _lib.Context(0)
    full = warm.fit_core(x, k, precision)
    assert warm.reserved_bytes() > left
    warm.close()
    ctx = _lib.Context(0)
    with little_memory(left):
        got = ctx.fit_core(x, k, precision)
    for key in ("knn_ids", "src", "dst"):
        np.testing.assert_array_equal(got[key], full[key])
    for key in ("knn_sq", "core_sq", "wsq"):
        np.testing.assert_array_equal(bits(got[key]), bits(full[key]))
