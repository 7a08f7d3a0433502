"""Rows that are not finite at the device entry points, which do not look at them: where rows are
ordered by cells, such rows stay inside the order, the other rows' neighbours are unchanged, and a
fit ends in the error that it ends in without the order."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic
from tests.test_gpu_first_calls import self_knn
from tests.test_gpu_ops import bits, gpu_knn

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def with_bad_rows(n, d, seed):
    x = synthetic.gaussian_mixture(n, d, 9, seed=seed)
    x[[0, n // 2, n - 1], 0] = np.nan  # the first row is a pivot
    x[n // 3:n // 3 + 40, d - 1] = np.nan
    return x


def device_fit(ctx, x, min_samples, precision):
    n, d = x.shape
    data = torch.from_numpy(x).cuda()
    out = [torch.empty(s, dtype=t, device="cuda") for s, t in (
        ((n, min_samples), torch.int32), ((n, min_samples), torch.float32), (n, torch.float32),
        (n - 1, torch.int32), (n - 1, torch.int32), (n - 1, torch.float32))]
    torch.cuda.synchronize()
    ctx.fit_core_device(data.data_ptr(), n, d, min_samples, precision, *[t.data_ptr() for t in out])


# (2100 rows: fewer cells than rows' worth of 256 pivots; from 65,536 rows all 256; the plain ones
# past n^2 d = 1e10 in spatial order)
@pytest.mark.parametrize("n,d", [(1500, 8), (2100, 16), (9001, 128), (65_537, 3), (70_000, 9)])
@pytest.mark.parametrize("precision", [_lib.PRECISION_PLAIN, _lib.PRECISION_BF16_REFINED])
@pytest.mark.parametrize("min_samples", [1, 5])
def test_fits_of_rows_that_are_not_numbers_end_in_the_same_error(gpu_ctx, n, d, precision,
                                                                 min_samples):
    with pytest.raises(ValueError, match="candidate index is out of range"):
        device_fit(gpu_ctx, with_bad_rows(n, d, n), min_samples, precision)
    device_fit(gpu_ctx, synthetic.gaussian_mixture(n, d, 9, seed=n), min_samples, precision)


@pytest.mark.parametrize("n,d,k", [(2100, 16, 5), (3001, 200, 10), (66_001, 20, 15)])
def test_neighbours_of_a_set_with_rows_that_are_not_numbers(gpu_ctx, n, d, k):
    x = with_bad_rows(n, d, k)
    ids, ds = gpu_knn(gpu_ctx, x, x, k)          # two arrays: the plain sweep
    ids2, ds2 = self_knn(gpu_ctx, x, k)          # one array: the screen
    np.testing.assert_array_equal(ids2, ids)
    np.testing.assert_array_equal(bits(ds2), bits(ds))
    bad = ~np.isfinite(x).all(axis=1)
    assert (ids[bad] == n).all() and not np.isin(ids[~bad], np.flatnonzero(bad)).any()
