"""The tensor-core screens on rows of 129 to 256 features (three and four 64-column K blocks):
the accumulation model and the bound at the wider K, and whole fits against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests import test_gpu_accumulation as A
from tests.test_gpu_fit import assert_fit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["bf16", "fp16"])
@pytest.mark.parametrize("d", [129, 192, 193, 256])
@pytest.mark.parametrize("name", ["mixed_exponents", "cancellation", "equal_magnitudes",
                                  "one_giant"])
def test_accumulation_model_at_wider_rows(gpu_ctx, fmt, d, name):
    A.test_accumulation_within_a_quarter_of_the_model(gpu_ctx, fmt, d, name)


@pytest.mark.parametrize("fmt", ["bf16", "fp16"])
@pytest.mark.parametrize("d", [129, 200, 256])
@pytest.mark.parametrize("offset,tiny", [(0.0, False), (10.0, False), (1000.0, False), (3.0, True)])
def test_bound_at_wider_rows(gpu_ctx, fmt, d, offset, tiny):
    A.test_bound_never_exceeds_the_reference_distance(gpu_ctx, fmt, d, offset, tiny)


@pytest.mark.parametrize("precision", ["bf16_refined", "fp16_refined"])
@pytest.mark.parametrize("d,k", [(129, 15), (192, 1), (193, 32), (256, 5)])
@pytest.mark.parametrize("family", ["vmf", "blobs", "lattice"])
def test_wide_fits_run_the_screens_and_equal_the_oracle(gpu_ctx, family, d, k, precision):
    n = 2600
    if family == "vmf":
        x = synthetic.vmf_like(n=n, d=d, clusters=12, seed=d)
    elif family == "blobs":
        x = synthetic.blobs_with_noise(n=n, d=d, centers=6, seed=d)
    else:  # many tied distances and duplicates
        x = np.random.default_rng(d).integers(0, 2, size=(n, d)).astype(np.float32)
        x[1::3] = x[::3][: x[1::3].shape[0]]
    got = gpu_ctx.fit_core(x, k, _lib.PRECISIONS[precision])
    assert got["stats"]["screen_tile_pairs"] > 0
    assert_fit_equal(got, O.fit_core(x, k))


def test_more_than_256_features_stay_refused(gpu_ctx):
    x = np.zeros((2100, 257), np.float32)
    x[:, 0] = np.arange(2100)
    for precision in _lib.PRECISIONS.values():
        with pytest.raises(OverflowError, match="at most 256 features"):
            gpu_ctx.fit_core(x, 5, precision)
