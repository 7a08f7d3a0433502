"""Sweeps in spatial order that leave out tiles by the triangle inequality: plain f32 fits large
enough to use it against the oracle, and large prediction batches against the same batch in pieces
too small for it."""
from __future__ import annotations

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_fit import assert_fit_equal

pytestmark = pytest.mark.gpu


def point_sets():
    """n^2 d >= 1e10, the smallest work that takes the spatial order."""
    rng = np.random.default_rng(17)
    yield "blobs_noise", synthetic.blobs_with_noise(n=6401, d=250, centers=12, seed=1), 5
    yield "mixture", synthetic.gaussian_mixture(8999, 127, 9, seed=2), 50
    yield "aniso", synthetic.anisotropic_mixture(n=12_600, d=64, components=20, seed=3), 10
    yield "vmf", synthetic.vmf_like(n=9000, d=128, clusters=12, seed=4), 15
    # ties across tiles, duplicates in different cells
    yield "lattice", rng.integers(0, 2, size=(10_000, 101)).astype(np.float32), 4
    yield "two_points", np.repeat(np.float32([[0.0], [3.0]]), 4000, axis=0) * np.ones((1, 160), np.float32), 7
    base = (50 * rng.normal(size=(30, 200)))[rng.integers(0, 30, 7200)]
    yield "far_duplicates", base.astype(np.float32), 33
    yield "ms1", synthetic.gaussian_mixture(7100, 200, 5, seed=5), 1
    yield "k130", synthetic.gaussian_mixture(7169, 199, 6, seed=6), 130
    # squared distances overflow between clusters and within one of them
    huge = synthetic.gaussian_mixture(6500, 240, 8, seed=7)
    huge[::3] *= np.float32(1e19)
    yield "overflow", huge, 5
    yield "tiny", synthetic.gaussian_mixture(6500, 240, 8, seed=8) * np.float32(1e-24), 5


@pytest.mark.parametrize("name,x,ms", list(point_sets()), ids=lambda v: v if isinstance(v, str) else "")
def test_plain_fits_in_spatial_order_equal_the_oracle(gpu_ctx, name, x, ms):
    assert float(x.shape[0]) ** 2 * x.shape[1] >= 1e10
    got = gpu_ctx.fit_core(x, ms, _lib.PRECISION_PLAIN)
    assert_fit_equal(got, O.fit_core(x, ms))


@pytest.mark.parametrize("n,d,ms,m", [(20_000, 64, 5, 4096), (6000, 250, 17, 2001),
                                      (30_001, 33, 40, 2500)])
def test_large_prediction_batches_equal_small_ones(n, d, ms, m):
    x = synthetic.gaussian_mixture(n + m, d, 12, seed=n)
    x[n::7] += 30.0  # queries far from every cluster
    model = cg.HDBSCAN(min_cluster_size=50, min_samples=ms, precision="fp16_refined").fit(x[:n])
    p = model.to_predictor()
    batch = x[n:]
    assert float(m) * n * d >= 2e9
    whole = p.approximate_predict(batch, True)
    parts = [p.approximate_predict(batch[a:a + 200], True) for a in range(0, m, 200)]
    for got, exp in zip(whole, zip(*parts)):
        np.testing.assert_array_equal(got, np.concatenate(exp))
