"""The one-CTA forest steps of small fits on either side of their thread counts: alone and in packs whose
largest fit decides, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_fit import assert_fit_equal

pytestmark = pytest.mark.gpu


def rows(n):
    if n < 10:
        return np.random.default_rng(n).normal(size=(n, 3)).astype(np.float32)
    return synthetic.gaussian_mixture(n, 7, 3, seed=n)


@pytest.mark.parametrize("n", [2, 3, 31, 33, 255, 257, 511, 512, 513, 1024, 2047])
@pytest.mark.parametrize("others", [(), (2, 40), (300, 5)])
def test_small_fits_equal_the_oracle(gpu_ctx, n, others):
    sets = [rows(m) for m in (n, *others)]
    for got, x in zip(gpu_ctx.fit_core_packed([(x, 4, _lib.PRECISION_PLAIN) for x in sets]), sets):
        assert_fit_equal(got, O.fit_core(x, 4))
    assert_fit_equal(gpu_ctx.fit_core(sets[0], 4, _lib.PRECISION_PLAIN), O.fit_core(sets[0], 4))
