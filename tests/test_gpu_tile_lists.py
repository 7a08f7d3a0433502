"""Screens over lists of tiles: refined fits of well separated data, large enough to leave out the
tiles that are too far away, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_fit import assert_fit_equal

pytestmark = pytest.mark.gpu

FIRST_ROWS = 16384  # smallest fit whose screens may run lists


def point_sets():
    rng = np.random.default_rng(23)
    # the first fit with lists and the one before; last tiles and balls of one and of many rows
    for n in (FIRST_ROWS - 1, FIRST_ROWS, FIRST_ROWS + 1, FIRST_ROWS + 64, FIRST_ROWS + 129):
        yield f"mixture_{n}", synthetic.gaussian_mixture(n, 32, 12, seed=n), 5
    yield "k32", synthetic.gaussian_mixture(16_551, 64, 9, seed=1), 32
    yield "k1", synthetic.gaussian_mixture(17_000, 20, 25, seed=2), 1
    yield "odd_d", synthetic.gaussian_mixture(16_507, 77, 16, seed=3), 10
    yield "wide", synthetic.gaussian_mixture(16_400, 250, 8, seed=4), 7
    yield "aniso", synthetic.anisotropic_mixture(n=18_345, d=64, components=20, seed=5), 10
    yield "blobs_noise", synthetic.blobs_with_noise(n=16_999, d=48, centers=12, seed=6), 5
    # tight clusters far from the origin: bf16 bounds too loose, split or fp16 operands
    yield "far_tight", (synthetic.gaussian_mixture(16_401, 48, 10, seed=7) * 0.01
                        + 5 * rng.normal(size=48)).astype(np.float32), 6
    # duplicates within and across tiles, and equal distances between clusters
    base = (20 * rng.normal(size=(40, 36))).astype(np.float32)
    yield "duplicates", base[rng.integers(0, 40, 16_800)], 4
    grid = np.stack(np.meshgrid(np.arange(3), np.arange(3), np.arange(2)), -1).reshape(-1, 3)
    cells = rng.integers(0, len(grid), 17_000)
    lattice = np.concatenate([40.0 * grid[cells], rng.integers(0, 2, size=(17_000, 9))], 1)
    yield "lattice", lattice.astype(np.float32), 3


@pytest.mark.parametrize("precision", [_lib.PRECISION_BF16_REFINED, _lib.PRECISION_FP16_REFINED])
@pytest.mark.parametrize("name,x,ms", list(point_sets()), ids=lambda v: v if isinstance(v, str) else "")
def test_listed_screens_equal_the_oracle(gpu_ctx, name, x, ms, precision):
    assert_fit_equal(gpu_ctx.fit_core(x, ms, precision), O.fit_core(x, ms))


def test_lists_leave_tiles_out(gpu_ctx):
    x = synthetic.gaussian_mixture(20_000, 64, 20, seed=9)
    got = gpu_ctx.fit_core(x, 5, _lib.PRECISION_BF16_REFINED)
    blocks, tiles = -(-x.shape[0] // 128), -(-x.shape[0] // 256)
    rounds = got["stats"]["rounds"]
    assert got["stats"]["screen_tile_pairs"] < 0.8 * blocks * tiles * (1 + rounds)
    assert_fit_equal(got, O.fit_core(x, 5))
