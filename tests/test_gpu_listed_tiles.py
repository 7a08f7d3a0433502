"""How many tiles the kNN screen of a refined fit visits: a part of them where the cells lie apart and the
lists are used, all of them where they do not."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


def list_screen_tiles(ctx, x, min_samples):
    """(tiles of the kNN list screen, tiles of a full one): the fit's tiles without its rounds' and
    without the second screen of inconclusive rows, which visits every tile."""
    stats = ctx.fit_core(x, min_samples, _lib.PRECISION_FP16_REFINED)["stats"]
    rounds = sum(r["tiles"] for r in ctx.round_stats())
    n = x.shape[0]
    tiles = -(-n // 256)
    again = -(-stats["rescreened_rows"] // 128) * tiles
    return stats["screen_tile_pairs"] - rounds - again, -(-n // 128) * tiles


def test_lists_leave_out_most_tiles_of_separated_clusters(gpu_ctx):
    some, every = list_screen_tiles(gpu_ctx, synthetic.gaussian_mixture(50_000, 64, 20, seed=9), 5)
    assert 0 < some < 0.5 * every


def test_rows_without_separated_cells_visit_every_tile(gpu_ctx):
    rng = np.random.default_rng(4)
    x = rng.normal(size=(20_000, 64)).astype(np.float32)
    some, every = list_screen_tiles(gpu_ctx, x / np.linalg.norm(x, axis=1, keepdims=True), 5)
    assert some == every
