"""The register-tiled exact sweeps (64 queries x 128 references, 16-feature stages) at the edges
of their tiles, list widths and splits, bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_ops import bits, gpu_candidates, gpu_knn

pytestmark = pytest.mark.gpu


def rows(kind: str, n: int, d: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    if kind == "lattice":  # few distinct distances: ties decided by id
        return rng.integers(0, 3, size=(n, d)).astype(np.float32)
    if kind == "overflow":  # infinite squared distances beside finite ones
        x = rng.normal(size=(n, d))
        x[rng.random(n) < 0.4] *= 1e20
        return x.astype(np.float32)
    return rng.normal(size=(n, d)).astype(np.float32)


@pytest.mark.parametrize("squared", [True, False])
@pytest.mark.parametrize("kind,nq,nr,d,k", [
    ("normal", 1, 1, 1, 1), ("lattice", 63, 127, 15, 2), ("lattice", 64, 128, 16, 31),
    ("lattice", 65, 129, 17, 32), ("normal", 130, 300, 33, 33), ("lattice", 64, 257, 2, 64),
    ("normal", 65, 700, 5, 65), ("lattice", 66, 500, 7, 128), ("normal", 30, 900, 3, 129),
    ("lattice", 70, 600, 4, 256), ("normal", 20, 400, 6, 257), ("normal", 70, 260, 256, 10),
    ("overflow", 90, 300, 12, 20), ("overflow", 70, 200, 9, 150), ("normal", 3, 20_000, 10, 10),
    ("lattice", 200, 5000, 3, 1), ("normal", 64, 40, 8, 50), ("overflow", 65, 129, 4, 1)])
def test_knn_at_tile_and_list_edges(gpu_ctx, kind, nq, nr, d, k, squared):
    q, r = rows(kind, nq, d, 1), rows(kind, nr, d, 2)
    r[: min(nq, nr)] = q[: min(nq, nr)]  # exact zeros beside the excluded self
    for exclude, offset in ((True, 0), (True, 5), (False, 0)):
        ids, ds = gpu_knn(gpu_ctx, q, r, k, exclude, offset, squared)
        eids, eds = O.exact_neighbors(q, r, k, exclude_self=exclude, query_offset=offset,
                                      squared=squared)
        np.testing.assert_array_equal(ids, eids)
        np.testing.assert_array_equal(bits(ds), bits(eds))


@pytest.mark.parametrize("kind,n,d,comps", [
    ("normal", 2, 1, 2), ("lattice", 63, 15, 3), ("lattice", 64, 16, 2), ("lattice", 129, 17, 64),
    ("normal", 257, 256, 5), ("overflow", 300, 12, 7), ("lattice", 1000, 3, 1),
    ("lattice", 5000, 4, 9), ("normal", 5000, 31, 5000)])
@pytest.mark.parametrize("sort", [True, False])
def test_candidates_at_tile_edges(gpu_ctx, kind, n, d, comps, sort):
    """Sorted labels make uniform query tiles, which skip the reference tiles of their own
    component."""
    rng = np.random.default_rng(n + d)
    x = rows(kind, n, d, 3)
    core = rng.uniform(0, d, size=n).astype(np.float32)
    core[rng.random(n) < 0.3] = 0.0
    core[rng.random(n) < 0.05] = np.inf
    comp = rng.integers(0, comps, size=n).astype(np.int32)
    if sort:
        comp = np.sort(comp)
    w, j = gpu_candidates(gpu_ctx, x, core, comp)
    ew, ej = O.boruvka_candidates(x, core, comp)
    np.testing.assert_array_equal(bits(w), bits(ew))
    np.testing.assert_array_equal(j, ej)
