"""Device memory that calls hold: what a call takes is kept in the context's workspace, counted and
given back with it."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


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
