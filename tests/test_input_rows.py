"""Rows that an estimator keeps are its own, whatever holds the caller's float32 rows."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import cuscan_gb300 as cg
import cuscan_gb300.hdbscan as hmod


class Holder:
    def __init__(self, rows):
        self.rows = rows

    def __array__(self, dtype=None, copy=None):
        return self.rows if dtype is None else self.rows.astype(dtype)


@pytest.mark.parametrize("wrap", [lambda a: a, lambda a: a[:, :], Holder, torch.from_numpy,
                                  lambda a: np.asfortranarray(a)])
def test_fit_keeps_no_view_of_the_callers_rows(wrap, monkeypatch):
    rows = np.arange(24, dtype=np.float32).reshape(8, 3)
    seen = []

    def record(x, finite_rows, **kwargs):
        seen.append(x)
        return {}

    monkeypatch.setattr(hmod, "fit_hdbscan", record)
    X = wrap(rows)
    cg.HDBSCAN(min_cluster_size=2).fit(X)
    x, = seen
    assert not np.may_share_memory(x, rows) and not np.may_share_memory(x, np.asarray(X))
    assert x.flags.c_contiguous and x.dtype == np.float32
    np.testing.assert_array_equal(x, rows)
