"""Calls of one context on different streams: each waits for the work of the one before it, which may
still be queued on its own stream when its call has returned."""
from __future__ import annotations

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import _lib, synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DELAY = 200_000_000  # cycles: about 0.1 s


def queued_call(ctx):
    """A small call queued behind a delay on a stream of its own; the event behind it."""
    n, d = 300, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(n, d, generator=g, device="cuda")
    core = torch.zeros(n, device="cuda")
    comp = torch.arange(n, device="cuda", dtype=torch.int32) // 10
    w = torch.empty(n, device="cuda")
    dst = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    side, done = torch.cuda.Stream(), torch.cuda.Event()

    def call():
        ctx.boruvka_candidates(x.data_ptr(), core.data_ptr(), comp.data_ptr(), n, d, w.data_ptr(),
                               dst.data_ptr(), side.cuda_stream)

    call()  # kernels loaded and buffers there: nothing in the queued call waits for the device
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(DELAY)
        call()
        done.record(side)
    assert not done.query()
    return done, (x, core, comp, w, dst)


@pytest.fixture(scope="module")
def model():
    x = synthetic.gaussian_mixture(8300, 64, 10, seed=3)
    return cg.HDBSCAN(min_cluster_size=50, min_samples=5, precision="fp16_refined").fit(x[:8000]), x


CALLS = {
    "fit": lambda ctx, m, x: ctx.fit_core(x[:500], 5, _lib.PRECISION_PLAIN),
    "refined_fit": lambda ctx, m, x: ctx.fit_core(x[:2100], 5, _lib.PRECISION_BF16_REFINED),
    "pack": lambda ctx, m, x: ctx.fit_core_packed([(x[:400], 5, _lib.PRECISION_PLAIN)]),
    "predictor": lambda ctx, m, x: cg.prediction.Predictor.from_state(
        *m.to_predictor()._predictor.export_state(), ctx),
    "release": lambda ctx, m, x: ctx.release_workspace(),
}


@pytest.mark.parametrize("name", CALLS)
def test_a_call_waits_for_the_work_before_it(gpu_ctx, model, name):
    for _ in range(2):
        CALLS[name](gpu_ctx, *model)
    done, kept = queued_call(gpu_ctx)
    CALLS[name](gpu_ctx, *model)
    assert done.query()


@pytest.mark.parametrize("m", [100, 4096])
def test_a_prediction_waits_for_the_work_before_it(gpu_ctx, model, m):
    fitted, x = model
    predictor = fitted.to_predictor()
    batch = np.concatenate([x[8000:]] * 14)[:m]
    for _ in range(2):
        predictor.approximate_predict(batch)
    done, kept = queued_call(gpu_ctx)
    predictor.approximate_predict(batch)
    assert done.query()


def test_device_calls_wait_on_the_device_not_on_the_host(gpu_ctx):
    g = torch.Generator(device="cuda").manual_seed(2)
    n, d, k = 500, 8, 5
    x = torch.rand(n, d, generator=g, device="cuda")
    ids = torch.empty((n, k), dtype=torch.int32, device="cuda")
    ds = torch.empty((n, k), device="cuda")
    other, second = torch.cuda.Stream(), torch.cuda.Event()
    other.wait_stream(torch.cuda.current_stream())

    def call():
        gpu_ctx.exact_knn(x.data_ptr(), n, x.data_ptr(), n, d, k, True, 0, True, ids.data_ptr(),
                          ds.data_ptr(), other.cuda_stream)

    call()
    first, kept = queued_call(gpu_ctx)
    call()
    second.record(other)
    assert not first.query()
    second.synchronize()
    assert first.query()
