"""Operations that order rows on a context that no fit has run on, in device memory that held something
else: the first exact_knn of a set against itself, and the first predictor, on a new context and
after release_workspace."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cuscan_gb300 as cg
from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_ops import bits

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def fill_free_memory(pattern=0x5A):
    """Small and large device blocks filled with a pattern and given back, so that the allocations
    that follow are handed memory that is not zero."""
    cuda = C.CDLL("libcuda.so.1")
    blocks = []
    for size, count in ((64, 512), (256, 512), (512, 256), (8 << 10, 256), (64 << 10, 64),
                        (1 << 20, 32), (16 << 20, 4)):
        for _ in range(count):
            at = C.c_uint64(0)
            assert cuda.cuMemAlloc_v2(C.byref(at), C.c_size_t(size)) == 0
            assert cuda.cuMemsetD8_v2(at, C.c_ubyte(pattern), C.c_size_t(size)) == 0
            blocks.append(at)
    assert cuda.cuCtxSynchronize() == 0
    for at in blocks:
        assert cuda.cuMemFree_v2(at) == 0


def self_knn(ctx, x, k):
    """exact_knn of one array against itself, the form that may take the screen."""
    n, d = x.shape
    rows = torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()
    ids = torch.empty((n, k), dtype=torch.int32, device="cuda")
    ds = torch.empty((n, k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.exact_knn(rows.data_ptr(), n, rows.data_ptr(), n, d, k, True, 0, True, ids.data_ptr(),
                  ds.data_ptr())
    torch.cuda.synchronize()
    return ids.cpu().numpy(), ds.cpu().numpy()


def searches_spatially(predictor, m):
    """Whether a batch of m queries is searched in spatial order: its bound has the order's arrays."""
    k, n = 2 * predictor.min_samples, predictor.n_finite
    lists = 8 * k * min(512 * 152 + m, m * -(-(-(-n // 128)) // 2))
    plain = 4 * m * predictor.n_features_in_ + 8 * m * k + lists + (1 << 20)
    bound = cg.load().cuscan_predict_workspace_bytes(predictor.handle, m)
    assert bound >= plain
    return bound > plain


@pytest.mark.parametrize("n,d,k", [(2048, 32, 5), (5003, 64, 10), (2600, 200, 15)])
@pytest.mark.parametrize("released", [False, True])
def test_exact_knn_needs_no_fit_before_it(gpu_ctx, n, d, k, released):
    x = synthetic.gaussian_mixture(n, d, 9, seed=n)
    ctx = _lib.Context(0)
    if released:
        ctx.fit_core(x[:2100], 5, _lib.PRECISION_BF16_REFINED)
        ctx.release_workspace()
    fill_free_memory()
    for _ in range(2):
        ids, ds = self_knn(ctx, x, k)
        eids, eds = O.exact_neighbors(x, x, k)
        np.testing.assert_array_equal(ids, eids)
        np.testing.assert_array_equal(bits(ds), bits(eds))


@pytest.mark.parametrize("restored", [False, True])
def test_a_predictor_needs_no_fit_before_it(restored):
    n, d, m = 66_000, 16, 4096
    x = synthetic.gaussian_mixture(n + m, d, 10, seed=3)
    model = cg.HDBSCAN(min_cluster_size=50, min_samples=5, precision="fp16_refined").fit(x[:n])
    if restored:
        arrays, meta = model.to_predictor()._predictor.export_state()
        ctx = _lib.Context(0)
        fill_free_memory()
        predictor = cg.prediction.Predictor.from_state(arrays, meta, ctx)
    else:
        cg.context(0).release_workspace()
        fill_free_memory()
        predictor = model.to_predictor()._predictor
    # a batch large enough for the spatial search, against pieces searched plainly
    assert searches_spatially(predictor, m) and not searches_spatially(predictor, 200)
    whole = predictor.predict(x[n:])
    parts = [predictor.predict(x[a:a + 200]) for a in range(n, n + m, 200)]
    for got, exp in zip(whole, zip(*parts)):
        np.testing.assert_array_equal(got, np.concatenate(exp))
