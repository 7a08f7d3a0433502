"""Operations recorded into a CUDA graph: what can be captured, on a context that has not run them
before."""
from __future__ import annotations

import numpy as np
import pytest

from cuscan_gb300 import _lib, synthetic
from oracle import oracle as O
from tests.test_gpu_first_calls import self_knn
from tests.test_gpu_ops import bits, gpu_knn

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def captured_knn(ctx, q, r, k, exclude_self, squared):
    """The lists of a captured and replayed exact_knn."""
    n, d = q.shape
    ids = torch.full((n, k), -7, dtype=torch.int32, device="cuda")
    ds = torch.full((n, k), -7.0, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            ctx.exact_knn(q.data_ptr(), n, r.data_ptr(), r.shape[0], d, k, exclude_self, 0, squared,
                          ids.data_ptr(), ds.data_ptr(), stream.cuda_stream)
    torch.cuda.synchronize()
    assert (ids == -7).all()
    graph.replay()
    torch.cuda.synchronize()
    return ids.cpu().numpy(), ds.cpu().numpy()


@pytest.mark.parametrize("k", [33, 100, 200])
@pytest.mark.parametrize("squared", [True, False])
def test_wide_lists_are_captured_without_a_call_before(k, squared):
    x = synthetic.gaussian_mixture(3001, 20, 7, seed=k)
    q = torch.from_numpy(x).cuda()
    ctx = _lib.Context(0)
    # the kernels' attributes, on another context
    gpu_knn(_lib.Context(0), x, x, k, True, 0, squared)
    ids, ds = captured_knn(ctx, q, q, k, True, squared)
    assert ctx.reserved_bytes() == 0
    eids, eds = O.exact_neighbors(x, x, k, squared=squared)
    np.testing.assert_array_equal(ids, eids)
    np.testing.assert_array_equal(bits(ds), bits(eds))


@pytest.mark.parametrize("n,d,k", [(2048, 129, 5), (2500, 256, 15), (2100, 40, 10)])
def test_a_set_against_itself_is_captured(n, d, k):
    x = synthetic.gaussian_mixture(n, d, 7, seed=d)
    q = torch.from_numpy(x).cuda()
    ctx = _lib.Context(0)
    eids, eds = O.exact_neighbors(x, x, k)
    for _ in range(2):  # before and after a call outside a capture
        ids, ds = captured_knn(ctx, q, q, k, True, True)
        np.testing.assert_array_equal(ids, eids)
        np.testing.assert_array_equal(bits(ds), bits(eds))
        ids, ds = self_knn(ctx, x, k)
        np.testing.assert_array_equal(ids, eids)
        np.testing.assert_array_equal(bits(ds), bits(eds))
