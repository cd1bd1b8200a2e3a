"""Exact kNN at a very large dimension (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_dimension_above_four_million(cuda, song):
    """Two query tiles with lo parts (values that take more than 8 bits) of 2^17
    chunks of 32 dimensions: their size in bytes does not fit 32 bits."""
    torch = cuda
    dim, n, nq, used = (1 << 22) + 32, 6, 130, 40
    rng = np.random.default_rng(1)
    at = torch.from_numpy(rng.choice(dim, used, replace=False)).cuda()
    bv = rng.integers(0, 100, (n, used)).astype(np.float32)
    qv = rng.integers(0, 600, (nq, used)).astype(np.float32)
    b = torch.zeros((n, dim), device="cuda")
    q = torch.zeros((nq, dim), device="cuda")
    b[:, at] = torch.from_numpy(bv).cuda()
    q[:, at] = torch.from_numpy(qv).cuda()
    ids = torch.empty((nq, n), dtype=torch.int32, device="cuda")
    d = torch.empty((nq, n), device="cuda")
    song.exact_knn_device(b, n, dim, q, nq, n, ids, d, stream=torch.cuda.current_stream())
    want = ((qv[:, None].astype(np.int64) - bv[None].astype(np.int64)) ** 2).sum(2)
    order = np.argsort(want, axis=1, kind="stable")
    np.testing.assert_array_equal(ids.cpu().numpy(), order)
    np.testing.assert_array_equal(d.cpu().numpy(), np.take_along_axis(want, order, 1).astype(np.float32))
