"""Exact kNN at the edges of its tiles, lists and splits (GPU).

Integer vectors in [0, 255] with dim <= 128 against an int64 brute force,
bit for bit: one and two query tiles per CTA (128, 129, 256, 257 queries),
list lengths of 64 and 256 (k = 16 and 17), k at its maximum, fewer bases
than a tile, whole tiles and one base more, many splits of one query tile,
few distinct rows (ties across splits and lists cut among equal distances).
"""
import numpy as np
import pytest

from test_gpu_groundtruth import _check_float, _exact_int, _gt, _int_data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,dim,k", [
    (128, 128, 32, 16), (129, 129, 33, 17), (4096, 256, 128, 16), (4097, 257, 128, 17),
    (127, 1, 8, 127), (30000, 3, 64, 128), (60000, 40, 16, 1), (9000, 513, 100, 64),
])
def test_integer_edges_exact(cuda, n, nq, dim, k):
    base, q = _int_data(n, nq, dim, seed=n + k)
    ids, d = _gt().knn(base, q, k)
    ref_ids, ref_d = _exact_int(base, q, k)
    np.testing.assert_array_equal(ids, ref_ids)
    np.testing.assert_array_equal(d, ref_d.astype(np.float32))


@pytest.mark.parametrize("k", [10, 100])
def test_ties_across_splits(cuda, k):
    rng = np.random.default_rng(k)
    proto = rng.integers(0, 256, size=(6, 48)).astype(np.float32)
    base = proto[rng.integers(0, 6, size=20000)]
    q = np.concatenate([proto, proto + 1.0]).astype(np.float32)
    ids, d = _gt().knn(base, q, k)
    ref_ids, ref_d = _exact_int(base, q, k)
    np.testing.assert_array_equal(ids, ref_ids)
    np.testing.assert_array_equal(d, ref_d.astype(np.float32))


@pytest.mark.parametrize("n,nq,dim,k", [(3000, 300, 960, 100), (3000, 100, 515, 10), (2000, 140, 260, 17)])
def test_wide_float_rows(cuda, n, nq, dim, k):
    """Queries that do not fit in shared memory (hi and lo), and rows whose
    stride is not a multiple of 4 floats."""
    rng = np.random.default_rng(dim)
    base = rng.random(size=(n, dim), dtype=np.float32)
    q = rng.random(size=(nq, dim), dtype=np.float32)
    ids, d = _gt().knn(base, q, k)
    _check_float(base, q, ids, d, k, rel=3e-5)


def test_calls_on_two_threads(cuda):
    """Two threads at once: their workspaces are their own."""
    import threading
    base, q = _int_data(20000, 200, 64, seed=8)
    ref_ids, ref_d = _exact_int(base, q, 10)
    out = {}

    def work(i):
        out[i] = [_gt().knn(base, q, 10) for _ in range(3)]

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for i in range(2):
        for ids, d in out[i]:
            np.testing.assert_array_equal(ids, ref_ids)
            np.testing.assert_array_equal(d, ref_d.astype(np.float32))


@pytest.mark.parametrize("n,nq,k", [(20000, 130, 17), (20000, 130, 100), (40000, 7, 128), (9000, 257, 64)])
@pytest.mark.parametrize("order", ["ascending", "descending"])
def test_neighbours_in_one_split(cuda, n, nq, k, order):
    """Bases sorted by their distance from where the queries lie: all neighbours
    come from the first split, or from the last one."""
    rng = np.random.default_rng(n + k)
    level = np.sort(rng.integers(0, 200, size=n))
    base = (level[:, None] + rng.integers(0, 8, size=(n, 24))).astype(np.float32)
    if order == "descending":
        base = base[::-1].copy()
    q = rng.integers(0, 8, size=(nq, 24)).astype(np.float32)
    ids, d = _gt().knn(base, q, k)
    ref_ids, ref_d = _exact_int(base, q, k)
    np.testing.assert_array_equal(ids, ref_ids)
    np.testing.assert_array_equal(d, ref_d.astype(np.float32))
