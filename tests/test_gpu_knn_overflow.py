"""Exact kNN where FP32 overflows (GPU).

One dimension of BF16 values makes every product exact, so the distance is
(|q|^2 - 2 q b) + |b|^2 in FP32 and numpy gives the same bits.  With values
near 1e19 the term 2 q b overflows for some rows and their distance is -inf:
they come first, wherever in the base they stand and whatever the threshold
is by then.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bf16(x):
    return (np.asarray(x, np.float32).view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)


def ordered(q, base, k):
    with np.errstate(over="ignore", invalid="ignore"):
        qn, bn = (np.float64(q) ** 2).astype(np.float32), (base.astype(np.float64) ** 2).astype(np.float32)
        d = ((qn - np.float32(2) * (np.float32(q) * base)) + bn) + np.float32(0)
    assert not np.isnan(d).any()
    ids = np.lexsort((np.arange(len(d)), d))[:k]
    return ids, d[ids]


@pytest.mark.parametrize("n,k", [(300, 4), (5000, 4), (5000, 40), (40000, 1)])
def test_overflowing_products(cuda, song, n, k):
    rng = np.random.default_rng(n + k)
    base = bf16(rng.uniform(0.95e19, 1.05e19, n).astype(np.float32))
    late = rng.choice(np.arange(n // 2, n), 3, replace=False)
    base[late] = bf16(np.float32([1.5e19, 1.6e19, 1.7e19]))  # 2 * 1.2e19 * 1.5e19 > FLT_MAX
    q = bf16(np.float32([1.2e19, 1.0e19, -1.2e19, 3.0, 1.25e19]))
    ids, d = song.exact_knn(base[:, None], q[:, None], k)
    for i in range(len(q)):
        want, wd = ordered(q[i], base, k)
        np.testing.assert_array_equal(ids[i], want, err_msg=f"query {i}")
        np.testing.assert_array_equal(d[i], wd, err_msg=f"query {i}")
