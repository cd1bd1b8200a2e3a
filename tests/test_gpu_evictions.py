"""One push that evicts the same queue slot many times (GPU).

A full queue of near nodes meets an adjacency row whose 32 nodes come closer
one by one and are all farther than the rest of the queue: the first is
appended (or evicts), then each takes the slot of the one before it.  The last
writer's id must be the one that stays.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(ef, dim):
    """Seeds 0, n/4, n/2, 3n/4; near nodes in chained rows of the second seed;
    the descending row belongs to node 0, which is expanded after them."""
    n = 4 * (ef + 64)
    s = n // 4
    x = np.full(n, 1000.0, np.float32)
    adj = np.full((n, 32), -1, np.int32)
    x[[s, 2 * s, 3 * s]] = 1.0, 2.0, 3.0
    near = list(range(s + 1, s + 1 + max(ef - 5, 0)))
    x[near] = 4.0 + np.arange(len(near)) / 8.0
    owner = s
    for i in range(0, len(near), 32):
        part = near[i:i + 32]
        adj[owner, :len(part)] = part
        owner = part[-1]
    x[0] = 500.0
    far = list(range(1, 33))
    x[far] = 900.0 - np.arange(32)
    adj[0] = far
    base = np.zeros((n, dim), np.float32)
    base[:, 0] = x
    return base, adj


@pytest.mark.parametrize("dim", [4, 300])
@pytest.mark.parametrize("ef", [5, 6, 33, 64, 97, 160, 256, 257])
def test_last_of_a_descending_row_stays(cuda, song, oracle, ef, dim):
    base, adj = _case(ef, dim)
    q = np.zeros((40, dim), np.float32)
    k = ef
    tr = song.GpuSearchTrace()
    with song.KernelGraph(len(base), dim, base, song.Params(pq_size=ef, bf_words=256), adj=adj) as g:
        g.upload_to_gpu()
        ids = song.gpu_search(g, q, 40, k, ef_search=ef, trace=tr).reshape(40, k)
    oids, otr = oracle.search_l2(base, adj, 32, q, k, ef, pq_size=ef, bf_words=256)
    assert 32 in oids[0]  # the closest of the row, after 31 others
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr.queries, otr)
