"""Float row distances of the search against the oracle (GPU).

Ids and all twelve trace counters equal the oracle's, so every distance that
the search compared has the bits of the reference's summation order.  Sizes
sit at the edges of the row reader: rows of less than one 16-byte load, the
last load partly past dim, one load below and above a pass (8 lanes x 8
loads x 4 floats = 256), more than one pass; seed counts of 1 to 9 make the
first pass read 1 to 9 rows (4 and 8 are its tile edges).  The queries start
at an odd float, so the caller's rows have no alignment.
"""
import numpy as np
import pytest

from conftest import knn_graph

pytestmark = pytest.mark.gpu


def _run(cuda, song, g, q, k, ef):
    torch = cuda
    nq, dim = q.shape
    buf = torch.empty(nq * dim + 1, device="cuda")
    buf[1:] = torch.from_numpy(q.reshape(-1)).cuda()
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    tr = torch.empty((nq, 12), dtype=torch.int32, device="cuda")
    ids_nt = torch.empty_like(ids)
    song.search_device(g, buf[1:], nq, k, ef, ids, tr)
    song.search_device(g, buf[1:], nq, k, ef, ids_nt)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(ids.cpu().numpy(), ids_nt.cpu().numpy())
    return ids.cpu().numpy(), tr.cpu().numpy()


@pytest.mark.parametrize("dim,nmp", [(1, 1), (3, 2), (4, 3), (5, 4), (31, 5), (33, 7), (127, 8),
                                     (130, 9), (252, 4), (256, 4), (257, 4), (260, 5), (515, 8)])
def test_float_rows_match_oracle(cuda, song, ds, oracle, dim, nmp):
    m = ds.angular_mixture(600, 40, dim=dim, n_comp=4, seed=dim)
    adj = knn_graph(m.base, 32, 24, seed=dim)
    p = song.Params(pq_size=48, bf_words=64, n_multiprobe=nmp)
    with song.KernelGraph(600, dim, m.base, p, adj=adj) as g:
        g.upload_to_gpu()
        ids, tr = _run(cuda, song, g, m.queries, 10, 48)
    oids, otr = oracle.search_l2(m.base, adj, 32, m.queries, 10, 48, pq_size=48, bf_words=64, n_multiprobe=nmp)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr, otr)


@pytest.mark.parametrize("dim", [5, 100, 128, 200, 256])
def test_float_queries_on_byte_rows_match_oracle(cuda, song, ds, oracle, dim):
    """An index with byte rows and queries that are not whole numbers: the
    float path of the byte-row instances, reading the caller's query rows."""
    m = ds.int_mixture(600, 40, dim=dim, n_comp=4, seed=dim)
    q = (m.queries + np.float32(0.37)).astype(np.float32)
    q[::5] = m.queries[::5]
    adj = knn_graph(m.base, 32, 24, seed=dim)
    p = song.Params(pq_size=48, bf_words=64)
    with song.KernelGraph(600, dim, m.base, p, adj=adj) as g:
        g.upload_to_gpu()
        assert g.u8_rows() > 0
        ids, tr = _run(cuda, song, g, q, 10, 48)
    oids, otr = oracle.search_l2(m.base, adj, 32, q, 10, 48, pq_size=48, bf_words=64)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr, otr)


def test_query_too_large_for_shared_memory(cuda, song, ds, oracle):
    """Filters so large that four warps leave no room for their queries: the
    search reads the query from global memory instead."""
    m = ds.angular_mixture(500, 20, dim=256, n_comp=4, seed=3)
    adj = knn_graph(m.base, 32, 24, seed=3)
    bfw = 7180  # 4 x 57,440 bytes of filters; the queries would take 4,096 more
    p = song.Params(pq_size=32, bf_words=bfw)
    with song.KernelGraph(500, 256, m.base, p, adj=adj) as g:
        g.upload_to_gpu()
        ids, tr = _run(cuda, song, g, m.queries, 10, 32)
    oids, otr = oracle.search_l2(m.base, adj, 32, m.queries, 10, 32, pq_size=32, bf_words=bfw)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr, otr)
