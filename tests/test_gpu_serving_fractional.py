"""Serving queries that are not whole numbers on an index with byte rows (GPU).

Such a query is compared with the float rows and read from its ring slot in
device memory throughout the search.  The slots are rewritten while the
kernel runs, so with one CTA, 8 slots and 25 times as many requests every
slot is read again and again by the same SM: each result must be that of the
request in the slot, ids and trace as searched alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,ef", [(8000, 128, 64), (8000, 37, 64), (40, 128, 16), (40, 8, 16)])
def test_reused_slots_hold_the_new_query(cuda, song, ds, n, dim, ef):
    """The small indexes stay in the SM's first-level cache beside the query."""
    nq, slots, k = 200, 8, 10
    m = ds.int_mixture(n, nq, dim=dim, n_comp=16, seed=dim)
    q = (m.queries + np.float32(0.375)).astype(np.float32)
    adj = song.build_graph(m.base, song.Params())
    with song.KernelGraph(n, dim, m.base, song.Params(pq_size=64), adj=adj) as g:
        g.upload_to_gpu()
        tr = song.GpuSearchTrace()
        want, _ = song.gpu_search_ex(g, song.SearchOpts(), q, nq, k, ef, trace=tr)
        cfg = song.ServerConfig(max_k=k, max_ef=ef, ring_slots=slots, max_ctas=1, idle_exit_us=2_000_000)
        with song.Server(g, cfg) as srv:
            for s in range(0, nq, slots):
                t0 = srv.submit(q[s:s + slots], np.full(slots, k, np.int32), np.full(slots, ef, np.int32),
                                np.zeros(slots, np.int32))
                for i in range(slots):
                    ids, _, t = srv.wait(t0 + i, k, timeout_us=30_000_000)
                    np.testing.assert_array_equal(ids, want[s + i], err_msg=f"request {s + i}")
                    np.testing.assert_array_equal(t, tr.queries[s + i], err_msg=f"trace {s + i}")
