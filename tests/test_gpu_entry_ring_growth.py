"""The call that grows a learned index's entry ring is right at once (GPU).

The ring's arrival counters must be zero before the entry launch on the
caller's non-blocking stream: for fresh indexes and batches that each grow
the ring, the first call on such a stream gives what a later call gives.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_call_after_growth(cuda, song, ds):
    torch = cuda
    n, dim = 6000, 32
    m = ds.int_mixture(n, 9000, dim=dim, n_comp=16, seed=9)
    adj = song.build_graph(m.base, song.Params())
    q = torch.from_numpy(m.queries).cuda()
    own = torch.arange(0, n, 10, dtype=torch.int32, device="cuda")
    train = torch.from_numpy(m.base[::10].copy()).cuda()
    o = song.SearchOpts(learned=True, stop_threshold=1.0, entry=song.ENTRY_NEAREST, beam=2)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        with song.KernelGraph(n, dim, m.base, song.Params(pq_size=64), adj=adj) as g:
            g.upload_to_gpu()
            song.learn(g, train, len(own), own, song.LearnParams(ef=32, entry_steps=2, stop_steps=2, batch=64,
                                                                 entry_hubs=2048))
            for nq in (40, 1100, 2500, 9000):
                got = []
                for _ in range(2):
                    ids = torch.full((nq, 10), -7, dtype=torch.int32, device="cuda")
                    torch.cuda.synchronize()
                    song.search_device_ex(g, o, q, nq, 10, 48, ids, stream=stream)
                    stream.synchronize()
                    got.append(ids.cpu().numpy())
                np.testing.assert_array_equal(got[0], got[1], err_msg=f"{nq} queries")
                assert (got[0] >= 0).all()
