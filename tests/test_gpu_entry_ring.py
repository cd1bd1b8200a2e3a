"""Learned searches of very different batch sizes through one ring (GPU).

The entry stage's buffers are a ring of 16 slots that calls of any size take
in turn.  Small calls must leave the slots ready for a large one: a batch of
8,320 queries (65 query tiles) gives the same results before and after 40
calls of 3 to 700 queries, and each small call those of its own slice.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_batches_do_not_disturb_a_large_one(cuda, song, ds):
    torch = cuda
    m = ds.int_mixture(6000, 8320, dim=32, n_comp=16, seed=5)
    adj = song.build_graph(m.base, song.Params())
    q = torch.from_numpy(m.queries).cuda()
    o = song.SearchOpts(learned=True, stop_threshold=1.0, entry=song.ENTRY_NEAREST, beam=2)
    with song.KernelGraph(6000, 32, m.base, song.Params(pq_size=64), adj=adj) as g:
        g.upload_to_gpu()
        own = torch.arange(0, 6000, 10, dtype=torch.int32, device="cuda")
        song.learn(g, torch.from_numpy(m.base[::10]).cuda(), 600, own,
                   song.LearnParams(ef=32, entry_steps=2, stop_steps=2, batch=64, entry_hubs=2048))

        def run(lo, n):
            ids = torch.empty((n, 10), dtype=torch.int32, device="cuda")
            song.search_device_ex(g, o, q[lo:lo + n].contiguous(), n, 10, 48, ids)
            return ids

        before = run(0, 8320)
        torch.cuda.synchronize()
        before = before.cpu().numpy()
        rng = np.random.default_rng(1)
        for _ in range(40):
            n = int(rng.integers(3, 700))
            lo = int(rng.integers(0, 8320 - n))
            got = run(lo, n)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(got.cpu().numpy(), before[lo:lo + n])
        after = run(0, 8320)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(after.cpu().numpy(), before)
