"""Exact kNN and BitHash on one stream while searches run on another (GPU).

Their CTAs take an SM's whole tensor memory, which the search's CTAs use for
their queues: they start as those end.  All three give what they give alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_three_kernels_share_the_device(cuda, song, ds):
    torch = cuda
    n, nq, dim = 20000, 4000, 64
    m = ds.int_mixture(n, nq, dim=dim, n_comp=16, seed=12)
    adj = song.build_graph(m.base, song.Params())
    b = torch.from_numpy(m.base).cuda()
    q = torch.from_numpy(m.queries).cuda()
    h = song.BitHash(dim, 3, 256)
    R = torch.from_numpy(h.R).cuda()
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    with song.KernelGraph(n, dim, m.base, song.Params(pq_size=400), adj=adj) as g:
        g.upload_to_gpu()

        def buffers():
            return (torch.full((4, nq, 10), -7, dtype=torch.int32, device="cuda"),
                    torch.full((nq, 10), -7, dtype=torch.int32, device="cuda"),
                    torch.full((nq, 10), -7.0, device="cuda"),
                    torch.full((n, 8), -7, dtype=torch.int32, device="cuda"))

        def searches(out):
            for part in out:
                song.search_device(g, q, nq, 10, 400, part, stream=sa)

        def others(ids, d, codes):
            h.project_device(R, b, n, codes, stream=sb)
            song.exact_knn_device(b, n, dim, q, nq, 10, ids, d, stream=sb)
            h.project_device(R, b, n, codes, stream=sb)

        alone = buffers()
        torch.cuda.synchronize()
        searches(alone[0])
        torch.cuda.synchronize()
        others(*alone[1:])
        torch.cuda.synchronize()
        for _ in range(3):
            both = buffers()
            torch.cuda.synchronize()
            searches(both[0])
            others(*both[1:])
            searches(both[0])
            torch.cuda.synchronize()
            for x, y in zip(alone, both):
                np.testing.assert_array_equal(x.cpu().numpy(), y.cpu().numpy())
