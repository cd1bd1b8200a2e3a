"""Searches whose queues live in registers, at the edges of their sizes (GPU).

Ids and traces equal the oracle's for queue sizes on both sides of every
size at which the kernel changes (64, 128, 160 and 256 slots; more is the
other queue) and for sizes that are not whole groups of 32, on data with many
tied distances (few distinct rows, so the queues' slot order decides),
untied floats and Hamming codes; enough queries for the 161 .. 256 slot
queues to take either kernel.  The precision form on integers and the learned
form from the reference's seeds compute the same search, so they are compared
with the plain one at each size.
"""
import numpy as np
import pytest

from conftest import knn_graph

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 64, 65, 128, 129, 160, 161, 256, 257]


def _tied(rng, n, dim):
    proto = rng.integers(0, 9, size=(60, dim)).astype(np.float32)
    return proto[rng.integers(0, 60, size=n)]


def _data(kind, rng, ds):
    if kind == "tied":
        return _tied(rng, 900, 12), _tied(rng, 50, 12)
    m = ds.angular_mixture(900, 50, dim=40, n_comp=4, seed=7)
    return m.base, m.queries


@pytest.mark.parametrize("ef", SIZES)
@pytest.mark.parametrize("kind", ["tied", "float"])
def test_l2_matches_oracle(cuda, song, ds, oracle, kind, ef):
    rng = np.random.default_rng(ef)
    base, q = _data(kind, rng, ds)
    adj = knn_graph(base, 32, 24, seed=ef)
    p = song.Params(pq_size=ef, bf_words=40)
    k = min(ef, 12)
    tr = song.GpuSearchTrace()
    with song.KernelGraph(900, base.shape[1], base, p, adj=adj) as g:
        g.upload_to_gpu()
        ids = song.gpu_search(g, q, 50, k, ef_search=ef, trace=tr).reshape(50, k)
        ids_nt = song.gpu_search(g, q, 50, k, ef_search=ef).reshape(50, k)
        many = np.tile(q, (16, 1))  # 200 CTAs of four queries: more than one per SM
        ids_many = song.gpu_search(g, many, 800, k, ef_search=ef).reshape(16, 50, k)
    oids, otr = oracle.search_l2(base, adj, 32, q, k, ef, pq_size=ef, bf_words=40)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr.queries, otr)
    np.testing.assert_array_equal(ids_nt, oids)
    for part in ids_many:
        np.testing.assert_array_equal(part, oids)


@pytest.mark.parametrize("words,ef", [(1, 64), (3, 65), (5, 128), (8, 160), (16, 161), (17, 256), (32, 257)])
def test_hamming_matches_oracle(cuda, song, oracle, words, ef):
    rng = np.random.default_rng(words)
    bits = rng.random((900, words * 32)) < 0.5
    codes = np.packbits(bits, axis=1, bitorder="little").view(np.uint32).reshape(900, words)
    q = codes[rng.integers(0, 900, 50)] ^ (rng.random((50, words)) < 0.1).astype(np.uint32)
    adj = knn_graph(bits.astype(np.float32), 32, 24, seed=words)
    tr = song.GpuSearchTrace()
    with song.HashKernelGraph(900, codes, song.Params(pq_size=ef, bf_words=64), adj=adj) as g:
        g.upload_to_gpu()
        ids = song.gpu_search(g, q, 50, 10, ef_search=ef, trace=tr).reshape(50, 10)
    oids, otr = oracle.search_hamming(codes, adj, 32, q, 10, ef, pq_size=ef, bf_words=64)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(tr.queries, otr)


@pytest.mark.parametrize("ef", [33, 64, 128, 160, 256, 257])
def test_other_forms_equal_the_plain_search(cuda, song, ef):
    torch = cuda
    rng = np.random.default_rng(ef)
    base, q = _tied(rng, 900, 12), _tied(rng, 50, 12)
    adj = knn_graph(base, 32, 24, seed=ef)
    dq = torch.from_numpy(q).cuda()
    with song.KernelGraph(900, 12, base, song.Params(pq_size=ef, bf_words=64), adj=adj) as g:
        g.upload_to_gpu()
        song.set_precision(g, song.PREC_BF16)
        own = torch.arange(0, 900, 3, dtype=torch.int32, device="cuda")
        song.learn(g, torch.from_numpy(base[::3]).cuda(), 300, own,
                   song.LearnParams(ef=32, entry_steps=2, stop_steps=2, batch=64, entry_hubs=128))
        forms = [song.SearchOpts(), song.SearchOpts(precision=song.PREC_BF16),
                 song.SearchOpts(learned=True, stop_threshold=1.0, entry=song.ENTRY_SEEDS)]
        got = []
        for o in forms:
            ids = torch.empty((50, 10), dtype=torch.int32, device="cuda")
            d = torch.empty((50, 10), device="cuda")
            tr = torch.empty((50, 12), dtype=torch.int32, device="cuda")
            song.search_device_ex(g, o, dq, 50, 10, ef, ids, d, tr)
            torch.cuda.synchronize()
            got.append([x.cpu().numpy() for x in (ids, d, tr)])
        rr = torch.empty((50, 10), device="cuda")
        ids = torch.empty((50, 10), dtype=torch.int32, device="cuda")
        song.search_device_ex(g, song.SearchOpts(precision=song.PREC_BF16, rerank=True), dq, 50, 10, ef, ids, rr)
        torch.cuda.synchronize()
    for form in got[1:]:
        for a, b in zip(form, got[0]):
            np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(rr.cpu().numpy(), got[0][1])  # the same distances; ties by id
