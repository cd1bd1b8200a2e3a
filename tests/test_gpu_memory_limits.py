"""Calls on a device that is almost full (GPU).

The workspace that the library keeps between calls is given back to
allocations that would fail, and what is only there for speed (the byte copy
of a build's rows, lists for all queries of an exact kNN at once) is not
required: each call gives the result it gives with room to spare.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


class NearlyFull:
    """Leaves about `free_mb` of the device free while the block runs."""

    def __init__(self, torch, free_mb):
        self.torch, self.free = torch, free_mb * MB

    def __enter__(self):
        self.torch.cuda.synchronize()
        self.torch.cuda.empty_cache()
        left = self.torch.cuda.mem_get_info()[0]
        self.block = self.torch.empty((left - self.free) // (2 * MB) * (2 * MB), dtype=self.torch.uint8, device="cuda")

    def __exit__(self, *exc):
        del self.block
        self.torch.cuda.empty_cache()


def knn_device(torch, song, b, q, k):
    ids = torch.empty((q.shape[0], k), dtype=torch.int32, device="cuda")
    d = torch.empty((q.shape[0], k), device="cuda")
    song.exact_knn_device(b, b.shape[0], b.shape[1], q, q.shape[0], k, ids, d, stream=torch.cuda.current_stream())
    return ids, d


def give_back(song):
    """Destroying an index gives the kept workspace back."""
    rows = np.zeros((4, 4), np.float32)
    with song.KernelGraph(4, 4, rows, song.Params(), adj=np.full((4, 32), -1, np.int32)) as g:
        g.upload_to_gpu()


@pytest.fixture
def kept(cuda, song):
    """A call that leaves about 800 MB of workspace with the library."""
    torch = cuda
    give_back(song)
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    b = torch.randint(0, 255, (1_000_000, 192), device="cuda", dtype=torch.int32).float()
    q = b[:64].clone()
    knn_device(torch, song, b, q, 10)
    del b, q
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info()[0] > 700 * MB
    yield torch
    give_back(song)


def test_other_allocators_get_it_right_after_a_call(cuda, song):
    """Without a synchronisation in between: the call's workspace is free, not
    only on its way to be."""
    torch = cuda
    b = torch.randint(0, 255, (1_000_000, 192), device="cuda", dtype=torch.int32).float()
    q = b[:64].clone()
    ids = torch.empty((64, 10), dtype=torch.int32, device="cuda")
    d = torch.empty((64, 10), device="cuda")
    knn_device(torch, song, b, q, 10)
    give_back(song)
    with NearlyFull(torch, 1100):  # the call takes about 800 of them
        song.exact_knn_device(b, b.shape[0], 192, q, 64, 10, ids, d, stream=torch.cuda.current_stream())
        other = torch.empty(600 * MB, dtype=torch.uint8, device="cuda")
        del other


def test_larger_workspace_than_the_kept_one(kept, song):
    torch = kept
    b = torch.randint(0, 255, (1_150_000, 192), device="cuda", dtype=torch.int32).float()
    q = b[:64].clone()
    with NearlyFull(torch, 250):
        ids, d = knn_device(torch, song, b, q, 1)
    assert torch.equal(ids[:, 0].cpu(), torch.arange(64, dtype=torch.int32)) and not d.any()


def test_host_codes_get_the_kept_workspace(kept, song):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((250_000, 512), dtype=np.float32)  # 512 MB on the device
    h = song.BitHash(512, seed=5, hash_bits=64)
    want = h.project_all(x[:1000])
    with NearlyFull(kept, 300):
        got = h.project_all(x)
    np.testing.assert_array_equal(got[:1000], want)


def test_host_knn_gets_the_kept_workspace(kept, song):
    rng = np.random.default_rng(4)
    b = rng.integers(0, 100, (200_000, 448)).astype(np.float32)  # 358 MB, and as much workspace
    q = b[:20] + 1.0
    want, wd = song.exact_knn(b[:1000], q, 5)
    with NearlyFull(kept, 250):
        ids, d = song.exact_knn(b, q, 5)
    for i in range(20):  # each query is row i plus 1: distance 448, the nearest by far
        assert ids[i, 0] == want[i, 0] == i and d[i, 0] == wd[i, 0] == 448.0


def test_build_without_room_for_byte_rows(cuda, song):
    torch = cuda
    n, dim = 600_000, 256  # 614 MB of rows, 77 MB of adjacency, 154 MB of byte rows
    rng = np.random.default_rng(6)
    centres = rng.integers(20, 230, (64, dim))
    rows = (centres[rng.integers(0, 64, n)] + rng.integers(-20, 20, (n, dim))).astype(np.float32)
    p = song.Params(search_degree=8, ef_construction=24)
    want = song.build_graph(rows, p)
    give_back(song)
    with NearlyFull(torch, 614 + 77 + 90):
        got = song.build_graph(rows, p)
    np.testing.assert_array_equal(got, want)
    give_back(song)


def test_knn_without_room_for_all_lists(cuda, song):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(7)
    b = torch.randn((1000, 8), device="cuda", generator=g)
    q = torch.randn((200_000, 8), device="cuda", generator=g)  # lists of 410 MB
    want, wd = knn_device(torch, song, b, q, 17)
    give_back(song)
    with NearlyFull(torch, 200):
        ids, d = knn_device(torch, song, b, q, 17)
    assert torch.equal(ids, want) and torch.equal(d, wd)
