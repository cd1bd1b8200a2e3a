"""BitHash vectors and hyperplanes whose sums have no bound (GPU).

A norm near underflow or not finite sends the bits that it touches to the
sequential sum, and no others: codes stay bit for bit the oracle's, for one
such hyperplane among 128 and for any number of such vectors per 32 (around
the 128 and 1,024 bits of a warp where the kernel changes its way of
summing), and the time stays within a small multiple of the ordinary one.
"""
import numpy as np
import pytest

from test_gpu_bithash_edges import _project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [40, 256, 333])
def test_hyperplanes(cuda, song, oracle, dim):
    rng = np.random.default_rng(dim)
    R = rng.normal(size=(288, dim)).astype(np.float32)
    x = rng.normal(size=(300, dim)).astype(np.float32)
    with np.errstate(all="ignore"):
        R[3] = 0.0
        R[4] = -0.0
        R[40] *= np.float32(1e-20)
        R[41] *= np.float32(1e-44)
        R[100] *= np.float32(1e20)
        R[101] *= np.float32(1e6)
        R[130, 5] = np.inf
        R[131, 6], R[131, 7] = np.inf, -np.inf
        R[132, 8] = np.nan
        R[133] = np.float32(3.4e38)
        R[256:] *= np.float32(1e-13)
        x[7] = 0.0
        x[8] *= np.float32(1e-20)
        x[9, 3] = np.inf
        x[10, 4] = np.nan
        x[11] *= np.float32(1e25)
        x[12] = np.float32(3.4e38)
        x[13] *= np.float32(1e-13)
        np.testing.assert_array_equal(_project(cuda, song, R, x), oracle.bithash_project(R, x))


@pytest.mark.parametrize("dim,off", [(96, 0), (97, 0), (96, 1), (300, 0)])
def test_some_vectors_of_each_32(cuda, song, oracle, dim, off):
    rng = np.random.default_rng(dim + off)
    R = rng.normal(size=(160, dim)).astype(np.float32)
    counts = [0, 1, 2, 3, 7, 8, 9, 16, 31, 32]
    x = rng.normal(size=(32 * len(counts) + 5, dim)).astype(np.float32)
    for i, c in enumerate(counts):
        x[32 * i + rng.permutation(32)[:c]] *= np.float32(1e-20)
    x[-5:] *= np.float32(1e-20)
    np.testing.assert_array_equal(_project(cuda, song, R, x, off), oracle.bithash_project(R, x))


@pytest.mark.parametrize("n,dim,bits", [(1, 4097, 32), (33, 4100, 160), (150, 5000, 512), (700, 4099, 96)])
def test_many_dimensions(cuda, song, oracle, n, dim, bits):
    """Above 4,096 dimensions every bit is a sequential sum, on tiles of 32 to
    128 vectors."""
    rng = np.random.default_rng(n)
    R = rng.normal(size=(bits, dim)).astype(np.float32)
    x = rng.normal(size=(n, dim)).astype(np.float32)
    np.testing.assert_array_equal(_project(cuda, song, R, x), oracle.bithash_project(R, x))


def test_time_does_not_hang_on_them(cuda, song):
    torch = cuda
    n, dim, bits = 60_000, 256, 512
    h = song.BitHash(dim, 2, bits)
    g = torch.Generator(device="cuda").manual_seed(1)
    x0 = torch.randn((n, dim), device="cuda", generator=g)
    codes = torch.empty((n, bits // 32), dtype=torch.int32, device="cuda")

    def ms(x, R):
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            h.project_device(R, x, n, codes, stream=torch.cuda.current_stream())
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    R0 = torch.from_numpy(h.R).cuda()
    base = ms(x0, R0)
    for scale in (0.0, 1e-20):
        R = R0.clone()
        R[5] *= scale
        assert ms(x0, R) < 4 * base
    x = x0.clone()
    x[::32] *= 1e-20
    assert ms(x, R0) < 6 * base
    assert ms(x0 * 1e-20, R0) < 25 * base


def test_more_tiles_than_marks(cuda, song):
    """More than 1,024 tiles per CTA: a mark stands for a run of tiles.  The
    codes of all vectors at once are those of slices that need no runs."""
    torch = cuda
    n, dim, bits = 1_300_000, 8, 2048
    h = song.BitHash(dim, 4, bits)
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((n, dim), device="cuda", generator=g)
    for tile in torch.randint(0, n // 128, (300,), generator=torch.Generator().manual_seed(3)).tolist():
        x[tile * 128:tile * 128 + 100] *= 1e-20
    x[-40:] *= 1e-20
    R = torch.from_numpy(h.R).cuda()
    R[7] = 0.0
    whole = torch.full((n, bits // 32), -1, dtype=torch.int32, device="cuda")
    part = torch.full((n, bits // 32), -2, dtype=torch.int32, device="cuda")
    h.project_device(R, x, n, whole, stream=torch.cuda.current_stream())
    for s in range(0, n, 100_000):
        m = min(100_000, n - s)
        h.project_device(R, x[s:s + m], m, part[s:s + m], stream=torch.cuda.current_stream())
    assert torch.equal(whole, part)
