"""BitHash codes where the tensor-core kernel changes path (GPU).

Bit for bit against the oracle's sequential projection: tiles of 128 vectors
and 128 hyperplanes with remainders, dimensions around the 32-wide chunk and
around the limit of resident hyperplanes (256), rows without 16-byte
alignment; and data whose sums the tensor cores may not decide: sums that
are zero or rounding noise in every bit, zero vectors, values near under-
and overflow, infinities and NaN.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _project(cuda, song, R, x, off=0):
    """Codes by the device entry point; `off` floats of misalignment."""
    torch = cuda
    bits, dim = R.shape
    n = x.shape[0]
    bh = song.BitHash(dim, 1, bits)
    d_R = torch.from_numpy(np.ascontiguousarray(R)).cuda()
    buf = torch.zeros(n * dim + off, device="cuda")
    buf[off:] = torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda()
    codes = torch.full((n, bits // 32), -1, dtype=torch.int32, device="cuda")
    bh.project_device(d_R, buf[off:], n, codes)
    torch.cuda.synchronize()
    return codes.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n,dim,bits,off", [
    (1, 1, 32, 0), (127, 31, 32, 1), (128, 32, 128, 0), (129, 33, 160, 2), (385, 255, 96, 0),
    (700, 256, 512, 0), (700, 257, 256, 0), (300, 289, 1024, 0), (40000, 64, 128, 0), (260, 960, 64, 0),
])
def test_gaussian_edges(cuda, song, oracle, n, dim, bits, off):
    rng = np.random.default_rng(n + dim)
    R = oracle.bithash_matrix(dim, bits, seed=dim)
    x = rng.normal(size=(n, dim)).astype(np.float32)
    np.testing.assert_array_equal(_project(cuda, song, R, x, off), oracle.bithash_project(R, x))


@pytest.mark.parametrize("dim", [64, 200, 320])
def test_sums_near_zero(cuda, song, oracle, dim):
    """Every second element undoes the one before it, up to rounding noise:
    all bits of these vectors hang on the sequential sum's roundings."""
    rng = np.random.default_rng(dim)
    R = rng.normal(size=(256, dim)).astype(np.float32)
    R[:, 1::2] = R[:, 0::2]
    x = rng.normal(size=(400, dim)).astype(np.float32)
    x[:, 1::2] = -x[:, 0::2]
    x[::3, 1::2] *= np.float32(1 + 2.0 ** -20)
    x[5] = 0.0
    x[6] = -0.0
    np.testing.assert_array_equal(_project(cuda, song, R, x), oracle.bithash_project(R, x))


def test_extreme_values(cuda, song, oracle):
    rng = np.random.default_rng(9)
    R = rng.normal(size=(128, 96)).astype(np.float32)
    x = rng.normal(size=(300, 96)).astype(np.float32)
    x[10:20] *= np.float32(1e-38)
    x[20:30] *= np.float32(1e-44)
    x[30:40] *= np.float32(1e37)
    x[40:50] *= np.float32(3e38)
    x[50, 3] = np.inf
    x[51, 3], x[51, 4] = np.inf, -np.inf
    x[52, 7] = np.nan
    x[53:60, ::2] *= np.float32(1e-30)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(_project(cuda, song, R, x), oracle.bithash_project(R, x))
