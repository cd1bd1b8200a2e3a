"""The allocation-free graph build over rows that are slices of a wide matrix.

The row stride is the caller's and may be far larger than the dimension: the
build must neither refuse it nor give another graph than the rows alone.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,ld", [(300, 16384), (300, 304), (40, 16384), (7, 4096)])
def test_wide_stride(cuda, song, ds, dim, ld):
    torch = cuda
    n = 700
    L = song.load_library()
    fn = L.song_build_graph_noalloc
    fn.argtypes = [C.c_int, C.c_void_p, C.c_int64, C.c_int, C.c_int, C.POINTER(song._Params),
                   C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    rows = ds.l1_mixture(n, 1, dim=dim, n_comp=8, seed=dim).base
    p = song.Params(block_size=32, fixed_degree=31)
    want = song.build_graph(rows, p)
    wide = torch.full((n, ld), 77.0, device="cuda")
    wide[:, :dim] = torch.from_numpy(rows).cuda()
    adj = torch.full((n, 32), 123, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = torch.cuda.current_stream().cuda_stream
    assert fn(song.KIND_L2, wide.data_ptr(), n, dim, ld, C.byref(p._c()), 32, 0, adj.data_ptr(), st) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(adj.cpu().numpy(), want)
