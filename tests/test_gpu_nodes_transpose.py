"""The transposition of the node radiosity's neighbour lists, both ways, at the edges of its 32 x 32 tiles and with more lists than
a grid has rows of blocks (2,097,120): every pair in its place."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (31, 16), (33, 33), (1000, 64), (2_097_121, 1), (2_100_001, 3)])
def test_transposition_and_back(n, k):
    from vtwin import _lib

    transpose = getattr(_lib.load(), "_ZN3vtk20launch_transpose_nbrEPK5uint2jjPS0_P11CUstream_st")   # vtk::launch_transpose_nbr
    transpose.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p]
    transpose.restype = None
    pairs = torch.arange(2 * n * k, dtype=torch.int32, device="cuda").reshape(n, k, 2)
    there, back = torch.full((k, n, 2), -1, dtype=torch.int32, device="cuda"), torch.full_like(pairs, -1)
    torch.cuda.synchronize()
    transpose(pairs.data_ptr(), n, k, there.data_ptr(), None)
    transpose(there.data_ptr(), k, n, back.data_ptr(), None)
    torch.cuda.synchronize()
    assert torch.equal(there, pairs.transpose(0, 1)) and torch.equal(back, pairs)
