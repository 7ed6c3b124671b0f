"""Sizes of scratch that the library asks for, worked out on the host: no GPU is needed."""
import ctypes

import pytest


@pytest.mark.parametrize("heads", [1, 2, 4, 8])
@pytest.mark.parametrize("c", [4, 8, 16, 20, 32, 47, 64])
def test_weights_of_a_full_last_tile_are_in_the_workspace(heads, c):
    """The lane groups of a warp read weights for as many edges as the longest of their tiles has, in steps of up to eight: a
    last tile of one edge is read as if it were full."""
    import cxgnncomp_backend as be
    fn = be._lib.cxg_gat_fused_weights_room
    fn.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_size_t)]
    fn.restype = ctypes.c_int
    tile, room = ctypes.c_int(0), ctypes.c_size_t(0)
    taken = 0
    for base in (1, 5000, 430_000, 530_000, 1_050_000, 2_300_000, 20_000_000, 300_000_000):
        assert fn(1000, base, heads, c, ctypes.byref(tile), ctypes.byref(room)) == 0
        step = max(tile.value, 1)
        for nnz in (base, base // step * step + 1, base // step * step + step // 2, base // step * step + step):
            assert fn(1000, nnz, heads, c, ctypes.byref(tile), ctypes.byref(room)) == 0
            if tile.value == 0:
                continue
            taken += 1
            last = (nnz - 1) // tile.value * tile.value
            assert (last + (tile.value + 7) // 8 * 8) * heads * 4 <= room.value, (nnz, tile.value)
    # rows of up to 512 bytes in whole vectors come here from 128 MB on, others always but where vectors lie across heads
    assert taken > 0 or (c == 47 and heads >= 4)


@pytest.mark.parametrize("n_src,feat,bf16,want", [
    (33_554_432, 47, False, 8 << 30), (33_554_433, 47, False, 0), (16_777_216, 101, False, 8 << 30), (16_777_217, 101, False, 0),
    (33_554_432, 101, True, 8 << 30), (111_000_000, 47, False, 0)])
def test_copied_rows_have_a_limit(n_src, feat, bf16, want):
    """A copy of x in whole lines is at most 8 GiB, however often the graph reads a row."""
    import cxgnncomp_backend as be
    fn = be._lib.cxg_spmm_csr_rows_size
    fn.argtypes, fn.restype = [ctypes.POINTER(be.SpmmDesc), ctypes.c_int64, ctypes.POINTER(ctypes.c_size_t)], ctypes.c_int
    desc = be.SpmmDesc()
    desc.n_dst, desc.nnz, desc.feat, desc.heads = 1000, 13 * n_src, feat, 1
    desc.dtype = be.CXG_BF16 if bf16 else be.CXG_F32
    desc.ptr_bytes = desc.idx_bytes = 8
    size = ctypes.c_size_t(1)
    assert fn(ctypes.byref(desc), n_src, ctypes.byref(size)) == 0
    assert size.value == want
