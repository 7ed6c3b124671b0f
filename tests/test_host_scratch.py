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
