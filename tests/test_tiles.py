"""The shapes behind the indices of fwi_get_tiles and fwi_set_tiles."""
import ctypes as C

from fwi3d_b200 import lib


def test_both_kernels_have_a_table_of_shapes():
    tables = lib.tile_table(), lib.tile_table(backward=True)
    assert len(tables[0]) == len(tables[1]) and tables[0] != tables[1]
    for tz, tx in tables[1]:
        assert tz % 4 == 0 and tx % 2 == 0 and 0 < tz + 8 <= 256 and 0 < tx + 8 <= 256
    so, x = lib.load(), C.c_int()
    for bad in (-1, len(tables[1])):
        assert so.fwi_backward_tile_shape(bad, C.byref(x), C.byref(x)) == 1
    assert so.fwi_backward_tile_shape(0, None, C.byref(x)) == 1
