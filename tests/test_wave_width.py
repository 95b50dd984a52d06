"""The width of the widest wave, which decides the number of clusters and whether tickets are taken late: at
least the blocks that any tile of those superblocks has in one wave, recounted block by block, and no more than
a whole tile's.  Host code; no device call."""
import ctypes as C

import numpy as np
import pytest

COL, ROW = 22, 30  # waves from a superblock to the next one right, and down
INSIDE = np.array([[0, 1, 4, 5, 8, 9, 14, 15], [2, 3, 6, 7, 12, 13, 16, 17], [4, 7, 10, 11, 14, 17, 20, 21],
                   [8, 9, 12, 13, 18, 19, 22, 23], [10, 13, 16, 19, 22, 23, 28, 29], [14, 15, 20, 21, 26, 27, 30, 31],
                   [16, 21, 24, 25, 28, 31, 34, 35], [22, 23, 26, 27, 32, 33, 36, 37]])


def _widest(nbx, nby):
    y, x = np.mgrid[0:nby, 0:nbx]
    return int(np.bincount((COL * (x >> 3) + ROW * (y >> 3) + INSIDE[y & 7, x & 7]).ravel()).max())


@pytest.mark.parametrize("sizes", ["small", "large"])
def test_no_tile_has_a_wider_wave(mt_lib, sizes):
    f = mt_lib.load()._ZN3mth11widest_waveEii
    f.restype, f.argtypes = C.c_int, (C.c_int, C.c_int)
    grid = range(1, 81, 1) if sizes == "small" else (1, 64, 97, 240, 333, 512)
    for nbx in grid:
        for nby in grid:
            cols, rows = -(-nbx // 8), -(-nby // 8)
            got = f(cols, rows)
            assert _widest(nbx, nby) <= got, (nbx, nby)
            if nbx % 8 == 0 and nby % 8 == 0:
                assert got == _widest(nbx, nby), (nbx, nby)
