"""The pieces in which host arrays cross to and from the device: they cover the
array once, and no copy has a pitch beyond what a 2-D copy may have (CPU)."""
import ctypes as C

import pytest

import bnm_cuda_b200 as B

PIECE = 128 * 1024  # values

# rows, values per row, values from row to row on the device: single rows up to and past 2^29 values (FCDs of 803
# series of 668,746 values), series of a batch with removed frames in front, rows longer than a piece, far rows
CASES = [(1, 70_000, 70_000), (1, PIECE, PIECE), (1, PIECE + 1, PIECE + 1), (1, 1 << 29, 1 << 29),
         (1, 803 * 668_746, 803 * 668_746), (64, 585 * 100, 625 * 100), (5, 505 * 130, 520 * 130),
         (3, 1100 * 130, 1110 * 130), (2000, 180, 240), (300, 1000, 1000), (40, 2000, 1 << 29), (3, PIECE + 5, 1 << 30)]


@pytest.mark.parametrize("rows,length,pitch", CASES)
def test_pieces_cover_the_array_once(rows, length, pitch):
    f = B.lib().bnm_transfer_piece
    f.argtypes, f.restype = [C.c_int64] * 4 + [C.POINTER(C.c_int64)], C.c_int64
    out = (C.c_int64 * 5)()
    count, at = f(rows, length, pitch, -1, out), 0
    for k in range(count):
        f(rows, length, pitch, k, out)
        host, dev, r, n, contiguous = out
        row, col = divmod(at, length)
        assert host == at and dev == row * pitch + col
        assert 0 < r * n <= PIECE and (n == length or r == 1)
        assert contiguous == (r == 1 or pitch == length)
        assert contiguous or 4 * pitch < 1 << 31
        at += r * n
    assert at == rows * length
