"""The row windows a volume runs with (host only): the last one split and narrow
ones on fewer lanes where that is fewer x-tiles."""
import ctypes

import pytest

from niftyrec_gb300._lib import load


def windows(size, k):
    L, n = load(), ctypes.c_int(0)
    out = (ctypes.c_int * (5 * 64))()
    assert L.nrgb_volume_windows((ctypes.c_int * 3)(*size), k, out, 64, ctypes.byref(n)) == 0
    return [tuple(out[5 * i:5 * i + 5]) for i in range(n.value)]


def tiles(nx, lanes):
    return -(-nx // (1024 // lanes))


@pytest.mark.parametrize("k", [0, 1, 5, 9, 11, 15])
@pytest.mark.parametrize("nx", [1, 31, 32, 33, 64, 65, 66, 97, 128, 129, 132, 256])
def test_windows_partition_the_rows(k, nx):
    """As the unsplit windows: starts and valid ranges on multiples of 4, valid
    ranges a partition in order, every valid row's PSF support in its window; and
    no more x-tiles than the unsplit windows on 32 lanes."""
    L, r = load(), (k - 1) // 2 if k else 0
    for ny in list(range(1, 300)) + [511, 512, 513, 1000]:
        expect, cost = 0, 0
        for row0, rows, lo, hi, lanes in windows((nx, ny, 16), k):
            assert row0 % 4 == 0 and 0 < rows <= 4 * lanes and lanes in (8, 16, 32) and row0 + rows <= ny
            assert 0 <= lo < hi <= rows and row0 + lo == expect
            assert (row0 + lo) % 4 == 0 and ((row0 + hi) % 4 == 0 or row0 + hi == ny)
            for y in (row0 + lo, row0 + hi - 1):
                assert max(0, y - r) >= row0 and min(ny - 1, y + r) < row0 + rows, (ny, y)
            expect, cost = row0 + hi, cost + tiles(nx, lanes)
        assert expect == ny
        out, n = (ctypes.c_int * (4 * 64))(), ctypes.c_int(0)
        assert L.nrgb_row_windows(ny, k, out, 64, ctypes.byref(n)) == 0
        assert cost <= n.value * tiles(nx, 32), ny


def test_lanes_and_splits():
    assert windows((256, 256, 256), 15) == [(0, 128, 0, 120, 32), (112, 128, 8, 120, 32), (224, 32, 8, 32, 8)]
    assert [w[1::3] for w in windows((192, 192, 192), 15)] == [(128, 32), (64, 16), (32, 8)]
    assert [w[4] for w in windows((66, 60, 10), 11)] == [16] and [w[4] for w in windows((32, 60, 10), 11)] == [32]
    # the separated PSF in shared memory (too many planes for the launch parameters): 32 lanes, no split
    assert [w[4] for w in windows((192, 192, 257), 15)] == [32, 32]


def test_refusals():
    L, n, out = load(), ctypes.c_int(0), (ctypes.c_int * 5)()
    size = ctypes.c_int * 3
    for s, k in (((0, 8, 8), 5), ((8, 0, 8), 5), ((8, 8, 0), 5), ((8, 8, 8), 4), ((8, 8, 8), 17), ((8, 8, 8), -1)):
        assert L.nrgb_volume_windows(size(*s), k, out, 1, ctypes.byref(n)) == 2
    assert L.nrgb_volume_windows(size(256, 256, 256), 15, out, 1, ctypes.byref(n)) == 2 and n.value == 3
