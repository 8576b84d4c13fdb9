"""The gridding tiles' segment tables (cg_tiles.cuh), on the CPU: for every grid
length a plan or a NUFFT can have and every kernel width, the hive rows that a tile
and its halo list must fit the table that the launch allocates, and one periodic
wrap must take each of them into the grid."""
import ctypes

import pytest

T = 16  # cells of a gridding tile along an axis


@pytest.fixture(scope="module")
def lib(host_index):
    host_index.t_raw_hive_lo.restype = host_index.t_raw_hive_hi.restype = ctypes.c_int
    return host_index


def _lengths(most):
    for n in range(4, most + 1, 2):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            yield n


def _slots(lib, nf2, nw, W):
    slots, planes = ctypes.c_int(), ctypes.c_int()
    lib.t_grid_tiling(64, nf2, nw, W, ctypes.byref(slots), ctypes.byref(planes))
    return slots.value, planes.value


@pytest.mark.parametrize("W", range(2, 17))
def test_hive_rows_fit_the_table(lib, W):
    lo, hi = (W - 1) // 2, (W + 1) // 2
    for nf in _lengths(520):
        if nf < 2 * W:
            continue
        nh = (nf - 1) // 8 + 1
        most = 0
        for t0 in range(0, nf, T):
            cells = range(t0 - hi, min(t0 + T, nf) + lo)
            assert -nf <= cells[0] and cells[-1] < 2 * nf
            # hives of the cells, wrapped ones below 0 and from nh on
            listed = set()
            for c in cells:
                listed.add(c // 8 if 0 <= c < nf else ((c + nf) // 8 - nh if c < 0 else nh + (c - nf) // 8))
            a = lib.t_raw_hive_lo(cells[0], nf, nh)
            b = lib.t_raw_hive_hi(cells[-1], nf, nh)
            assert (a, b) == (min(listed), max(listed)) and -nh <= a and b < 2 * nh, (nf, t0)
            most = max(most, b - a + 1)
        for nw in (2 * W, 2 * W + 2, 48, 54, 200):
            if nw < 2 * W:
                continue
            slots, planes = _slots(lib, nf, nw, W)
            # three runs of every listed row of every plane that reaches the item
            assert 3 * most * (planes + W) <= slots, (nf, nw, most, slots)
