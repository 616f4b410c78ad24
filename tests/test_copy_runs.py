"""CPU test of the download's choice of strided copies: a run of rows goes in one
copy only where every row lies in the pinned allocation of the first."""
import ctypes

import pytest

BASE, B = 1 << 20, 800  # first address, bytes of a row


def _runs(nb, dst, src, ranges, nbytes=B):
    u = lambda v: (ctypes.c_uint64 * max(1, len(v)))(*v)  # noqa: E731
    run = (ctypes.c_int32 * len(dst))()
    rc = nb.load().nb_selftest_copy_runs(len(dst), u(dst), u(src), nbytes, len(ranges),
                                         u([r[0] for r in ranges]), u([r[1] for r in ranges]), run)
    assert rc == nb._lib.NB_OK
    return list(run)


def _rows(n, step, first=BASE):
    return [first + k * step for k in range(n)]


SRC = _rows(10, 1024, 1 << 40)


@pytest.mark.parametrize("step", [B, B + 8, 4096])
def test_one_allocation(nb, step):
    rows = _rows(10, step)
    whole = [(BASE, rows[9] + B)]
    assert _runs(nb, rows, SRC, whole) == [10] + [0] * 9
    # one byte short of the last row, of the last but one; the first row before it
    assert _runs(nb, rows, SRC, [(BASE, rows[9] + B - 1)]) == [9] + [0] * 8 + [1]
    assert _runs(nb, rows, SRC, [(BASE, rows[8] + B - 1)]) == [8] + [0] * 7 + [1, 1]
    assert _runs(nb, rows, SRC, [(BASE + 1, rows[9] + B)]) == [1, 9] + [0] * 8
    assert _runs(nb, rows, SRC, []) == [1] * 10


def test_rows_of_several_allocations(nb):
    """Evenly spaced rows whose ends are pinned and whose middle is not, or is
    another allocation: no copy spans them."""
    rows = _rows(10, 4096)
    ends = [(rows[0], rows[0] + B), (rows[9], rows[9] + B)]
    assert _runs(nb, rows, SRC, ends) == [1] * 10
    assert _runs(nb, rows, SRC, [(r, r + B) for r in rows]) == [1] * 10
    assert _runs(nb, rows, SRC, [(r, r + 4096) for r in rows]) == [1] * 10
    halves = [(rows[0], rows[4] + B), (rows[5], rows[9] + B)]
    assert _runs(nb, rows, SRC, halves) == [5, 0, 0, 0, 0, 5, 0, 0, 0, 0]
    gap = [(rows[0], rows[3] + B), (rows[6], rows[9] + B)]
    assert _runs(nb, rows, SRC, gap) == [4, 0, 0, 0, 1, 1, 4, 0, 0, 0]


def test_spacing(nb):
    whole = [(0, 1 << 62)]
    assert _runs(nb, _rows(10, B - 8), SRC, whole) == [1] * 10           # overlapping
    assert _runs(nb, _rows(10, 4096)[::-1], SRC, whole) == [1] * 10      # descending
    assert _runs(nb, [BASE] * 10, SRC, whole) == [1] * 10                # one array for all
    some = _rows(10, 4096)
    some[2] = some[6] = 0                                                # not wanted
    assert _runs(nb, some, SRC, whole) == [2, 0, 1, 3, 0, 0, 1, 3, 0, 0]
    odd = _rows(10, 4096)
    odd[5] += 8
    assert _runs(nb, odd, SRC, whole) == [5, 0, 0, 0, 0, 2, 0, 3, 0, 0]
    src = list(SRC)
    src[4] += 256
    # rows 4 and 5 are then less than a row apart
    assert _runs(nb, _rows(10, 4096), src, whole) == [4, 0, 0, 0, 1, 5, 0, 0, 0, 0]
    far = _rows(10, (1 << 30) + 8)
    assert _runs(nb, far, SRC, whole) == [1] * 10
    assert _runs(nb, [BASE], SRC[:1], whole) == [1]


def test_arguments(nb):
    f = nb.load().nb_selftest_copy_runs
    run = (ctypes.c_int32 * 2)()
    u = (ctypes.c_uint64 * 2)(1, 2)
    bad = nb._lib.NB_ERR_INVALID_ARG
    assert f(0, u, u, 8, 0, None, None, run) == bad
    assert f(2, u, u, 0, 0, None, None, run) == bad
    assert f(2, u, u, 8, 1, None, None, run) == bad
    assert f(2, None, u, 8, 0, None, None, run) == bad
