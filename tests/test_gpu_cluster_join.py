"""GPU test of the join of a block whose parts are one cluster: the sums of all
parts to the last bit, and nothing at all when one part gave up waiting (no
partial sum is stored, kicked with or counted as a step)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _join(nb, parts, gave_up, n):
    acc, vel, t = np.full((3, 128), np.nan), np.full((3, 128), np.nan), ctypes.c_double(-1.0)
    L = nb._lib
    rc = L.load().nb_selftest_cluster_join(0, parts, gave_up, n, L.dptr(acc), L.dptr(vel), ctypes.byref(t))
    assert rc == L.NB_OK
    return acc, vel, t.value


@pytest.mark.parametrize("n", [1, 31, 127, 128])
@pytest.mark.parametrize("parts", range(1, 9))
def test_sums(nb, parts, n):
    acc, vel, t = _join(nb, parts, -1, n)
    # integers below 2^24 and carries of parts x (k + 1) 2^-40: every step is exact
    want = np.zeros((3, 128))
    for k in range(3):
        want[k, :n] = (2.0 ** parts - 1) + parts * np.arange(n) + parts * (k + 1) * 2.0 ** -40
    np.testing.assert_array_equal(acc, want)
    np.testing.assert_array_equal(vel, 0.5 * want)
    assert t == 0.5


@pytest.mark.parametrize("parts", range(1, 9))
def test_a_part_that_gave_up_leaves_everything_as_it_was(nb, parts):
    for gave_up in range(parts):
        for n in (1, 128):
            acc, vel, t = _join(nb, parts, gave_up, n)
            assert not acc.any() and not vel.any() and t == 0.0
