"""GPU test of the paths that memory or the GPU's room would choose: the sort by the
chain of kernels at the sizes that a cluster sorts, and an engine without
staging buffers."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [2, 6, 8])
@pytest.mark.parametrize("n", [1, 2, 511, 513, 2047, 2049, 8193, 30000, 65537, 131072, 131073])
def test_sorts_agree(nb, n, passes):
    L = nb._lib
    r = np.random.default_rng(n)
    key = r.integers(0, 1 << 63, n, dtype=np.uint64) << np.uint64(1) | r.integers(0, 2, n, dtype=np.uint64)
    key[::3] = key[0]  # ties
    low = key & np.uint64((1 << (8 * passes)) - 1)
    want = np.argsort(low, kind="stable").astype(np.int32)
    for chain in (0, 1):
        perm = np.full(n, -1, dtype=np.int32)
        rc = L.load().nb_selftest_sort(0, n, key.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), passes, chain,
                                       perm.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
        assert rc == L.NB_OK
        np.testing.assert_array_equal(perm, want)


def test_sort_arguments(nb):
    L = nb._lib
    k, p = (ctypes.c_uint64 * 1)(), (ctypes.c_int32 * 1)()
    for n, passes in ((0, 8), (1, 3), (1, 0), (1, 10)):
        assert L.load().nb_selftest_sort(0, n, k, passes, 0, p) == L.NB_ERR_INVALID_ARG


def test_engine_without_staging(nb):
    """Systems that move one at a time: the bits of those that move in batches."""
    L = nb._lib
    sizes = [1, 64, 3000, 5000, 200]
    ds = [nb.plummer(n, seed=n) if n > 1 else {"pos": np.ones((1, 3)), "vel": np.ones((1, 3)), "mass": np.ones(1)}
          for n in sizes]
    got = []
    for without in (0, 1):
        eng = nb.Engine(max_particles=sum(sizes), max_systems=len(sizes))
        assert L.load().nb_selftest_engine(eng.handle, L.NB_SELFTEST_NO_STAGING, without) == L.NB_OK
        ids = [eng.submit(d, 0.02, 1e-3, 2 + k) for k, d in enumerate(ds)]
        eng.run_until_idle()
        got.append([eng.fetch(i, n) for i, n in zip(ids, sizes)])
    assert L.load().nb_selftest_engine(eng.handle, L.NB_SELFTEST_NO_STAGING, 0) == L.NB_OK
    for a, b in zip(*got):
        for k in ("pos", "vel"):
            np.testing.assert_array_equal(a[k], b[k])
