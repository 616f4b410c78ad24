"""GPU test of nb_download into evenly spaced rows that are not one pinned
allocation: rows pinned one by one with pageable ones between them, and two
halves of a buffer pinned apart."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 65536  # a multiple of the host's page size


@pytest.mark.parametrize("how", ["ends", "alternate", "each", "halves", "all"])
def test_rows_of_several_allocations(nb, how):
    torch = pytest.importorskip("torch")
    from astronbodysim import _lib as L

    n = 8192  # rows of 64 KB
    r = np.random.default_rng(1)
    d = {"pos": r.normal(0, 1, (n, 3)), "vel": r.normal(0, 1, (n, 3)), "mass": np.ones(n)}
    sim = nb.Simulation(d, ForceSofteningTable=[0.1] * 6, TimeStep=1e-3)
    acc = r.normal(0, 1, (n, 3))
    sim.upload_acc(acc)
    want = np.concatenate([d["pos"].T, d["vel"].T, acc.T, np.zeros((1, n))])
    raw = np.full((12 * PAGE) // 8, np.nan)
    first = -(-raw.ctypes.data // PAGE) * PAGE
    rows = [first + k * PAGE for k in range(10)]
    pins = {"ends": [(0, 1), (9, 1)], "alternate": [(k, 1) for k in range(0, 10, 2)],
            "each": [(k, 1) for k in range(10)], "halves": [(0, 5), (5, 5)], "all": [(0, 10)]}[how]
    rt = torch.cuda.cudart()
    for k, count in pins:
        assert int(rt.cudaHostRegister(rows[k], count * PAGE, 0)) == 0
    try:
        ptr = [ctypes.cast(a, ctypes.POINTER(ctypes.c_double)) for a in rows]
        L.check(sim.handle, L.load().nb_download(sim.handle, *ptr, None, None))
        k0 = (first - raw.ctypes.data) // 8
        np.testing.assert_array_equal(raw[k0:k0 + 10 * n].reshape(10, n), want)
    finally:
        for k, _ in pins:
            assert int(rt.cudaHostUnregister(rows[k])) == 0
