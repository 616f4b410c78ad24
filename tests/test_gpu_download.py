"""GPU test of nb_download into arrays of every arrangement: evenly spaced pinned
rows (one strided copy), rows with gaps, reversed rows, pageable rows, single
arrays, and sizes on both sides of the strided copy's limit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 65536, 65537])
@pytest.mark.parametrize("how", ["pinned", "padded", "reversed", "pageable", "some"])
def test_download_arrangements(nb, n, how):
    torch = pytest.importorskip("torch")
    from astronbodysim import _lib as L

    r = np.random.default_rng(n)
    d = {"pos": r.normal(0, 1, (n, 3)), "vel": r.normal(0, 1, (n, 3)), "mass": np.ones(n)}
    sim = nb.Simulation(d, ForceSofteningTable=[0.1] * 6, TimeStep=1e-3)
    acc = r.normal(0, 1, (n, 3))
    sim.upload_acc(acc)
    want = np.concatenate([d["pos"].T, d["vel"].T, acc.T, np.zeros((1, n))])
    width = n + 7 if how == "padded" else n
    buf = torch.full((10, width), float("nan"), dtype=torch.float64, pin_memory=how != "pageable")
    rows = [buf[9 - k] if how == "reversed" else buf[k] for k in range(10)]
    take = (0, 1, 4, 5, 6, 9) if how == "some" else range(10)
    ptr = [ctypes.cast(rows[k].data_ptr(), ctypes.POINTER(ctypes.c_double)) if k in take else None
           for k in range(10)]
    L.check(sim.handle, L.load().nb_download(sim.handle, *ptr, None, None))
    for k in range(10):
        got = rows[k].numpy()
        if k in take:
            np.testing.assert_array_equal(got[:n], want[k])
            assert np.all(np.isnan(got[n:]))
        else:
            assert np.all(np.isnan(got))
