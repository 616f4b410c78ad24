"""GPU test of the engine's batched admission and retirement: more systems than a
batch's table holds, more particles than its buffer holds, a system larger than
the buffer, and systems that are suspended and resumed beside them.  With no
steps a system comes back as it went in (the two half kicks cancel up to the
rounding of v + k - k)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, seed):
    r = np.random.default_rng(seed)
    return {"pos": r.normal(0.0, 1.0, (n, 3)), "vel": r.normal(0.0, 1.0, (n, 3)), "mass": r.uniform(0.5, 1.5, n) / n}


@pytest.mark.parametrize("sizes", [[1, 2, 3, 5, 7] * 220, [20000] * 9 + [3], [64, 160000, 1, 149000, 200]])
def test_systems_come_back(nb, sizes):
    eng = nb.Engine(max_particles=sum(sizes), max_systems=len(sizes))
    for _ in range(2):  # the second round reuses ranges and slots in another order
        ds = [_system(n, k) for k, n in enumerate(sizes)]
        ids = [eng.submit(d, 0.5, 1e-6, 0) for d in ds]
        eng.run_until_idle()
        for d, i, n in zip(ds, ids, sizes):
            got = eng.fetch(i, n)
            np.testing.assert_array_equal(got["pos"], d["pos"])
            np.testing.assert_allclose(got["vel"], d["vel"], rtol=0, atol=1e-14)
        sizes = sizes[::-1]
    st = eng.stats()
    assert st["running"] == 0 and st["resident_particles"] == 0


def test_resumed_beside_new_systems(nb):
    kw = dict(max_particles=1 << 15, max_systems=8)
    d, others = _system(3000, 1), [_system(500, 2), _system(700, 3)]
    ref = nb.Engine(**kw)
    i = ref.submit(d, 0.05, 1e-3, 20)
    ref.run_until_idle()
    want = ref.fetch(i, 3000)
    eng = nb.Engine(**kw)
    i = eng.submit(d, 0.05, 1e-3, 20)
    eng.run(7)
    eng.suspend(i)
    a = eng.submit(others[0], 0.05, 1e-3, 4)
    eng.resume(i)
    b = eng.submit(others[1], 0.05, 1e-3, 6)
    eng.run_until_idle()
    got = eng.fetch(i, 3000)
    np.testing.assert_array_equal(got["pos"], want["pos"])
    np.testing.assert_array_equal(got["vel"], want["vel"])
    assert eng.fetch(a, 500)["pos"].shape == (500, 3) and eng.fetch(b, 700)["pos"].shape == (700, 3)
