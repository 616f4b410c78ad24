"""GPU test of the engine's partial sums when the memory for them ends: a system's
split depends on its size alone, so with room for one block's sums, for a few
blocks', or for all, alone or in a mix, its results are the same bits.  The
largest size has more blocks than leave it the most parts (the cap on a
system's items)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES, STEPS, H, DT = [300, 1500, 4100, 9000, 70001], [3, 2, 3, 1, 2], 0.02, 1e-3


def _run(nb, sizes, limit, **kw):
    L = nb._lib
    eng = nb.Engine(max_particles=1 << 17, max_systems=8, **kw)
    assert L.load().nb_selftest_engine(eng.handle, L.NB_SELFTEST_PARTIAL_ROWS, limit) == L.NB_OK
    ids = [eng.submit(nb.plummer(n, seed=n), H, DT, STEPS[SIZES.index(n)]) for n in sizes]
    eng.run_until_idle()
    return {n: eng.fetch(i, n) for n, i in zip(sizes, ids)}


@pytest.mark.parametrize("law,shape", [("spline", (128, 2)), ("plummer", (256, 2)), ("spline", (128, 1))])
def test_results_do_not_depend_on_the_memory(nb, law, shape):
    kw = dict(law=law, block=shape[0], i_per_thread=shape[1])
    want = _run(nb, SIZES, 0, **kw)
    for sizes, limit in [(SIZES, 1), (SIZES, 17), (SIZES, 100)] + [([n], 40) for n in SIZES]:
        got = _run(nb, sizes, limit, **kw)
        for n in sizes:
            for k in ("pos", "vel"):
                np.testing.assert_array_equal(got[n][k], want[n][k], err_msg="n %d limit %d" % (n, limit))


def test_largest_system_against_the_single_system_path(nb):
    """One step of the capped split: velocities within 2e-4 dt max|a| (each form's
    accelerations are within 1e-4 of the exact ones)."""
    n = SIZES[-1]
    d = nb.plummer(n, seed=n)
    eng = nb.Engine(max_particles=1 << 17, max_systems=8)
    i = eng.submit(d, H, DT, 1)
    eng.run_until_idle()
    got = eng.fetch(i, n)
    sim = nb.Simulation(d, ForceSofteningTable=[H] * 6, TimeStep=DT, TimeEnd=1.0)
    nb.run(sim, nsteps=1)
    ref = nb.get_all_data(sim)
    amax = np.abs(ref["acc"]).max()
    assert np.abs(got["vel"] - ref["vel"]).max() <= 2e-4 * DT * amax
    assert np.abs(got["pos"] - ref["pos"]).max() <= 2e-4 * DT * DT * amax


def test_growing_mix(nb):
    """Admissions that outgrow the buffer while others run: as each alone."""
    want = _run(nb, SIZES, 0)
    eng = nb.Engine(max_particles=1 << 17, max_systems=8, max_steps_per_call=1)
    ids = {}
    for n in SIZES:
        ids[n] = eng.submit(nb.plummer(n, seed=n), H, DT, STEPS[SIZES.index(n)])
        eng.run(1)
    eng.run_until_idle()
    for n in SIZES:
        got = eng.fetch(ids[n], n)
        for k in ("pos", "vel"):
            np.testing.assert_array_equal(got[k], want[n][k])
