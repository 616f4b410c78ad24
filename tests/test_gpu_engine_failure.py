"""GPU test of the engine when the copy of a batch of systems fails on the host
(nb_selftest_engine makes the n-th one fail): no system runs whose particles are
not in the arena, none is lost, and the results after the error are those of an
engine that met none, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 20000 particles take 1.1 of a batch's 8 MB: seven to a batch, so nine systems take two
SIZES, STEPS, H, DT = [20000] * 9 + [300], [2] * 9 + [3], 0.05, 1e-3


def _submit(nb, eng):
    return [eng.submit(nb.plummer(n, seed=k + 1), H, DT, s) for k, (n, s) in enumerate(zip(SIZES, STEPS))]


def _engine(nb):
    return nb.Engine(max_particles=sum(SIZES), max_systems=len(SIZES))


@pytest.fixture(scope="module")
def undisturbed(nb):
    eng = _engine(nb)
    ids = _submit(nb, eng)
    eng.run_until_idle()
    return [eng.fetch(i, n) for i, n in zip(ids, SIZES)]


def _finish(eng, ids, undisturbed):
    eng.run_until_idle()
    for i, n, want in zip(ids, SIZES, undisturbed):
        got = eng.fetch(i, n)
        for k in ("pos", "vel"):
            np.testing.assert_array_equal(got[k], want[k])
    st = eng.stats()
    assert st["running"] == 0 and st["done"] == len(SIZES)


@pytest.mark.parametrize("which,running", [(1, 0), (2, 7)])
def test_failed_admission(nb, undisturbed, which, running):
    L = nb._lib
    eng = _engine(nb)
    ids = _submit(nb, eng)
    assert L.load().nb_selftest_engine(eng.handle, L.NB_SELFTEST_FAIL_MOVE, which) == L.NB_OK
    with pytest.raises(L.NbodyError) as err:
        eng.run()
    assert err.value.code == L.NB_ERR_CUDA and "self-test" in str(err.value)
    states = [eng.poll(i)[0] for i in ids]
    assert states == [L.NB_REQ_RUNNING] * running + [L.NB_REQ_QUEUED] * (len(ids) - running)
    st = eng.stats()
    assert st["queued"] == len(ids) - running and st["resident_particles"] == 20000 * running
    _finish(eng, ids, undisturbed)


def test_selftest_arguments(nb):
    L = nb._lib
    eng = _engine(nb)
    f = L.load().nb_selftest_engine
    assert f(eng.handle, 99, 1) == L.NB_ERR_INVALID_ARG
    assert f(eng.handle, L.NB_SELFTEST_FAIL_MOVE, -1) == L.NB_ERR_INVALID_ARG
    assert f(None, L.NB_SELFTEST_FAIL_MOVE, 1) == L.NB_ERR_INVALID_ARG


@pytest.mark.parametrize("which,done", [(1, 0), (2, 8)])
def test_failed_retirement(nb, undisturbed, which, done):
    """20000 particles take 0.96 MB on the way back, eight to a batch.  Those
    copied before the failure are done; the others are kicked back once."""
    L = nb._lib
    eng = _engine(nb)
    ids = _submit(nb, eng)
    assert eng.run(1) == 1
    assert L.load().nb_selftest_engine(eng.handle, L.NB_SELFTEST_FAIL_MOVE, which) == L.NB_OK
    with pytest.raises(L.NbodyError) as err:
        eng.run(1)
    assert err.value.code == L.NB_ERR_CUDA
    states = [eng.poll(i)[0] for i in ids]
    assert states == [L.NB_REQ_DONE] * done + [L.NB_REQ_RUNNING] * (len(ids) - done)
    assert eng.drain_done() == ids[:done]
    _finish(eng, ids, undisturbed)
    assert eng.drain_done() == ids[done:]
