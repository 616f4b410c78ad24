"""GPU test of what a step does inside its kernels and no call does by itself: the
drift that rides on the pack between two sorts, against the same products and
sums in numpy, bit for bit; the step in explicit launch shapes against single
operations; and the cluster join of small systems against no split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOFT = [0.01, 0.02, 0.005, 0.03, 0.01, 0.04]
# tiles of 128, 256 and 512 sources, partial and full
SIZES = [1, 129, 1000, 4096, 33001, 140001]


def _data(nb, n):
    d = nb.plummer(n, seed=n) if n > 2 else {"pos": np.full((n, 3), 0.1), "vel": np.full((n, 3), 0.25)}
    d["mass"] = np.random.default_rng(n).uniform(0.5, 1.5, n) / n
    d["collection"] = np.random.default_rng(n + 1).integers(1, 7, n)
    return d


def _start(nb, d, **kw):
    sim = nb.Simulation(d, ForceSofteningTable=SOFT, **kw)
    nb.compute_force(sim)
    nb.init_timesteps(sim)
    nb.leapfrog_half_kick(sim, +1)
    return sim


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("n", SIZES)
def test_drift_and_kick_of_constant_steps(nb, n, law):
    dt, t = 1e-3, 0.0
    sim = _start(nb, _data(nb, n), TimeStep=dt, TimeEnd=1.0, law=law)
    a = nb.get_all_data(sim)
    for k in range(3):  # the first step sorts, the others drift in the pack
        nb.step(sim, 1)
        b = nb.get_all_data(sim)
        np.testing.assert_array_equal(b["pos"], a["pos"] + a["vel"] * ((t + dt) - t))
        np.testing.assert_array_equal(b["vel"], a["vel"] + b["acc"] * dt)
        t, a = t + dt, b
    # single operations on the same state: the pack's sources are the drifted ones
    nb.compute_force(sim)
    np.testing.assert_allclose(nb.get_all_data(sim)["acc"], b["acc"], rtol=0, atol=2e-4 * np.abs(b["acc"]).max())


@pytest.mark.parametrize("n", SIZES)
def test_drift_of_adaptive_steps(nb, n):
    sim = _start(nb, _data(nb, n), TimeEnd=4.0, MaxStep=1e-2)
    unit = 4.0 / (1 << 30)
    a, t = nb.get_all_data(sim), sim.time()[0]
    for _ in range(4):
        nb.step(sim, 1)
        b, now = nb.get_all_data(sim), sim.time()[0]
        assert now > t
        np.testing.assert_array_equal(b["pos"], a["pos"] + a["vel"] * (float(now - t) * unit))
        t, a = now, b


@pytest.mark.parametrize("shape", [(128, 1, 4, 128, 6), (128, 2, 3, 256, 3), (128, 4, 1, 256, 4), (256, 1, 8, 256, 4),
                                   (256, 2, 2, 512, 4), (256, 1, 1, 512, 3)])
@pytest.mark.parametrize("n", [130, 3001])
def test_explicit_shapes(nb, n, shape):
    """Every step sorts, so that single operations see the same order: the same bits."""
    block, ipt, js, tj, stages = shape
    dt, steps = 1e-3, 3
    kw = dict(TimeStep=dt, TimeEnd=1.0, block=block, i_per_thread=ipt, j_split=js, tile_j=tj, stages=stages,
              resort_every=1)
    d = _data(nb, n)
    a, b = _start(nb, d, **kw), _start(nb, d, **kw)
    nb.step(a, steps)
    t = 0.0
    for _ in range(steps):
        t = t + dt
        nb.drift_particles_const_timestep(b, t)
        nb.compute_force(b)
        nb.advance_and_find_timestep(b)
    ga, gb = nb.get_all_data(a), nb.get_all_data(b)
    for k in ("pos", "vel", "acc"):
        np.testing.assert_array_equal(ga[k], gb[k])


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("n", [129, 1000, 1025, 3841, 6144])
def test_cluster_join_against_no_split(nb, n, law):
    """Accelerations alone, which is what the cluster form computes: joins of
    compensated sums (about 48 bits), relative 1e-12 of the largest."""
    got = []
    for kw in ({}, dict(block=128, i_per_thread=1, j_split=1, tile_j=128)):
        sim = nb.Simulation(_data(nb, n), ForceSofteningTable=SOFT, TimeStep=1e-3, law=law, **kw)
        nb.compute_force(sim)
        got.append(nb.get_all_data(sim)["acc"])
    assert np.abs(got[0] - got[1]).max() <= 1e-12 * np.abs(got[1]).max()
