"""GPU test of the constant step whose drift rides on the pack and whose kick and
join ride on the force kernel, against the same step from its single
operations, and of the built-in j-split against an explicit one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 127, 128, 129, 1000, 3841, 16385, 33000, 70001]


def _data(nb, n):
    d = nb.plummer(n, seed=n) if n > 2 else {"pos": np.array([[0.1, 0.2, 0.3], [0.4, -0.1, 0.2]])[:n],
                                             "vel": np.full((n, 3), 0.25), "mass": np.full(n, 0.5)}
    d["mass"] = np.random.default_rng(n).uniform(0.5, 1.5, n) / n
    return d


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("n", SIZES)
def test_fused_step_is_the_step_of_single_operations(nb, n, law):
    """drift, force, kick as calls of their own: the same operations in the same
    order, so bit-identical; several softening lengths, so h comes by type."""
    dt, steps = 1e-3, 3
    d = _data(nb, n)
    d["collection"] = np.random.default_rng(n + 1).integers(1, 7, n)
    kw = dict(ForceSofteningTable=[0.01, 0.02, 0.005, 0.03, 0.01, 0.04], TimeStep=dt, TimeEnd=1.0, law=law,
              resort_every=1)
    a, b = nb.Simulation(d, **kw), nb.Simulation(d, **kw)
    for s in (a, b):
        nb.compute_force(s)
        nb.leapfrog_half_kick(s, +1)
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
    assert a.time() == b.time()
    assert nb.counters(a) == (steps, float(steps) * n * n)


@pytest.mark.parametrize("n", SIZES[3:])
def test_builtin_split_against_no_split(nb, n):
    """Any split joins compensated sums (about 48 bits): relative 1e-12 of the
    largest acceleration between the built-in split and no split on the same
    tiles, with the potential."""
    d = _data(nb, n)
    tj = 128 if n < 1 << 15 else 256
    ipt = 1 if n < 1 << 16 else 2
    a = nb.Simulation(d, ForceSofteningTable=[0.01] * 6)
    b = nb.Simulation(d, ForceSofteningTable=[0.01] * 6, block=128, i_per_thread=ipt, j_split=1, tile_j=tj)
    got = []
    for s in (a, b):
        nb.compute_force(s, want_potential=True)
        got.append(nb.get_all_data(s))
    for k in ("acc", "pot"):
        assert np.abs(got[0][k] - got[1][k]).max() <= 1e-12 * np.abs(got[1][k]).max()


@pytest.mark.parametrize("n,points", [(3000, 1), (3000, 129), (3000, 40000), (300, 100000)])
def test_probes_against_no_split(nb, n, points):
    """Probes share the split of the particles as far as its scratch goes (the
    last case has no room for a second part): against a handle whose probes
    are not split, on the same tiles."""
    d, h = nb.plummer(n, seed=3), 0.01
    q = np.random.default_rng(4).normal(0.0, 1.0, (points, 3))
    got = []
    for kw in ({}, dict(block=128, i_per_thread=1, j_split=1, tile_j=128)):
        sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, **kw)
        got.append(nb.force_and_potential_at_points(sim, q, h))
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("n_active", [1, 128, 129, 1000, 40000])
def test_active_list_is_split_on_the_device(nb, n_active):
    """The active targets of an adaptive step get more parts the fewer they are:
    their accelerations against those of all particles (1e-12 of the largest),
    the others keep theirs."""
    n, h = 40000, 0.01
    d = nb.plummer(n, seed=9)
    kw = dict(ForceSofteningTable=[h] * 6, TimeEnd=1.0, MaxStep=1e-2)
    full = nb.Simulation(d, **kw)
    nb.compute_force(full)
    ref = nb.get_all_data(full)["acc"]
    act = np.sort(np.random.default_rng(2).permutation(n)[:n_active])
    end = np.full(n, 4096, dtype=np.int64)
    end[act] = 0
    sim = nb.Simulation(d, **kw)
    sim.upload_acc(np.full((n, 3), 7.0))
    sim.upload_bins(np.zeros(n, dtype=np.int64), end)
    nb.compute_force(sim)
    got = nb.get_all_data(sim)["acc"]
    rest = np.setdiff1d(np.arange(n), act)
    assert np.all(got[rest] == 7.0)
    e = np.linalg.norm(got[act] - ref[act], axis=1) / np.linalg.norm(ref[act], axis=1)
    assert np.median(e) <= 1e-6 and np.quantile(e, 0.99) <= 1e-5 and e.max() <= 1e-4


@pytest.mark.parametrize("resort", [1, 3, 5, 16])
@pytest.mark.parametrize("adaptive", [False, True])
def test_steps_do_not_depend_on_how_they_are_asked_for(nb, resort, adaptive):
    """Calls of 1 .. 17 steps replay graphs of one or four steps between the sorts:
    the same states as one step at a time, bit for bit."""
    d = nb.plummer(700, seed=2)
    kw = dict(ForceSofteningTable=[0.02] * 6, TimeEnd=4.0, resort_every=resort, MaxStep=1e-2)
    kw.update({} if adaptive else {"TimeStep": 1e-3})
    a, b = nb.Simulation(d, **kw), nb.Simulation(d, **kw)
    for s in (a, b):
        nb.compute_force(s)
        nb.init_timesteps(s)
        nb.leapfrog_half_kick(s, +1)
    for k in (1, 2, 9, 4, 17, 3, 5):
        nb.step(a, k)
        for _ in range(k):
            nb.step(b, 1)
        ga, gb = nb.get_all_data(a), nb.get_all_data(b)
        for key in ("pos", "vel", "acc", "ti_endstep"):
            np.testing.assert_array_equal(ga[key], gb[key])
    assert a.time() == b.time() and nb.counters(a) == nb.counters(b)


@pytest.mark.parametrize("n", [1, 127, 129, 1000, 33000, 131072, 131073])
def test_adaptive_step_is_the_step_of_single_operations(nb, n):
    """Start, pack with drift and counts, list and kick of the adaptive step
    against min end step, drift, force and kick as calls of their own: the same
    operations, so bit-identical (the last sizes: lists from counts that each
    block sums, and from a scan)."""
    d = _data(nb, n)
    d["collection"] = np.random.default_rng(n + 1).integers(1, 7, n)
    kw = dict(ForceSofteningTable=[0.01, 0.02, 0.005, 0.03, 0.01, 0.04], TimeEnd=4.0, MaxStep=1e-2, resort_every=1)
    a, b = nb.Simulation(d, **kw), nb.Simulation(d, **kw)
    for s in (a, b):
        nb.compute_force(s)
        nb.init_timesteps(s)
        nb.leapfrog_half_kick(s, +1)
    total = 0.0
    for _ in range(6):
        nb.step(a, 1)
        nb.drift_particles_adaptive_timestep(b, nb.find_min_endstep(b))
        total += float(nb.active_count(b)) * n
        nb.compute_force(b)
        nb.advance_and_find_timestep(b)
        ga, gb = nb.get_all_data(a), nb.get_all_data(b)
        for k in ("pos", "vel", "acc", "ti_begstep", "ti_endstep"):
            np.testing.assert_array_equal(ga[k], gb[k])
        assert a.time() == b.time()
    assert nb.counters(a) == (6, total)
