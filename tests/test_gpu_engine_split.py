"""GPU test of the engine's force with the j-tiles of a system split over several
work items: sizes at and around the edges of the rule (8 tiles of 256 are the
fewest that are split), alone and in a mix (bit-identical), for every launch shape."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law,shape", [("spline", (128, 1)), ("spline", (128, 2)), ("spline", (256, 1)),
                                       ("spline", (256, 2)), ("plummer", (128, 2))])
def test_split_systems_alone_and_in_the_mix(nb, law, shape):
    """Sizes: one tile; 15 full tiles; the first size with 16 tiles (a last tile
    of one source); a partial last part; 8 parts with a large system.  Against
    the single-system path the tiles differ: the bars of the other engine tests
    (positions 1e-8, velocities 1e-6)."""
    sizes, dt, h, nsteps = [200, 3840, 3841, 5000, 17001], 1e-3, 0.01, 6
    kw = dict(max_particles=1 << 16, max_systems=16, law=law, block=shape[0], i_per_thread=shape[1])
    ds = [nb.plummer(n, seed=n) for n in sizes]
    mix = nb.Engine(**kw)
    ids = [mix.submit(d, h, dt, nsteps) for d in ds]
    mix.run_until_idle()
    for n, d, i in zip(sizes, ds, ids):
        got = mix.fetch(i, n)
        alone = nb.Engine(**kw)
        k = alone.submit(d, h, dt, nsteps)
        alone.run_until_idle()
        a = alone.fetch(k, n)
        np.testing.assert_array_equal(got["pos"], a["pos"])
        np.testing.assert_array_equal(got["vel"], a["vel"])
        sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, TimeStep=dt, TimeEnd=1.0, law=law)
        nb.run(sim, nsteps=nsteps)
        ref = nb.get_all_data(sim)
        np.testing.assert_allclose(got["pos"], ref["pos"], rtol=0, atol=1e-8)
        np.testing.assert_allclose(got["vel"], ref["vel"], rtol=0, atol=1e-6)


@pytest.mark.parametrize("law", ["spline", "plummer"])
def test_split_edges(nb, law):
    """The first sizes that are split (8 tiles, the last of one source), the last
    that are not, parts of 4 and 6 tiles, and more parts with a partial last
    tile: bit-identical alone and in a mix, and one step within the mixed form's
    bar of the single-system path (each form's accelerations within 1e-4 of the
    exact ones, so velocities within 2e-4 dt max|a| of each other)."""
    sizes, dt, h = [255, 1792, 1793, 3000, 8100], 1e-3, 0.01
    ds = [nb.plummer(n, seed=n) for n in sizes]
    mix = nb.Engine(max_particles=1 << 16, max_systems=16, law=law)
    ids = [mix.submit(d, h, dt, 1) for d in ds]
    mix.run_until_idle()
    for n, d, i in zip(sizes, ds, ids):
        got = mix.fetch(i, n)
        alone = nb.Engine(max_particles=1 << 16, max_systems=16, law=law)
        k = alone.submit(d, h, dt, 1)
        alone.run_until_idle()
        a = alone.fetch(k, n)
        np.testing.assert_array_equal(got["pos"], a["pos"])
        np.testing.assert_array_equal(got["vel"], a["vel"])
        sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, TimeStep=dt, TimeEnd=1.0, law=law)
        nb.run(sim, nsteps=1)
        ref = nb.get_all_data(sim)
        amax = np.abs(ref["acc"]).max()
        assert np.abs(got["vel"] - ref["vel"]).max() <= 2e-4 * dt * amax
        assert np.abs(got["pos"] - ref["pos"]).max() <= 2e-4 * dt * dt * amax
