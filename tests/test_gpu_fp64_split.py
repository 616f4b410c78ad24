"""GPU test of the FP64 force whose sources are split over several CTAs (few
targets): against the oracle at the 1e-12 bar of the FP64 form, at the sizes
where the split changes (no part, parts of 32 sources, ragged parts, blocks
that leave no room for a second part), with an active list, and at probes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAR = 1e-12


def _rel(a, b):
    return np.linalg.norm(a - b, axis=-1) / np.maximum(np.linalg.norm(b, axis=-1), 1e-300)


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("n", [2, 63, 64, 129, 1000, 4097])
def test_fp64_split_matches_oracle(nb, oracle, n, law):
    h = 0.01
    d = nb.plummer(n, seed=n)
    sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, TimeStep=1e-3, precision="fp64", law=law)
    nb.compute_force(sim, want_potential=True)
    g = nb.get_all_data(sim)
    lw = 0 if law == "spline" else 1
    a, p = oracle.force(d["pos"], d["mass"], d["pos"], h, law=lw)
    assert _rel(g["acc"], a).max() <= BAR
    assert np.abs((g["pot"] - p) / p).max() <= BAR
    # probes: another number of target blocks against the same sources
    q = np.random.default_rng(n).normal(0.0, 1.0, (300, 3))
    acc, pot = nb.force_and_potential_at_points(sim, q, h)
    a, p = oracle.force(d["pos"], d["mass"], q, h, law=lw)
    assert _rel(acc, a).max() <= BAR
    assert np.abs((pot - p) / p).max() <= BAR


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("scale", [1e-60, 1e-46, 1e-3, 1e44, 1e46, 1e60])
def test_fp64_roots_over_the_exponent_range(nb, oracle, scale, law):
    """Lengths from 1e-60 to 1e60: squares inside, at the edges of and outside
    the range of the fast root, where the compiler's takes over."""
    n, h = 400, 0.02 * scale
    d = nb.plummer(n, seed=8)
    d["pos"] = d["pos"] * scale
    sim = nb.Simulation(d, G=3.7, ForceSofteningTable=[h] * 6, TimeStep=1e-3, precision="fp64", law=law)
    nb.compute_force(sim, want_potential=True)
    g = nb.get_all_data(sim)
    a, p = oracle.force(d["pos"], d["mass"], d["pos"], h, G=3.7, law=0 if law == "spline" else 1)
    assert (np.abs(g["acc"] - a).max(1) / np.abs(a).max(1)).max() <= BAR
    assert np.abs((g["pot"] - p) / p).max() <= BAR


@pytest.mark.parametrize("n_active", [1, 128, 129, 2500])
def test_fp64_split_with_active_list(nb, oracle, n_active):
    n, h = 3000, 0.02
    d = nb.plummer(n, seed=5)
    sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, TimeEnd=1.0, MaxStep=1e-2, precision="fp64")
    act = np.random.default_rng(1).permutation(n)[:n_active]
    end = np.full(n, 4096, dtype=np.int64)
    end[act] = 0
    sim.upload_acc(np.full((n, 3), 7.0))
    sim.upload_bins(np.zeros(n, dtype=np.int64), end)
    nb.compute_force(sim)
    g = nb.get_all_data(sim)
    a, _ = oracle.force(d["pos"], d["mass"], d["pos"][act], h)
    assert _rel(g["acc"][act], a).max() <= BAR
    rest = np.setdiff1d(np.arange(n), act)
    assert np.all(g["acc"][rest] == 7.0)
